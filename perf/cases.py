"""Workloads of the imaging path, each one call of the public Python binding.

The optics are those of the benchmark configurations: 193 nm, NA 1.35 in water,
annular, dipole and cross-quadrupole sources, clips of 512^2 to 4096^2 pixels
of 1 nm under up to five focus values.  Kinds of case:

* ``forward``  SOCS images of a batch of clips under ``focus`` kernel sets
  (SocsPlan.forward); ``tuned`` plans ran SocsPlan.autotune when they were made.
* ``mixed``    clips of three sizes in one call (SocsBatch.forward).
* ``adjoint``  image, resist loss and mask gradient (SocsPlan.vjp), one step of
  a mask optimisation.
* ``hopkins``  the image without the kernel truncation (TccPlan.hopkins): one
  coherent field per source point.
* ``optics``   a new source and focus stack to images: TccPlan, topk_batch (topk
  for one focus), SocsPlan.set_kernels, SocsPlan.forward of one clip.
* ``tcc``      the transmission cross coefficients of a new source (TccPlan,
  TccPlan.build).
"""
from __future__ import annotations

import functools
import math
import os
import sys

import numpy as np
import torch

PACKAGE = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "k-litho_b200")
if PACKAGE not in sys.path:
    sys.path.insert(0, PACKAGE)

LAMBDA, NA, N_WATER = 193.0, 1.35, 1.44
FOCUS_STEP_NM = 25.0
ALPHA, THRESHOLD = 50.0, 0.225
# source grids: name -> (points per side, inner radius or pole offset, outer radius or pole radius)
SOURCES = {"annular": (41, 0.6, 0.9), "dipole": (61, 0.7, 0.15), "quadrupole": (81, 0.75, 0.12)}


def listed():
    return [
        # one small clip, one focus: an interactive simulation; latency and launches
        {"name": "clip_512", "kind": "forward", "Lx": 512, "Ly": 512, "clips": 1, "focus": 1, "K": 24,
         "source": "annular", "tuned": False},
        # full-chip tiles under a focus stack, the throughput workload
        {"name": "tiles_1024", "kind": "forward", "Lx": 1024, "Ly": 1024, "clips": 48, "focus": 3, "K": 24,
         "source": "annular", "tuned": True},
        # the batched benchmark's mixture of clip sizes at a quarter of its count
        {"name": "mixed_sizes", "kind": "mixed", "n512": 32, "n1024": 48, "n2048": 16, "focus": 3, "K": 24,
         "source": "annular", "tuned": True},
        # layout windows cut without regard to the transform length
        {"name": "ragged_1000x744", "kind": "forward", "Lx": 1000, "Ly": 744, "clips": 7, "focus": 2, "K": 17,
         "source": "annular", "tuned": False},
        # the largest field, 64 kernels, five focus values
        {"name": "field_4096", "kind": "forward", "Lx": 4096, "Ly": 4096, "clips": 4, "focus": 5, "K": 64,
         "source": "quadrupole", "tuned": False},
        # mask optimisation: one small clip, a batch, and larger clips
        {"name": "adjoint_512", "kind": "adjoint", "Lx": 512, "Ly": 512, "clips": 1, "focus": 1, "K": 24,
         "source": "annular"},
        {"name": "adjoint_1024", "kind": "adjoint", "Lx": 1024, "Ly": 1024, "clips": 32, "focus": 1, "K": 24,
         "source": "annular"},
        {"name": "adjoint_2048", "kind": "adjoint", "Lx": 2048, "Ly": 2048, "clips": 4, "focus": 1, "K": 32,
         "source": "dipole"},
        # the reference image of klitho_tcc: every source point, no truncation
        {"name": "hopkins_1024", "kind": "hopkins", "Lx": 1024, "Ly": 1024, "clips": 2, "source": "annular"},
        # source optimisation: each trial source needs its kernels; more points
        # than the one-step solver takes, and the largest field at five focus values
        {"name": "optics_1024", "kind": "optics", "Lx": 1024, "Ly": 1024, "focus": 1, "K": 24, "source": "annular"},
        {"name": "optics_4096", "kind": "optics", "Lx": 4096, "Ly": 4096, "focus": 5, "K": 64,
         "source": "quadrupole"},
        # the TCC matrix itself, which klitho_tcc reports on
        {"name": "tcc_2048", "kind": "tcc", "Lx": 2048, "Ly": 2048, "source": "annular"},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["forward", "forward", "forward", "mixed", "adjoint", "adjoint", "hopkins", "optics", "tcc"])
    if kind == "mixed":
        return {"kind": kind, "n512": _log_int(rng, 2, 32), "n1024": _log_int(rng, 2, 48), "n2048": _log_int(rng, 1, 16),
                "focus": rng.randint(1, 3), "K": rng.randint(8, 24), "source": rng.choice(["annular", "dipole"]),
                "tuned": rng.random() < 0.5}
    if kind in ("optics", "tcc"):
        L = rng.choice([512, 768, 1024, 1536, 2048, 3072, 4096]) if kind == "optics" else rng.randint(512, 2304)
        source = rng.choice(["annular", "dipole", "quadrupole"])
        if source == "annular" and kind == "optics":
            L = min(L, 1536)
        case = {"kind": kind, "Lx": L, "Ly": L, "source": source}
        if kind == "optics":
            case.update(focus=rng.randint(1, 5) if source != "annular" else 1, K=rng.randint(12, 64 if L > 1024 else 32))
        return case
    # clips of the tuned sizes and arbitrary ones, up to the pixels of the largest listed batch
    if rng.random() < 0.5:
        Lx = Ly = rng.choice([512, 768, 1024, 1536, 2048, 3072])
    else:
        Lx, Ly = _log_int(rng, 400, 3000), _log_int(rng, 400, 3000)
    source = rng.choice(["annular", "dipole", "quadrupole"])
    if kind == "hopkins":
        while Lx * Ly > 1536 * 1536 or max(Lx, Ly) > 2048:
            Lx, Ly = max(400, Lx * 2 // 3), max(400, Ly * 2 // 3)
        return {"kind": kind, "Lx": Lx, "Ly": Ly, "clips": rng.randint(1, 2), "source": source}
    focus = rng.randint(1, 5) if kind == "forward" else 1
    most = max(1, min(64, int(48 * 1024 * 1024 * 2 / (Lx * Ly * focus))))
    case = {"kind": kind, "Lx": Lx, "Ly": Ly, "clips": _log_int(rng, 1, most), "focus": focus,
            "K": rng.randint(8, 48), "source": source}
    if kind == "forward":
        case["tuned"] = rng.random() < 0.3
    return case


# ---------------------------------------------------------------------------
# optics in 64 bits, by the definition
# ---------------------------------------------------------------------------

def _source_map(name, rng=None):
    """Source map (side x side float32, sum 1); `rng` gives every pixel of it an
    intensity of its own (a free-form source), else they are equal."""
    n, a, b = SOURCES[name]
    h = (n - 1) // 2
    y, x = np.mgrid[0:n, 0:n] - h
    if name == "annular":
        d = np.hypot(x, y)
        on = (d >= int(a * h)) & (d <= int(b * h))
    else:
        off, rad = int(a * h), int(b * h)
        poles = [(off, 0), (-off, 0)] + ([(0, off), (0, -off)] if name == "quadrupole" else [])
        on = np.zeros((n, n), dtype=bool)
        for px, py in poles:
            on |= np.hypot(x - px, y - py) <= rad
    w = on.astype(np.float32)
    if rng is not None:
        w *= rng.uniform(0.3, 1.0, size=w.shape).astype(np.float32)
    return (w / w.sum(dtype=np.float64)).astype(np.float32)


def _band(name, Lx, Ly):
    n, a, b = SOURCES[name]
    h = (n - 1) // 2
    y, x = np.nonzero(_source_map(name))
    sigma = np.float32(np.sqrt(((y - h) ** 2 + (x - h) ** 2).max())) / np.float32(h)
    f = lambda L: int(math.floor(np.float32(NA) * np.float32(L) * (np.float32(1) + np.float32(min(sigma, 1))) / np.float32(LAMBDA)))  # noqa: E731
    return f(Lx), f(Ly)


def _factor(src, focus_nm, Lx, Ly, Nx, Ny):
    """A[f, s] = sqrt(J_s) P(f + s) exp(i phase) on the GPU, f over the band, s over the source points."""
    h = (src.shape[0] - 1) // 2
    q, p = np.nonzero(src)
    J = torch.tensor(src[q, p], dtype=torch.float64, device="cuda")
    sx = torch.tensor((p - h) / h, dtype=torch.float64, device="cuda")
    sy = torch.tensor((q - h) / h, dtype=torch.float64, device="cuda")
    fx = torch.arange(-Nx, Nx + 1, dtype=torch.float64, device="cuda") * (LAMBDA / (Lx * NA))
    fy = torch.arange(-Ny, Ny + 1, dtype=torch.float64, device="cuda") * (LAMBDA / (Ly * NA))
    rho2 = (fy[:, None, None] + sy) ** 2 + (fx[None, :, None] + sx) ** 2
    phase = 2 * math.pi / LAMBDA * focus_nm * torch.sqrt((N_WATER ** 2 - rho2 * NA ** 2).clamp_min(0.0))
    A = torch.polar(torch.where(rho2 <= 1, J.sqrt(), 0.0), phase)
    return A.reshape(-1, len(p))


def _top(A, K):
    """Largest K eigenvalues of A A^H and the SOCS kernels that belong to them."""
    w, V = torch.linalg.eigh((A.conj().T @ A).cpu())
    w, V = w.flip(0)[:K], V.flip(1)[:, :K]
    w = w.clamp_min(1e-14 * float(w[0]))  # a small band can have fewer than K modes
    U = A @ V.to(A.device) / torch.sqrt(w).to(A.device)
    return w, U.conj().T.contiguous()


def _focus_values(n):
    return [FOCUS_STEP_NM * (i - n // 2) for i in range(n)]


@functools.lru_cache(maxsize=64)
def _kernels(source, Lx, Ly, focus, K):
    """Kernel sets that a program has from an earlier calculation: (focus, K, N)
    complex64 and (focus, K) float32 on the host, and the band."""
    Nx, Ny = _band(source, Lx, Ly)
    src = _source_map(source)
    sets = [_top(_factor(src, f, Lx, Ly, Nx, Ny), K) for f in _focus_values(focus)]
    return (np.stack([k.to(torch.complex64).cpu().numpy() for _, k in sets]),
            np.stack([w.to(torch.float32).cpu().numpy() for w, _ in sets]), Nx, Ny)


# ---------------------------------------------------------------------------
# masks
# ---------------------------------------------------------------------------

def _rect_masks(n, Lx, Ly, seed):
    """Unions of random rectangles of 40 to 120 nm, 25 to 40 % of the area."""
    rng = np.random.default_rng(seed)
    out = torch.empty((n, Ly, Lx), dtype=torch.float32, device="cuda")
    for i in range(n):
        r = max(1, int(round(-math.log(1 - rng.uniform(0.25, 0.40)) * Lx * Ly / 6400.0)))
        w, h = rng.integers(40, 121, r), rng.integers(40, 121, r)
        x, y = rng.integers(0, Lx - w), rng.integers(0, Ly - h)
        at = np.concatenate([y * (Lx + 1) + x, y * (Lx + 1) + x + w, (y + h) * (Lx + 1) + x, (y + h) * (Lx + 1) + x + w])
        sign = np.repeat(np.array([1, -1, -1, 1], dtype=np.int32), r)
        d = torch.zeros((Ly + 1) * (Lx + 1), dtype=torch.int32, device="cuda")
        d.index_add_(0, torch.from_numpy(at).cuda(), torch.from_numpy(sign).cuda())
        cover = d.view(Ly + 1, Lx + 1).cumsum(0, dtype=torch.int32).cumsum(1, dtype=torch.int32)
        out[i] = (cover[:Ly, :Lx] > 0).float()
    return out


def _smooth_masks(n, Lx, Ly, seed, sigma_px=12.0, gain=6.0):
    """Continuous masks in [0, 1], a mask optimisation's variable: filtered noise through a sigmoid."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    fy = torch.fft.fftfreq(Ly, device="cuda")[:, None]
    fx = torch.fft.rfftfreq(Lx, device="cuda")[None, :]
    filt = torch.exp(-2.0 * (math.pi * sigma_px) ** 2 * (fy ** 2 + fx ** 2))
    out = torch.empty((n, Ly, Lx), dtype=torch.float32, device="cuda")
    for i in range(n):
        z = torch.fft.irfft2(torch.fft.rfft2(torch.randn((Ly, Lx), generator=g, device="cuda")) * filt, s=(Ly, Lx))
        out[i] = torch.sigmoid(gain * z / z.std())
    return out


def _classes(case):
    return [(L, case["n%d" % L]) for L in (512, 1024, 2048)]


def _free_form(case, seed):
    return _source_map(case["source"], np.random.default_rng(seed))


def _defocus_arg(nm):
    return nm * NA * NA / LAMBDA


# ---------------------------------------------------------------------------
# the cases
# ---------------------------------------------------------------------------

def _socs_plan(case, Lx, Ly, clips, adjoint=False):
    import klitho
    krn, scales, Nx, Ny = _kernels(case["source"], Lx, Ly, case["focus"], case["K"])
    plan = klitho.SocsPlan(Lx, Ly, Nx, Ny, case["K"], nsets=case["focus"], max_clips=clips, adjoint=adjoint)
    for i in range(case["focus"]):
        plan.set_kernels(i, krn[i], scales[i])
    return plan


def prepare(case, seed):
    import klitho
    kind = case["kind"]
    new = lambda *shape, dtype=torch.float32: torch.empty(shape, dtype=dtype, device="cuda")  # noqa: E731
    if kind == "mixed":
        plans, masks, images = [], [], []
        for i, (L, n) in enumerate(_classes(case)):
            plans.append(_socs_plan(case, L, L, n))
            masks.append(_rect_masks(n, L, L, seed * 7919 + i))
            images.append(new(n, case["focus"], L, L))
            if case["tuned"]:
                plans[-1].autotune(masks[-1], images[-1])
        return {"kind": kind, "batch": klitho.SocsBatch(plans), "plans": plans, "masks": masks, "images": images}
    Lx, Ly = case["Lx"], case["Ly"]
    state = {"kind": kind, "case": dict(case)}
    if kind == "forward":
        n = case["clips"]
        state.update(plan=_socs_plan(case, Lx, Ly, n), masks=_rect_masks(n, Lx, Ly, seed), images=new(n, case["focus"], Ly, Lx))
        if case["tuned"]:
            state["plan"].autotune(state["masks"], state["images"])
    elif kind == "adjoint":
        n = case["clips"]
        state.update(plan=_socs_plan(case, Lx, Ly, n, adjoint=True), masks=_smooth_masks(n, Lx, Ly, seed),
                     targets=_rect_masks(n, Lx, Ly, seed + 1), grad=new(n, Ly, Lx), images=new(n, 1, Ly, Lx),
                     loss=new(n, dtype=torch.float64))
    elif kind == "hopkins":
        n = case["clips"]
        state.update(tcc=klitho.TccPlan(_source_map(case["source"]), NA, 0.0, Lx, Ly, n_medium=N_WATER),
                     masks=_rect_masks(n, Lx, Ly, seed), images=new(n, Ly, Lx))
    elif kind == "optics":
        Nx, Ny = _band(case["source"], Lx, Ly)
        state.update(source=_free_form(case, seed), masks=_rect_masks(1, Lx, Ly, seed), images=new(1, case["focus"], Ly, Lx),
                     plan=klitho.SocsPlan(Lx, Ly, Nx, Ny, case["K"], nsets=case["focus"], max_clips=1))
    else:
        state.update(source=_free_form(case, seed))
    return state


def run(state):
    import klitho
    kind = state["kind"]
    if kind == "mixed":
        state["batch"].forward(state["masks"], state["images"])
        return state["images"]
    if kind == "forward":
        state["plan"].forward(state["masks"], state["images"])
        return state["images"]
    if kind == "adjoint":
        state["plan"].vjp(state["masks"], state["targets"], state["grad"], state["loss"], state["images"],
                          alpha=ALPHA, threshold=THRESHOLD)
        return {"grad": state["grad"], "loss": state["loss"], "images": state["images"]}
    if kind == "hopkins":
        state["tcc"].hopkins(state["masks"], state["images"])
        return state["images"]
    case = state["case"]
    if kind == "optics":
        tccs = [klitho.TccPlan(state["source"], NA, _defocus_arg(f), case["Lx"], case["Ly"], n_medium=N_WATER)
                for f in _focus_values(case["focus"])]
        if len(tccs) == 1:
            sets = [tccs[0].topk(case["K"])]
        else:
            sets = list(zip(*klitho.TccPlan.topk_batch(tccs, case["K"])))
        for i, (krn, scales, _, _) in enumerate(sets):
            state["plan"].set_kernels(i, krn, scales)
        for t in tccs:
            t.close()
        state["plan"].forward(state["masks"], state["images"])
        return {"eigenvalues": np.stack([s[2] for s in sets]), "images": state["images"]}
    tcc = klitho.TccPlan(state["source"], NA, 0.0, case["Lx"], case["Ly"], n_medium=N_WATER)
    T = tcc.build()
    tcc.close()
    return T


def _points(name):
    return int(np.count_nonzero(_source_map(name)))


def _images_work(Lx, Ly, clips, focus, K, source):
    """Bytes and operations of SOCS images: one mask transform per clip, K
    band-limited fields and one synthesis per image, as fast transforms."""
    Nx, Ny = _band(source, Lx, Ly)
    gx, gy = 4 * Nx + 1, 4 * Ny + 1
    field = 5.0 * gx * math.log2(gx) * (2 * Ny + 1) + 5.0 * gy * math.log2(gy) * gx + 3.0 * gx * gy
    rows = 2.5 * Lx * Ly * math.log2(Lx)
    px = Lx * Ly
    return {"bytes": 4.0 * px * clips * (1 + focus) + 8.0 * focus * K * (2 * Nx + 1) * (2 * Ny + 1),
            "flops": clips * rows + clips * focus * (K * field + rows)}


def work(case):
    kind = case["kind"]
    if kind == "mixed":
        parts = [_images_work(L, L, n, case["focus"], case["K"], case["source"]) for L, n in _classes(case)]
        return {k: sum(p[k] for p in parts) for k in ("bytes", "flops")}
    Lx, Ly, source = case["Lx"], case["Ly"], case["source"]
    if kind == "forward":
        return _images_work(Lx, Ly, case["clips"], case["focus"], case["K"], source)
    if kind == "hopkins":
        return _images_work(Lx, Ly, case["clips"], 1, _points(source), source)
    if kind == "adjoint":
        w = _images_work(Lx, Ly, case["clips"], 1, case["K"], source)
        return {"bytes": w["bytes"] + 8.0 * Lx * Ly * case["clips"], "flops": 3.0 * w["flops"]}
    Nx, Ny = _band(source, Lx, Ly)
    N, S = float((2 * Nx + 1) * (2 * Ny + 1)), float(_points(source))
    if kind == "tcc":
        return {"bytes": 8.0 * N * N, "flops": 8.0 * N * N * S / 2}
    w = _images_work(Lx, Ly, 1, case["focus"], case["K"], source)
    m = min(N, S)
    solve = 8.0 * N * S * S / 2 + 16.0 / 3.0 * m ** 3 + 8.0 * N * S * case["K"]
    return {"bytes": w["bytes"] + case["focus"] * 8.0 * N * case["K"], "flops": w["flops"] + case["focus"] * solve}


def tolerance(case):
    # 32-bit transforms and sums throughout: four times the distance from 64 bits
    # seen over the ranges (images 7e-7, gradients 3e-6: the resist's slope
    # multiplies the image's rounding, TCC entries 4e-6 from 16-bit split products)
    return {"forward": {"rel": 3e-6}, "mixed": {"rel": 3e-6}, "hopkins": {"rel": 3e-6}, "adjoint": {"rel": 1.2e-5},
            "optics": {"rel": 5e-6}, "tcc": {"rel": 1.6e-5}}[case["kind"]]


# ---------------------------------------------------------------------------
# the same in 64 bits
# ---------------------------------------------------------------------------

def _band_index(L, N, device):
    return torch.arange(-N, N + 1, device=device) % L


def _image64(mask, H, scales, Nx, Ny):
    """SOCS image of one clip in 64 bits: fields on the smallest grid that holds
    their squares' band, interpolated to the clip by zero padding."""
    Ly, Lx = mask.shape
    iy, ix = _band_index(Ly, Ny, mask.device), _band_index(Lx, Nx, mask.device)
    M = (torch.fft.fft2(mask) / (Lx * Ly))[iy][:, ix]
    gx, gy = 4 * Nx + 1, 4 * Ny + 1
    jy, jx = _band_index(gy, Ny, mask.device), _band_index(gx, Nx, mask.device)
    I = 0.0
    for k in range(0, H.shape[0], 64):
        F = H[k:k + 64].reshape(-1, 2 * Ny + 1, 2 * Nx + 1) * M
        E = torch.zeros((F.shape[0], gy, gx), dtype=F.dtype, device=F.device)
        E[:, jy[:, None], jx] = F
        E = torch.fft.ifft2(E) * (gx * gy)
        I = I + torch.einsum("k,kyx->yx", scales[k:k + 64], E.real ** 2 + E.imag ** 2)
    T = torch.fft.fft2(I) / (gx * gy)
    ay, ax = _band_index(gy, 2 * Ny, mask.device), _band_index(gx, 2 * Nx, mask.device)
    cy, cx = _band_index(Ly, 2 * Ny, mask.device), _band_index(Lx, 2 * Nx, mask.device)
    full = torch.zeros((Ly, Lx), dtype=T.dtype, device=T.device)
    full = full.index_put((cy[:, None], cx), T[ay][:, ax])
    out = torch.fft.ifft2(full).real * (Lx * Ly)
    return torch.roll(out, (Ly % 2, Lx % 2), (0, 1))  # the centred spectra of odd periods


def _images64(masks, krn, scales, Nx, Ny):
    H = torch.as_tensor(krn).to("cuda", torch.complex128)
    w = torch.as_tensor(scales).to("cuda", torch.float64)
    out = torch.empty((masks.shape[0], H.shape[0]) + masks.shape[1:], dtype=torch.float64, device="cuda")
    for i in range(masks.shape[0]):
        for j in range(H.shape[0]):
            out[i, j] = _image64(masks[i].double(), H[j], w[j], Nx, Ny)
    return out


def exact(case, seed):
    kind = case["kind"]
    if kind == "mixed":
        out = []
        for i, (L, n) in enumerate(_classes(case)):
            krn, scales, Nx, Ny = _kernels(case["source"], L, L, case["focus"], case["K"])
            out.append(_images64(_rect_masks(n, L, L, seed * 7919 + i), krn, scales, Nx, Ny))
        return out
    Lx, Ly = case["Lx"], case["Ly"]
    if kind == "forward":
        return _images64(_rect_masks(case["clips"], Lx, Ly, seed), *_kernels(case["source"], Lx, Ly, case["focus"], case["K"]))
    if kind == "adjoint":
        masks, targets = _smooth_masks(case["clips"], Lx, Ly, seed), _rect_masks(case["clips"], Lx, Ly, seed + 1)
        krn, scales, Nx, Ny = _kernels(case["source"], Lx, Ly, 1, case["K"])
        H = torch.as_tensor(krn[0]).to("cuda", torch.complex128)
        w = torch.as_tensor(scales[0]).to("cuda", torch.float64)
        grads, losses, images = [], [], []
        for m, t in zip(masks, targets):
            m = m.double().requires_grad_()
            image = _image64(m, H, w, Nx, Ny)
            loss = ((torch.sigmoid(ALPHA * (image - THRESHOLD)) - t.double()) ** 2).sum()
            grads.append(torch.autograd.grad(loss, m)[0])
            losses.append(loss.detach())
            images.append(image.detach()[None])
        return {"grad": torch.stack(grads), "loss": torch.stack(losses), "images": torch.stack(images)}
    Nx, Ny = _band(case["source"], Lx, Ly)
    if kind == "hopkins":
        A = _factor(_source_map(case["source"]), 0.0, Lx, Ly, Nx, Ny)
        ones = torch.ones((1, A.shape[1]), dtype=torch.float64)
        return _images64(_rect_masks(case["clips"], Lx, Ly, seed), A.conj().T[None], ones, Nx, Ny)[:, 0]
    src = _free_form(case, seed)
    if kind == "tcc":
        A = _factor(src, 0.0, Lx, Ly, Nx, Ny)
        return torch.view_as_real(A @ A.conj().T)
    sets = [_top(_factor(src, f, Lx, Ly, Nx, Ny), case["K"]) for f in _focus_values(case["focus"])]
    images = [_images64(_rect_masks(1, Lx, Ly, seed), k[None], w[None], Nx, Ny)[0, 0] for w, k in sets]
    return {"eigenvalues": torch.stack([w for w, _ in sets]), "images": torch.stack(images)[None]}
