"""Host code of the library without a GPU: C++ programs under tests/harness link one of
its sources against a CUDA runtime of host memory and check what calls do where a test
on a GPU cannot (several devices, failing solves)."""
import os
import subprocess

import pytest

REPO = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(REPO, "k-litho_b200", "csrc")
HARNESS = os.path.join(REPO, "tests", "harness")


@pytest.mark.parametrize("program,source", [("upload_device", "kl_socs_api.cpp"), ("topk_outputs", "kl_tcc_api.cpp"),
                                            ("autotune_slices", "kl_socs_batch.cpp")])
def test_host_path(tmp_path, program, source):
    exe = str(tmp_path / program)
    cuda = os.environ.get("CUDA_HOME", "/usr/local/cuda")
    subprocess.run(["g++", "-O1", "-std=c++17", "-no-pie", "-I", CSRC, "-I", os.path.join(REPO, "include"),
                    "-I", os.path.join(cuda, "include"), os.path.join(HARNESS, program + ".cpp"), os.path.join(CSRC, source),
                    "-Wl,-z,lazy", "-Wl,--unresolved-symbols=ignore-all", "-o", exe], check=True)
    r = subprocess.run([exe], stdout=subprocess.PIPE, timeout=60, text=True)
    assert r.returncode == 0, r.stdout
