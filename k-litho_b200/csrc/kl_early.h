// kl_early.h -- switch of kl_launch.cuh.
#pragma once

namespace kl {
// whether this thread's launches may start ahead: not while stage events are
// recorded between the kernels, in concurrent branches, or where tables and kernels
// are not a plan's
inline thread_local bool t_early_launch = true;
// sets it for a scope; a scope inside one that turned it off cannot turn it on
struct EarlyLaunch {
  const bool before = t_early_launch;
  explicit EarlyLaunch(bool on) { t_early_launch = before && on; }
  ~EarlyLaunch() { t_early_launch = before; }
};
}  // namespace kl
