// Single-CTA scheduler kernel: see sm100_sched.cuh and sm100_sched_body.cuh.
#include "sm100_sched_body.cuh"
#include "profile.cuh"

namespace vafa {
namespace {

// One CTA per tile list: blockIdx.x picks the parameter set.
struct SchedLists {
  SchedParams p[3];
};
__global__ void __launch_bounds__(sched_impl::kSchedThreads) sched_kernel(const SchedParams p) { sched_impl::sched_build(p); }
__global__ void __launch_bounds__(sched_impl::kSchedThreads) sched_three_kernel(const SchedLists l) {
  if (blockIdx.x == 0) sched_impl::sched_build(l.p[0]);
  else if (blockIdx.x == 1) sched_impl::sched_build(l.p[1]);
  else sched_impl::sched_build(l.p[2]);
}

}  // namespace

int launch_scheduler(const SchedParams& p, cudaStream_t s) {
  LaunchScope scope(kKSched, s);
  sched_kernel<<<1, sched_impl::kSchedThreads, 0, s>>>(p);
  VAFA_LAUNCH_CHECK("sched_kernel");
  return 0;
}

int launch_scheduler_three(const SchedParams& a, const SchedParams& b, const SchedParams& c, cudaStream_t s) {
  LaunchScope scope(kKSched, s);
  sched_three_kernel<<<3, sched_impl::kSchedThreads, 0, s>>>(SchedLists{{a, b, c}});
  VAFA_LAUNCH_CHECK("sched_kernel");
  return 0;
}

}  // namespace vafa
