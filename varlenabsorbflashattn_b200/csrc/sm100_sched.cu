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

__global__ void __launch_bounds__(256) cu_check_kernel(const SchedParams p) { sched_impl::cu_check(p); }

void set_check(SchedParams& p, const CuCheck& check) {
  p.verdict = check.verdict;
  p.check_q = check.total_q; p.check_k = check.total_k; p.need_keys = check.need_keys;
}

}  // namespace

int launch_cu_check(const int32_t* cu_q, const int32_t* cu_k, int n_seg, cudaStream_t s, CuCheck* check) {
  SchedParams p{};
  p.cu_q = cu_q; p.cu_k = cu_k; p.n_seg = n_seg;
  set_check(p, *check);
  LaunchScope scope(kKSched, s);
  cu_check_kernel<<<1, 256, 0, s>>>(p);
  VAFA_LAUNCH_CHECK("cu_check_kernel");
  check->queued = true;
  VAFA_CUDA_CHECK(cudaEventRecord(check->done, s));
  return 0;
}

int launch_scheduler(const SchedParams& params, cudaStream_t s, CuCheck* check) {
  SchedParams p = params;
  if (check != nullptr) set_check(p, *check);
  LaunchScope scope(kKSched, s);
  sched_kernel<<<1, sched_impl::kSchedThreads, 0, s>>>(p);
  VAFA_LAUNCH_CHECK("sched_kernel");
  if (check != nullptr) {
    check->queued = true;
    VAFA_CUDA_CHECK(cudaEventRecord(check->done, s));
  }
  return 0;
}

int launch_scheduler_three(const SchedParams& a, const SchedParams& b, const SchedParams& c, cudaStream_t s) {
  LaunchScope scope(kKSched, s);
  sched_three_kernel<<<3, sched_impl::kSchedThreads, 0, s>>>(SchedLists{{a, b, c}});
  VAFA_LAUNCH_CHECK("sched_kernel");
  return 0;
}

}  // namespace vafa
