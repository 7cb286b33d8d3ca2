// The tracer kernel and its function-pointer tables, instantiated for single
// jobs in rcv_volume.cu and for job tables in rcv_trace_table.cu (two files so
// that they compile side by side).
#pragma once
#include "rcv_trace.cuh"

namespace rcv {

__device__ __forceinline__ void add_counts(unsigned long long* counters, const Counts& c) {
  if (counters == nullptr) return;
  const unsigned p = __reduce_add_sync(0xffffffffu, c.paths);
  const unsigned l = __reduce_add_sync(0xffffffffu, c.lookups);
  const unsigned n = __reduce_add_sync(0xffffffffu, c.nee_lookups);
  const unsigned s = __reduce_add_sync(0xffffffffu, c.scatters);
  const unsigned ge = __reduce_add_sync(0xffffffffu, c.grad_events);
  const unsigned ae = __reduce_add_sync(0xffffffffu, c.albedo_events);
  if ((threadIdx.x & 31) == 0) {
    atomicAdd(counters + RCV_COUNTER_PATHS, (unsigned long long)p);
    atomicAdd(counters + RCV_COUNTER_LOOKUPS, (unsigned long long)l);
    atomicAdd(counters + RCV_COUNTER_NEE_LOOKUPS, (unsigned long long)n);
    atomicAdd(counters + RCV_COUNTER_SCATTERS, (unsigned long long)s);
    if (ge) atomicAdd(counters + RCV_COUNTER_GRAD_EVENTS, (unsigned long long)ge);
    if (ae) atomicAdd(counters + RCV_COUNTER_ALBEDO_EVENTS, (unsigned long long)ae);
  }
}

// Resident blocks per SM that a tracer's registers are bounded for.  More
// warps hide more of the walk's latency but slow each of the longest paths, on
// which a launch ends: the single-state tracer of target renders 8 (64
// registers; 512^2 x 256 spp 7.80 ms, 9 blocks 7.85; with one step per iteration 5 /
// 6 / 7 / 8 / 9 blocks were 17.3 / 16.6 / 15.5 / 14.8 / 14.5 ms); the other primal
// passes alone end on their tails from 7 on (three map-lit DRT views 1.818 ms at
// 6, 1.837 at 7); the replays spill below 96 registers.
constexpr int tracer_blocks(int mode) {
  return mode == kSingle ? 8 : (mode == kReplay || mode == kForward ? 5 : 6);
}

template <int kMode, bool kSG, bool kCount, bool kEnv, bool kTable>
__global__ void __launch_bounds__(kTraceBlock, tracer_blocks(kMode)) trace_kernel(const __grid_constant__ VolJob J,
                                                            const __grid_constant__ Queue Q) {
  Counts cnt{0, 0, 0, 0, 0, 0};
  trace_persistent<kMode, kSG, kCount, kEnv, kTable>(J, Q, cnt);
  if (kCount) add_counts(Q.counters, cnt);
}

using TraceKernel = void (*)(VolJob, Queue);
// Job-table tracers by supergrid + 2 * counting, then by mode (null: a mode
// that the batched engine does not run).
extern const TraceKernel kJobTableTracers[4][kTraceModes];

}  // namespace rcv
