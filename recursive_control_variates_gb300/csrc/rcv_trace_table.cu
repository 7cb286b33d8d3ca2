// Tracer kernels of job tables (the batched engine): the two-state pass, the
// radiance passes of both adjoints and the replay, under the constant
// environment.
#include "rcv_trace_kernels.cuh"

namespace rcv {

#define RCV_TABLE_TRACERS(SG, COUNT)                                                              \
  {trace_kernel<kTwoState, SG, COUNT, false, true>, nullptr,                                      \
   trace_kernel<kAdjoint, SG, COUNT, false, true>,  trace_kernel<kReplay, SG, COUNT, false, true>, \
   nullptr,                                         trace_kernel<kTape, SG, COUNT, false, true>}

const TraceKernel kJobTableTracers[4][kTraceModes] = {RCV_TABLE_TRACERS(false, false), RCV_TABLE_TRACERS(true, false),
                                                      RCV_TABLE_TRACERS(false, true), RCV_TABLE_TRACERS(true, true)};

#undef RCV_TABLE_TRACERS

}  // namespace rcv
