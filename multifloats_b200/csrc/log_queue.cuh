// Elementwise logarithms with the two branches of the logarithm kept apart.
//
// log2_kernel evaluates arguments in (15/16, 17/16) by one polynomial and all
// others by a table and another one; both cost about 310 FP64 instructions.  A
// warp that holds both kinds runs both, and with arguments drawn evenly from
// [0.5, 2) nearly every warp does.  Here a warp whose lanes disagree puts its
// arguments into two queues of its own in shared memory and works on 32 of one
// kind whenever a queue holds as many; a warp whose lanes agree works on its
// registers.  Every element is evaluated by the same code, so the bits do not
// depend on the order.  2^24 elements (bound: FP64 issue): log on [0.5, 2) 730 ->
// 446 us, ragged 747 -> 487; on arguments of one kind 407 -> 414 (the votes; the
// next argument loaded ahead of the evaluation made it 419 and 475).
#pragma once

#include "dd_device.cuh"

namespace mfcuda {

template <int OP>
constexpr bool log_op = OP == MFCUDA_LOG || OP == MFCUDA_LOG2 || OP == MFCUDA_LOG10;

constexpr int LOG_WARPS = 8;  // 256 threads
struct LogQueue {
  double2 v[LOG_WARPS][2][64];
  double *y[LOG_WARPS][2][64];
};

// Calls load(e, v, y) for e = the elements of this thread in [0, n) (its argument
// and where the result goes), eval on each argument and store(y, r).
template <class Load, class Eval, class Store>
__device__ __forceinline__ void log_map(LogQueue &q, int64_t n, Load load, Eval eval, Store store) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const uint32_t below = (1u << lane) - 1;
  const int64_t stride = (int64_t)gridDim.x * blockDim.x;
  int64_t base = (int64_t)blockIdx.x * blockDim.x + warp * 32;
  int held[2] = {0, 0};  // arguments waiting: table kind, near-one kind
  for (;;) {
    mfdev::dd v = mfdev::make(2.0, 0.0);
    double *y = nullptr;
    int pop = held[0] >= 32 ? 0 : held[1] >= 32 ? 1 : -1;
    if (pop < 0) {
      if (base < n) {
        const bool live = base + lane < n;
        if (live) load(base + lane, v, y);
        base += stride;
        const bool near = v.hi > 15.0 / 16.0 && v.hi < 17.0 / 16.0;
        const uint32_t all = __ballot_sync(~0u, live), ones = __ballot_sync(~0u, live && near);
        if (ones != 0 && ones != all) {
          if (live) {
            const int at = near ? held[1] + __popc(ones & below) : held[0] + __popc(all & ~ones & below);
            q.v[warp][near][at] = make_double2(v.hi, v.lo);
            q.y[warp][near][at] = y;
          }
          held[1] += __popc(ones);
          held[0] += __popc(all & ~ones);
          __syncwarp();
          continue;
        }
      } else {
        pop = held[0] > 0 ? 0 : held[1] > 0 ? 1 : -1;
        if (pop < 0) return;
      }
    }
    if (pop >= 0) {  // the last 32 of a queue, or what is left of it
      const int take = min(32, held[pop]);
      held[pop] -= take;
      if (lane < take) {
        const double2 t = q.v[warp][pop][held[pop] + lane];
        v = mfdev::make(t.x, t.y);
        y = q.y[warp][pop][held[pop] + lane];
      } else if (pop == 1) {
        v = mfdev::make(1.0, 0.0);  // idle lanes take the branch of the others
      }
      __syncwarp();
    }
    const mfdev::dd r = eval(v);
    if (y) store(y, r);
  }
}

}  // namespace mfcuda
