// dg_frame.cuh -- the persistent frame kernel and its instantiation picker.
//
// frame_kernel<shape, interp, defgrad, mask> runs Schema::execute_correlation
// (or one Objective entry point, by mode) for every subset of a launch: one
// CTA per subset, handed out in order.  The instantiations
// live in frame_inst.cu (one unit per shape function, interpolation and
// mask); the unmasked kernels are exactly what they are without masks.
#pragma once

#include "dg_engine.cuh"

// launch bounds of the frame kernel: at most DG_MAX_THREADS threads per CTA
// (warps per subset <= DG_MAX_THREADS / 32) and DG_MIN_BLOCKS resident CTAs
// of that size per SM, which bounds its registers
#ifndef DG_MAX_THREADS
#define DG_MAX_THREADS 256
#endif
#ifndef DG_MIN_BLOCKS
#define DG_MIN_BLOCKS 2
#endif

namespace dg {

// ---------------------------------------------------------------------------
// the persistent frame kernel: one CTA (up to 8 warps) per subset
// ---------------------------------------------------------------------------
template <int SHAPE, int INTERP, bool DEFGRAD, bool MASK>
__global__ void __launch_bounds__(DG_MAX_THREADS, DG_MIN_BLOCKS) frame_kernel(const __grid_constant__ FrameArgs a) {
  Engine<SHAPE, INTERP, DEFGRAD, MASK> e(a);
  Ctl& c = ctl();
  if (a.plain_index >= 0) {
    if (blockIdx.x == 0) e.run(a.plain_index);
    return;
  }
  // the launch's subsets: all n, or the n_order listed in order
  const int count = a.order ? a.n_order : a.n;
  // The launch's subsets are handed out in order: the first gridDim.x to the
  // CTAs by number, the others from one counter, so that all CTAs advance
  // through the image together (a narrow band resident in L2) and a CTA that
  // finds the counter past the end is done.  Every subset is taken exactly
  // once and no CTA ever waits on another.  (With a queue per CTA and stealing,
  // a CTA had to find every one of the 296 or 592 queues empty before it could
  // leave: about 90 us at the end of every launch, most of a tracking wave's
  // time.  Handing out four neighbours at a time gained nothing: 53.5 against
  // 53.0 ms on the 158,404-subset frame.)
  for (int t = blockIdx.x; t < count;) {
    DG_PT(t_run);
    e.run(a.order ? a.order[t] : t);
    DG_PACC(0, t_run);
    if (count <= gridDim.x) return;
    __syncthreads();
    if (threadIdx.x == 0) c.work = gridDim.x + atomicAdd(a.work_counter, 1);
    __syncthreads();
    t = c.work;
    __syncthreads();
  }
}

typedef void (*FrameKernelFn)(FrameArgs);

// The frame kernels are instantiated in frame_inst.cu, compiled once per
// (shape function, interpolation, mask) so that the units build in
// parallel: frame_fn_s<shape>_i<interp>_m<mask>(defgrad) returns the kernel
// with or without deformed-image gradients.  MASK selects the instantiation
// whose passes test obstruction bitmaps and blocked polygons (only contexts
// with masks launch it).
#define DG_FRAME_FN_NAME(S, I, M) frame_fn_s##S##_i##I##_m##M
#define DG_DECLARE_FRAME_FN(S, I, M) FrameKernelFn DG_FRAME_FN_NAME(S, I, M)(bool defgrad);
DG_DECLARE_FRAME_FN(0, 0, 0) DG_DECLARE_FRAME_FN(0, 1, 0) DG_DECLARE_FRAME_FN(0, 2, 0)
DG_DECLARE_FRAME_FN(1, 0, 0) DG_DECLARE_FRAME_FN(1, 1, 0) DG_DECLARE_FRAME_FN(1, 2, 0)
DG_DECLARE_FRAME_FN(2, 0, 0) DG_DECLARE_FRAME_FN(2, 1, 0) DG_DECLARE_FRAME_FN(2, 2, 0)
DG_DECLARE_FRAME_FN(0, 0, 1) DG_DECLARE_FRAME_FN(0, 1, 1) DG_DECLARE_FRAME_FN(0, 2, 1)
DG_DECLARE_FRAME_FN(1, 0, 1) DG_DECLARE_FRAME_FN(1, 1, 1) DG_DECLARE_FRAME_FN(1, 2, 1)

#ifdef DG_PROFILE
// profiling builds: each unit adds its section timers into acc16 and clears them
#define DG_FRAME_PROF_NAME(S, I, M) frame_prof_s##S##_i##I##_m##M
#define DG_DECLARE_FRAME_PROF(S, I, M) int DG_FRAME_PROF_NAME(S, I, M)(unsigned long long* acc16);
DG_DECLARE_FRAME_PROF(0, 0, 0) DG_DECLARE_FRAME_PROF(0, 1, 0) DG_DECLARE_FRAME_PROF(0, 2, 0)
DG_DECLARE_FRAME_PROF(1, 0, 0) DG_DECLARE_FRAME_PROF(1, 1, 0) DG_DECLARE_FRAME_PROF(1, 2, 0)
DG_DECLARE_FRAME_PROF(2, 0, 0) DG_DECLARE_FRAME_PROF(2, 1, 0) DG_DECLARE_FRAME_PROF(2, 2, 0)
DG_DECLARE_FRAME_PROF(0, 0, 1) DG_DECLARE_FRAME_PROF(0, 1, 1) DG_DECLARE_FRAME_PROF(0, 2, 1)
DG_DECLARE_FRAME_PROF(1, 0, 1) DG_DECLARE_FRAME_PROF(1, 1, 1) DG_DECLARE_FRAME_PROF(1, 2, 1)
#endif

// The frame kernel of a configuration (nullptr for one this build leaves
// out: a unit compiled with DG_ONLY_BENCH_KERNEL returns only the affine /
// Keys-4 / deformed-gradient kernel).
inline FrameKernelFn pick_frame_kernel(int shape, int interp, bool defgrad, bool mask) {
  typedef FrameKernelFn (*Pick)(bool);
  static const Pick table[3][3][2] = {
      {{DG_FRAME_FN_NAME(0, 0, 0), DG_FRAME_FN_NAME(0, 0, 1)},
       {DG_FRAME_FN_NAME(0, 1, 0), DG_FRAME_FN_NAME(0, 1, 1)},
       {DG_FRAME_FN_NAME(0, 2, 0), DG_FRAME_FN_NAME(0, 2, 1)}},
      {{DG_FRAME_FN_NAME(1, 0, 0), DG_FRAME_FN_NAME(1, 0, 1)},
       {DG_FRAME_FN_NAME(1, 1, 0), DG_FRAME_FN_NAME(1, 1, 1)},
       {DG_FRAME_FN_NAME(1, 2, 0), DG_FRAME_FN_NAME(1, 2, 1)}},
      {{DG_FRAME_FN_NAME(2, 0, 0), nullptr}, {DG_FRAME_FN_NAME(2, 1, 0), nullptr}, {DG_FRAME_FN_NAME(2, 2, 0), nullptr}}};
  if (shape < 0 || shape > 2 || (shape == kAffineLean && mask) || interp < 0 || interp > 2) return nullptr;
  return table[shape][interp][mask ? 1 : 0](defgrad);
}

}  // namespace dg
