// Dispatch of the fused step over compile-time row lengths (each instantiation makes every thermal population
// offset an immediate). Included once per storage mode (fluid storage SP, thermal storage SQ) by step_f32.cu /
// step_f16.cu / step_bf16.cu / step_f32t16.cu, which compile in parallel.
#pragma once

#include "lattice_kernels.cuh"

namespace xac {

template <typename SP, typename SQ, bool kMacro, bool kOwn>
void launch_staged_rows(const StepLaunch& a) {
  // one block per row; the kernel's compile-time row length is its block size
#define XAC_QSTAGE(KT)                                                                                             \
  coupled_qstage_kernel<SP, SQ, kMacro, kOwn, KT><<<(unsigned)a.p.g.rows, KT, StageQ<SQ, KT>::kLen * sizeof(SQ), \
                                                   a.stream>>>(                                                   \
      (const SP*)a.Pin, (SP*)a.Pout, (const SQ*)a.Qin, (SQ*)a.Qout, a.link, a.qsrc, a.u_in, a.rho, a.ux, a.uy,     \
      a.uz, a.T0, a.p)
  switch (a.p.g.pitch) {
    case 32: XAC_QSTAGE(32); return;
    case 64: XAC_QSTAGE(64); return;
    case 96: XAC_QSTAGE(96); return;
    case 128: XAC_QSTAGE(128); return;
    case 160: XAC_QSTAGE(160); return;
    case 192: XAC_QSTAGE(192); return;
    case 224: XAC_QSTAGE(224); return;
    case 256: XAC_QSTAGE(256); return;
    case 288: XAC_QSTAGE(288); return;
    case 320: XAC_QSTAGE(320); return;
    default: return;
  }
#undef XAC_QSTAGE
}

template <typename SP, typename SQ>
void launch_staged_step(const StepLaunch& a) {
  if (a.macro && a.own) launch_staged_rows<SP, SQ, true, true>(a);
  else if (a.macro) launch_staged_rows<SP, SQ, true, false>(a);
  else if (a.own) launch_staged_rows<SP, SQ, false, true>(a);
  else launch_staged_rows<SP, SQ, false, false>(a);
}

template <typename SP, typename SQ, bool kMacro, bool kOwn>
void launch_rows(const StepLaunch& a) {
  const unsigned grid = (unsigned)(((long long)a.p.g.rows * a.p.g.pitch + a.block - 1) / a.block);
#define XAC_STEP(KT)                                                                                             \
  coupled_step_kernel<SP, SQ, kMacro, kOwn, KT><<<grid, a.block, 0, a.stream>>>(                                  \
      (const SP*)a.Pin, (SP*)a.Pout, (const SQ*)a.Qin, (SQ*)a.Qout, a.link, a.qsrc, a.u_in, a.rho, a.ux, a.uy,    \
      a.uz, a.T0, a.p)
  switch (a.p.g.pitch) {
    case 32: XAC_STEP(32); return;
    case 64: XAC_STEP(64); return;
    case 96: XAC_STEP(96); return;
    case 128: XAC_STEP(128); return;
    case 160: XAC_STEP(160); return;
    case 192: XAC_STEP(192); return;
    case 224: XAC_STEP(224); return;
    case 256: XAC_STEP(256); return;
    default: XAC_STEP(0);
  }
#undef XAC_STEP
}

template <typename SP, typename SQ>
void launch_row_step(const StepLaunch& a) {
  if (a.macro && a.own) launch_rows<SP, SQ, true, true>(a);
  else if (a.macro) launch_rows<SP, SQ, true, false>(a);
  else if (a.own) launch_rows<SP, SQ, false, true>(a);
  else launch_rows<SP, SQ, false, false>(a);
}

template <typename SP>
void launch_split_fluid(const SplitArgs& a, int block, bool plain, cudaStream_t s) {
  const unsigned grid = a.fblocks + a.eblocks;
  if (plain) split_fluid_kernel<SP, true><<<grid, block, 0, s>>>(a);
  else split_fluid_kernel<SP, false><<<grid, block, 0, s>>>(a);
}

template <typename SQ, bool kPlain>
void launch_split_rows(const SplitArgs& a, int block, cudaStream_t s) {
#define XAC_SPLIT(KT) split_thermal_kernel<SQ, kPlain, KT><<<a.tblocks, block, 0, s>>>(a)
  switch (a.p.g.pitch) {
    case 32: XAC_SPLIT(32); break;
    case 64: XAC_SPLIT(64); break;
    case 96: XAC_SPLIT(96); break;
    case 128: XAC_SPLIT(128); break;
    case 160: XAC_SPLIT(160); break;
    case 192: XAC_SPLIT(192); break;
    case 224: XAC_SPLIT(224); break;
    case 256: XAC_SPLIT(256); break;
    case 288: XAC_SPLIT(288); break;
    case 320: XAC_SPLIT(320); break;
    default: XAC_SPLIT(0);
  }
#undef XAC_SPLIT
}

template <typename SQ>
void launch_split_thermal(const SplitArgs& a, int block, bool plain, cudaStream_t s) {
  if (plain) launch_split_rows<SQ, true>(a, block, s);
  else launch_split_rows<SQ, false>(a, block, s);
}

}  // namespace xac
