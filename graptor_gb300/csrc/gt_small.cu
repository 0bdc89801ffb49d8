// The iteration of a small problem in two launches (sm_103a).
//
// Below about a million voxel-channels the iteration's five launches (dual update, forward
// projection, back projection, the two halves of the primal update) are bound by launches and
// by each kernel's latency, not by memory or arithmetic.  What does not depend on each other
// shares a launch, and the back projection goes straight into the update that needs it:
//
//   k_fwd_dual   blocks [0, nf): forward projection + data dual (reads ubar, f, lambda; writes
//                lambda, K u); the others: dual update (reads ubar, pbar, v, w; writes v, w)
//   k_bp_update  blocks [0, nb): back projection of a pixel's slices and, with K* lambda in
//                registers, their u / ubar update (reads lambda, v, u; writes u, ubar); the
//                others: the p / pbar half (reads v, w, p; writes p, pbar)
//
// Every value is computed by the kernels' own device code (gt_flat.cuh, gt_dual.cuh,
// gt_update.cuh), so the iterates are identical.  K* lambda is not written.
//
// Per iteration, three problems side by side, separate launches -> this form: 128^2 x 1
// slice, 60 angles 10.2 -> 8.1 us; 64^2 x 32, 71 angles 16.9 -> 13.7 us; 101^2 x 40, 33 angles
// 33.3 -> 32.1 us.  With 64 slices and more the register-blocked projectors, which have no
// two-launch form, win at 128^2; the autotuner times both forms (below 8M voxel-channels).
#include <cuda_runtime.h>

#include "gt_common.cuh"
#include "gt_dual.cuh"
#include "gt_flat.cuh"
#include "gt_update.cuh"

namespace gt {

namespace {

inline unsigned blocks(long long threads, int bs) { return (unsigned)((threads + bs - 1) / bs); }

// VW = 8: the flat forms, four slices per thread; VW = 1, 2, 4: the staged forms (S = VW)
constexpr int SMALL_NT = 128;
constexpr int STAGED_NT = 256;

template <int DIM, bool TGV, int CPL, int CMAX, int VW>
__global__ void __launch_bounds__(VW == 8 ? SMALL_NT : STAGED_NT) k_fwd_dual(const IterParams P, int disc, unsigned nf) {
  if (blockIdx.x >= nf) {
    dual_body<DIM, TGV, CPL, CMAX>(P, blockIdx.x - nf);
  } else if constexpr (VW == 8) {
    fwd_flat_body<4, 12>(P, disc, (long long)blockIdx.x * SMALL_NT + threadIdx.x);
  } else {
    __shared__ FwdStage<VW> sh;
    fwd_staged_body<VW>(P, disc, blockIdx.x, sh);
  }
}

template <int DIM, bool TGV, int VW>
__global__ void __launch_bounds__(SMALL_NT) k_bp_update(const IterParams P, unsigned nb) {
  constexpr int UW = VW == 8 ? 4 : VW;
  if (blockIdx.x >= nb) {
    update_body<DIM, TGV, UW, PART_P>(P, blockIdx.x - nb);
    return;
  }
  int pix, s0 = 0;
  float ks[UW];
  if constexpr (VW == 8) {
    if (!bp_flat_body<4, 8>(P, (long long)blockIdx.x * SMALL_NT + threadIdx.x, pix, s0, ks)) return;
  } else {
    __shared__ BpStage<VW> sh[SMALL_NT / 32];
    const int warp = threadIdx.x >> 5;
    if (!bp_staged_body<VW>(P, (long long)blockIdx.x * (SMALL_NT / 32) + warp, sh[warp], pix, ks)) return;
  }
  const int y = pix / P.d.N;
  primal_update<DIM, TGV, UW, PART_U>(P, pix - y * P.d.N, y, s0, ks);
}

template <int DIM, bool TGV, int CPL, int CMAX>
void fwd_dual(const IterParams &P, int disc, cudaStream_t st) {
  const Dims &d = P.d;
  const long long rays = (long long)d.nd * d.nang;
  const int nt = d.S <= 4 ? STAGED_NT : SMALL_NT;
  const unsigned nf = d.S <= 4 ? blocks(rays, FS_RAYS) : blocks(rays * (d.S / 4), SMALL_NT);
  const unsigned g = nf + blocks((long long)P.npix * d.Nz, nt);
  if (d.S == 1) k_fwd_dual<DIM, TGV, CPL, CMAX, 1><<<g, nt, 0, st>>>(P, disc, nf);
  else if (d.S == 2) k_fwd_dual<DIM, TGV, CPL, CMAX, 2><<<g, nt, 0, st>>>(P, disc, nf);
  else if (d.S == 4) k_fwd_dual<DIM, TGV, CPL, CMAX, 4><<<g, nt, 0, st>>>(P, disc, nf);
  else k_fwd_dual<DIM, TGV, CPL, CMAX, 8><<<g, nt, 0, st>>>(P, disc, nf);
}

template <int DIM, bool TGV>
void fwd_dual_c(const IterParams &P, int disc, int cpl, cudaStream_t st) {
  if (P.d.C == 1 && cpl == FROB) fwd_dual<DIM, TGV, FROB, 1>(P, disc, st);
  else if (P.d.C == 1) fwd_dual<DIM, TGV, UNCORR, 1>(P, disc, st);
  else if (cpl == FROB) fwd_dual<DIM, TGV, FROB, 4>(P, disc, st);
  else fwd_dual<DIM, TGV, UNCORR, 4>(P, disc, st);
}

template <int DIM, bool TGV, int VW>
void bp_update(const IterParams &P, cudaStream_t st) {
  const unsigned np = blocks((long long)P.npix * (P.d.S / (VW == 8 ? 4 : VW)), SMALL_NT);
  const unsigned nb = VW == 8 ? np : blocks(P.npix, BS_PIX * SMALL_NT / 32);
  k_bp_update<DIM, TGV, VW><<<TGV ? nb + np : nb, SMALL_NT, 0, st>>>(P, nb);
}

template <int DIM, bool TGV>
void bp_update_s(const IterParams &P, cudaStream_t st) {
  if (P.d.S == 1) bp_update<DIM, TGV, 1>(P, st);
  else if (P.d.S == 2) bp_update<DIM, TGV, 2>(P, st);
  else if (P.d.S == 4) bp_update<DIM, TGV, 4>(P, st);
  else bp_update<DIM, TGV, 8>(P, st);
}

}  // namespace

bool small_ok(const IterParams &P, int cpl) {
  return cpl != NUCL && P.d.C <= 4 && (P.d.S % 4 == 0 || P.d.S <= 2) && P.ray_start;
}

cudaError_t launch_small(const IterParams &P, int disc, int tgv, int cpl, cudaStream_t st) {
  if (P.d.dim == 3) {
    if (tgv) fwd_dual_c<3, true>(P, disc, cpl, st); else fwd_dual_c<3, false>(P, disc, cpl, st);
  } else {
    if (tgv) fwd_dual_c<2, true>(P, disc, cpl, st); else fwd_dual_c<2, false>(P, disc, cpl, st);
  }
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return e;
  if (P.d.dim == 3) {
    if (tgv) bp_update_s<3, true>(P, st); else bp_update_s<3, false>(P, st);
  } else {
    if (tgv) bp_update_s<2, true>(P, st); else bp_update_s<2, false>(P, st);
  }
  return cudaGetLastError();
}

}  // namespace gt
