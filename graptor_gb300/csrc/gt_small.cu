// The iteration of a problem of 1, 2 or 4 slices in two launches (sm_103a).
//
// There the iteration's five launches (dual update, forward projection, back projection, the
// two halves of the primal update) are bound by launches and by each kernel's latency, not by
// memory or arithmetic.  What does not depend on each other shares a launch, and the back
// projection goes straight into the update that needs it:
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
// 128^2 x 1 slice, 60 angles, per iteration: alone 15.3 us with separate launches, 13.9 us in
// this form; three problems at once (as slices and batches of small problems are solved) 10.2 ->
// 7.6 us.  With more slices separate launches win there: a launch's blocks all hold the
// registers of its larger half (64^2 x 32, three problems at once: 11.9 us an iteration with
// separate launches, 13.4 us in this form).  The tuner times a problem alone.
#include <cuda_runtime.h>

#include "gt_common.cuh"
#include "gt_dual.cuh"
#include "gt_flat.cuh"
#include "gt_update.cuh"

namespace gt {

namespace {

inline unsigned blocks(long long threads, int bs) { return (unsigned)((threads + bs - 1) / bs); }

constexpr int FWD_NT = 256, BP_NT = 128;  // S = VW slices

template <int DIM, bool TGV, int CPL, int CMAX, int VW>
__global__ void __launch_bounds__(FWD_NT, 1) k_fwd_dual(const IterParams P, int disc, unsigned nf) {
  if (blockIdx.x >= nf) {
    dual_body<DIM, TGV, CPL, CMAX>(P, blockIdx.x - nf);
  } else {
    __shared__ FwdStage<VW> sh;
    fwd_staged_body<VW>(P, disc, blockIdx.x, sh);
  }
}

template <int DIM, bool TGV, int VW>
__global__ void __launch_bounds__(BP_NT, 1) k_bp_update(const IterParams P, unsigned nb) {
  if (blockIdx.x >= nb) {
    update_body<DIM, TGV, VW, PART_P>(P, blockIdx.x - nb);
    return;
  }
  __shared__ BpStage<VW> sh[BP_NT / 32];
  const int warp = threadIdx.x >> 5;
  int pix;
  float ks[VW];
  if (!bp_staged_body<VW>(P, (long long)blockIdx.x * (BP_NT / 32) + warp, sh[warp], pix, ks)) return;
  const int y = pix / P.d.N;
  primal_update<DIM, TGV, VW, PART_U>(P, pix - y * P.d.N, y, 0, ks);
}

template <int DIM, bool TGV, int CPL, int CMAX>
void fwd_dual(const IterParams &P, int disc, cudaStream_t st) {
  const Dims &d = P.d;
  const long long rays = (long long)d.nd * d.nang;
  const unsigned nf = blocks(rays, FS_RAYS), g = nf + blocks((long long)P.npix * d.Nz, FWD_NT);
  if (d.S == 1) k_fwd_dual<DIM, TGV, CPL, CMAX, 1><<<g, FWD_NT, 0, st>>>(P, disc, nf);
  else if (d.S == 2) k_fwd_dual<DIM, TGV, CPL, CMAX, 2><<<g, FWD_NT, 0, st>>>(P, disc, nf);
  else k_fwd_dual<DIM, TGV, CPL, CMAX, 4><<<g, FWD_NT, 0, st>>>(P, disc, nf);
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
  const unsigned nb = blocks(P.npix, BS_PIX * BP_NT / 32);
  k_bp_update<DIM, TGV, VW><<<TGV ? nb + blocks(P.npix, BP_NT) : nb, BP_NT, 0, st>>>(P, nb);
}

template <int DIM, bool TGV>
void bp_update_s(const IterParams &P, cudaStream_t st) {
  if (P.d.S == 1) bp_update<DIM, TGV, 1>(P, st);
  else if (P.d.S == 2) bp_update<DIM, TGV, 2>(P, st);
  else bp_update<DIM, TGV, 4>(P, st);
}

}  // namespace

bool small_ok(const IterParams &P, int cpl) {
  return cpl != NUCL && (P.d.S <= 2 || P.d.S == 4) && P.d.C <= 4;
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
