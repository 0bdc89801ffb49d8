// Register-blocked back projector of the solver iteration (sm_103a): back projection
// `radon_ad`, radon_tgv_primal_dual_3d.py:818-844.
//
// What bounds it: every (pixel, angle) pair reads two detector taps of S slice values, and
// the loads' way back to the registers (128 bytes a clock and SM, broadcasts included)
// is the limit, then instruction issue.  So a loaded tap is shared between pixels, the
// geometry is kept as small as it can be, and the multiply-adds are done two at a time
// (fma.rn.f32x2, each half rounding as a scalar one).
//
// k_bp_tap: a warp owns 4 adjacent pixels of a row and 32 VW slices.  Along a row the
// detector coordinate moves by |cos| <= 1 per pixel, so the pixels' lower bins step by 0 or
// 1 -- one of 8 patterns per direction -- and their taps lie on 2 to 5 consecutive bins,
// each loaded once.  Which accumulator a product goes to must be known at compile time
// (registers cannot be indexed at run time), so the kernel branches once per angle on
// the pattern and loads exactly the bins it needs.  A table of 20 bytes per (row tile,
// angle) holds the first bin with the pattern and the 4 interpolation fractions; the lower
// weight 1 - p is recomputed.  A first form with both weights and a three-word header
// (48 bytes, three 16-byte broadcasts against five taps at 4 slices per lane) took
// 328 us on 256^2 x 60 x 4, 71 angles and 3635 us on 512^2 x 96 x 4, 141 angles; this one
// takes 213 us (8 slices per lane; 59 % of the write-back path busy, half of the issue
// slots) and 2628 us (4 per lane).
//
// k_bp_flat: a thread owns one pixel and VW slices, threads of a warp run on over pixels.
// With few slices per pixel a warp per tile leaves lanes idle; here a warp holds
// several pixels and the geometry is computed on the fly, UA angles at a time so that
// 2 UA loads are in flight.  64^2, 71 angles, 32 slices: 12.3 us (26.7 with one slice per thread,
// 25.9 with the loads one after another); 177^2, 45 angles, 16 slices: 14.4 us (37, 20.5).
//
// k_bp_staged: one, two or four slices; a warp computes the geometry and loads the taps of
// 8 pixels and 32 angles at once into shared memory, 8 lanes add them in order (a thread per
// pixel leaves the chain of its angles bare).  128^2 x 1, 60 angles, in the two-launch iteration:
// 22.1 us an iteration with a thread per pixel, 14.9 us; as a kernel of its own both take 10 us.
//
// Every pixel adds its taps in the reference's order (angles ascending, lower tap then
// upper tap) with the reference's weights, so all shapes give identical iterates.
#include <cuda_runtime.h>

#include "gt_common.cuh"
#include "gt_flat.cuh"
#include "gt_geom.cuh"
#include "gt_vec.cuh"

namespace gt {

namespace {

constexpr int ROW_P = 4;  // pixels per row tile

inline unsigned blocks(long long threads, int bs) { return (unsigned)((threads + bs - 1) / bs); }

// ---------------------------------------------------------------------------
// row-tile table
// ---------------------------------------------------------------------------
// Header of (row tile (x0 .. x0 + 3, y), angle o): the first bin of the tile's taps in
// the low 26 bits and pattern = dir * 8 + steps above them (bit r: the lower bin steps
// between pixels r and r + 1; dir 0: ascending from the first bin, dir 1: descending to it).
// TAP_EDGE: a tap is off the detector or the bins do not step like that; the kernel then
// takes each pixel by itself.  TAP_NONE: no pixel is inside (-1, nd).
constexpr unsigned TAP_EDGE = 1u << 31, TAP_NONE = 0xffffffffu;

// Per pixel radon_ad's detector coordinate t = x X + y Y + off, lower bin floor(t) and
// fraction p (:832-839), with the reference's arithmetic.
__device__ unsigned tap_entry(const float4 o, int x0, int y, int N, int nd, float4 *pout) {
  int lo[ROW_P];
  float p[ROW_P];
  int in = 0;
  bool edge = false;
#pragma unroll
  for (int r = 0; r < ROW_P; ++r) {
    const int x = min(x0 + r, N - 1);  // pixels past the row end repeat its last one (their sums are not stored)
    const float tt = __fadd_rn(__fadd_rn(__fmul_rn((float)x, o.x), __fmul_rn((float)y, o.y)), o.z);
    lo[r] = 0;
    p[r] = 0.f;
    if (!(tt > -1.f && tt < (float)nd)) continue;
    ++in;
    const float fl = floorf(tt);
    p[r] = fminf(__fsub_rn(tt, fl), 0x1.fffffep-1f);
    lo[r] = (int)fl;
    if (lo[r] < 0 || lo[r] > nd - 2) edge = true;
  }
  *pout = make_float4(p[0], p[1], p[2], p[3]);
  if (in == 0) return TAP_NONE;
  if (in < ROW_P) edge = true;
  bool up = true, down = true;
  unsigned pattern = 0;
#pragma unroll
  for (int r = 0; r + 1 < ROW_P; ++r) {
    const int dlt = lo[r + 1] - lo[r];
    up = up && (dlt == 0 || dlt == 1);
    down = down && (dlt == 0 || dlt == -1);
    pattern |= (unsigned)(dlt != 0) << r;
  }
  if (edge || (!up && !down)) return TAP_EDGE;
  if (!up) pattern |= 8u;
  return (unsigned)(up ? lo[0] : lo[ROW_P - 1]) | (pattern << 26);
}

// one thread per (row tile, angle)
__global__ void k_tap_fill(const float4 *__restrict__ ofs, int N, int nd, int nang, unsigned *__restrict__ hdr,
                           float4 *__restrict__ frac) {
  const int ntx = (N + ROW_P - 1) / ROW_P;
  const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= (long long)ntx * N * nang) return;
  const long long tile = t / nang;
  const int j = (int)(t - tile * nang);
  const int y = (int)(tile / ntx), tx = (int)(tile - (long long)y * ntx);
  hdr[t] = tap_entry(__ldg(ofs + j), tx * ROW_P, y, N, nd, frac + t);
}

// pixel r's lower tap for pattern PAT, as an index into the tile's bins
template <int PAT, int R>
struct RowTap {
  static constexpr int step(int r) { return (PAT >> r) & 1; }
  static constexpr int up_k(int r) { return r == 0 ? 0 : up_k(r - 1) + step(r - 1); }
  static constexpr int down_k(int r) { return r == ROW_P - 1 ? 0 : down_k(r + 1) + step(r); }
  static constexpr int k = (PAT & 8) ? down_k(R) : up_k(R);
};

template <int PAT, int VW>
__device__ __forceinline__ void tap_apply(VecAcc<VW> (&acc)[ROW_P], const float *__restrict__ lj, size_t S, int off2,
                                          const float4 f) {
  constexpr int NB = 2 + (PAT & 1) + ((PAT >> 1) & 1) + ((PAT >> 2) & 1);
  Vec<VW> T[NB];
#pragma unroll
  for (int m = 0; m < NB; ++m) T[m].load(lj + (size_t)m * S, off2);
  acc[0].fma(__fsub_rn(1.0f, f.x), T[RowTap<PAT, 0>::k]);
  acc[0].fma(f.x, T[RowTap<PAT, 0>::k + 1]);
  acc[1].fma(__fsub_rn(1.0f, f.y), T[RowTap<PAT, 1>::k]);
  acc[1].fma(f.y, T[RowTap<PAT, 1>::k + 1]);
  acc[2].fma(__fsub_rn(1.0f, f.z), T[RowTap<PAT, 2>::k]);
  acc[2].fma(f.z, T[RowTap<PAT, 2>::k + 1]);
  acc[3].fma(__fsub_rn(1.0f, f.w), T[RowTap<PAT, 3>::k]);
  acc[3].fma(f.w, T[RowTap<PAT, 3>::k + 1]);
}

// one pixel of an edge tile: each tap only where it is on the detector
template <int VW>
__device__ __forceinline__ void tap_edge(VecAcc<VW> &acc, const float *__restrict__ lj, size_t S, int off2, int nd,
                                         const float4 o, float xf, float yf) {
  const float tt = __fadd_rn(__fadd_rn(__fmul_rn(xf, o.x), __fmul_rn(yf, o.y)), o.z);
  if (!(tt > -1.f && tt < (float)nd)) return;
  const float fl = floorf(tt);
  const float p = fminf(__fsub_rn(tt, fl), 0x1.fffffep-1f);
  const int il = (int)fl;
  Vec<VW> v;
  if (il >= 0) {
    v.load(lj + (size_t)il * S, off2);
    acc.fma(__fsub_rn(1.0f, p), v);
  }
  if (il <= nd - 2) {
    v.load(lj + (size_t)(il + 1) * S, off2);
    acc.fma(p, v);
  }
}

// a block's 8 warps own 2 x 4 row tiles of one slice chunk (an 8 x 4 pixel region, whose taps
// overlap in L1); MINB resident blocks cap the registers
template <int VW, int MINB>
__global__ void __launch_bounds__(256, MINB) k_bp_tap(const IterParams P) {
  const Dims d = P.d;
  const int ntx = (d.N + ROW_P - 1) / ROW_P;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int tx = blockIdx.x * 2 + (warp & 1), y = blockIdx.y * 4 + (warp >> 1);
  if (tx >= ntx || y >= d.N) return;
  constexpr int LW = VW == 8 ? 4 : VW;
  const int s0 = blockIdx.z * 32 * VW + lane * LW;
  const bool va = s0 < d.S, vb = VW == 8 && s0 + 128 < d.S;
  const size_t S = d.S, jstride = (size_t)d.nd * S;
  const size_t tile = ((size_t)y * ntx + tx) * d.nang;
  const unsigned *__restrict__ hdr = P.tap_hdr + tile;
  const float4 *__restrict__ frac = P.tap_frac + tile;
  // lanes past S read the last slices (their sums are not stored)
  const float *__restrict__ lam = P.lam + min(s0, d.S - LW);
  const int off2 = vb ? 128 : 0;
  VecAcc<VW> acc[ROW_P];
#pragma unroll
  for (int r = 0; r < ROW_P; ++r) acc[r].zero();
  unsigned hn = __ldg(hdr);
  for (int j = 0; j < d.nang; ++j, lam += jstride) {
    const unsigned h = hn;
    if (j + 1 < d.nang) hn = __ldg(hdr + j + 1);
    if (h == TAP_NONE) continue;
    const float4 f = __ldg(frac + j);
    if (h & TAP_EDGE) {
      const float4 o = __ldg(P.ofs + j);
#pragma unroll
      for (int r = 0; r < ROW_P; ++r)
        tap_edge<VW>(acc[r], lam, S, off2, d.nd, o, (float)min(tx * ROW_P + r, d.N - 1), (float)y);
      continue;
    }
    const float *__restrict__ lj = lam + (size_t)(h & 0x3ffffffu) * S;
    switch (h >> 26) {
#define GT_TAP_CASE(c) \
  case c: tap_apply<c, VW>(acc, lj, S, off2, f); break;
      GT_TAP_CASE(0) GT_TAP_CASE(1) GT_TAP_CASE(2) GT_TAP_CASE(3) GT_TAP_CASE(4) GT_TAP_CASE(5)
      GT_TAP_CASE(6) GT_TAP_CASE(7) GT_TAP_CASE(8) GT_TAP_CASE(9) GT_TAP_CASE(10) GT_TAP_CASE(11)
      GT_TAP_CASE(12) GT_TAP_CASE(13) GT_TAP_CASE(14) GT_TAP_CASE(15)
#undef GT_TAP_CASE
      default: break;
    }
  }
  if (!va) return;
#pragma unroll
  for (int r = 0; r < ROW_P; ++r) {
    const int x = tx * ROW_P + r;
    float a[VW];
    acc[r].get(a);
    if (x < d.N) Vec<VW>::store(P.kstar + ((size_t)y * d.N + x) * S + s0, a, vb);
  }
}

template <int VW, int MINB>
void bp_tap(const IterParams &P, cudaStream_t st) {
  const int ntx = (P.d.N + ROW_P - 1) / ROW_P;
  const dim3 grid((ntx + 1) / 2, (P.d.N + 3) / 4, (P.d.S + 32 * VW - 1) / (32 * VW));
  k_bp_tap<VW, MINB><<<grid, 256, 0, st>>>(P);
}

template <int VW, int UA, int NT>
__global__ void __launch_bounds__(NT, 1) k_bp_flat(const IterParams P) {
  int pix, s0;
  float r[VW];
  if (!bp_flat_body<VW, UA>(P, (long long)blockIdx.x * NT + threadIdx.x, pix, s0, r)) return;
  Vec<VW>::store(P.kstar + (size_t)pix * P.d.S + s0, r, false);
}

template <int VW, int UA, int NT>
void bp_flat(const IterParams &P, cudaStream_t st) {
  k_bp_flat<VW, UA, NT><<<blocks((long long)(P.d.S / VW) * P.d.N * P.d.N, NT), NT, 0, st>>>(P);
}

template <int VW>
__global__ void __launch_bounds__(128, 1) k_bp_staged(const IterParams P) {
  __shared__ BpStage<VW> sh[4];
  const int warp = threadIdx.x >> 5;
  int pix;
  float r[VW];
  if (bp_staged_body<VW>(P, (long long)blockIdx.x * 4 + warp, sh[warp], pix, r))
    Vec<VW>::store(P.kstar + (size_t)pix * VW, r, false);
}

template <int VW>
void bp_staged(const IterParams &P, cudaStream_t st) {
  k_bp_staged<VW><<<blocks(P.npix, 4 * BS_PIX), 128, 0, st>>>(P);
}

}  // namespace

// ---------------------------------------------------------------------------
// host side
// ---------------------------------------------------------------------------
// (row tile, angle) pairs of the table; 0 where it does not apply (bins beyond the header's bits)
long long tap_entries(int N, int nd, int nang) {
  return nd < (1 << 26) ? (long long)((N + ROW_P - 1) / ROW_P) * N * nang : 0;
}

cudaError_t launch_tap_fill(const float4 *ofs, int N, int nd, int nang, unsigned *hdr, float4 *frac, cudaStream_t st) {
  const long long n = tap_entries(N, nd, nang);
  k_tap_fill<<<blocks(n, 128), 128, 0, st>>>(ofs, N, nd, nang, hdr, frac);
  return cudaGetLastError();
}

// k_bp_tap with vw slices per lane (8, 4: S a multiple of 4; 2: even S)
cudaError_t launch_bp_tap(const IterParams &P, int vw, cudaStream_t st) {
  if (vw == 8) bp_tap<8, 3>(P, st);
  else if (vw == 4) bp_tap<4, 4>(P, st);
  else bp_tap<2, 5>(P, st);
  return cudaGetLastError();
}

// k_bp_flat with vw slices per thread (4, 2 or 1, a divisor of S)
cudaError_t launch_bp_flat(const IterParams &P, int vw, cudaStream_t st) {
  if (vw == 4) bp_flat<4, 4, 64>(P, st);
  else if (vw == 2) bp_flat<2, 8, 64>(P, st);
  else bp_flat<1, 8, 64>(P, st);
  return cudaGetLastError();
}

// k_bp_staged (S = 1, 2 or 4)
cudaError_t launch_bp_staged(const IterParams &P, cudaStream_t st) {
  if (P.d.S == 4) bp_staged<4>(P, st);
  else if (P.d.S == 2) bp_staged<2>(P, st);
  else bp_staged<1>(P, st);
  return cudaGetLastError();
}

}  // namespace gt
