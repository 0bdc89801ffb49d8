// Forward projectors of the solver iteration (sm_103a): forward projection `radon` of
// ubar (radon_tgv_primal_dual_3d.py:773-816) fused with the data dual's update
// (update_lambda_KL :690-704, update_lambda_L2 :677-688).
//
// What bounds them: a ray sums about 2 N pixels of S slice values each, and the loads' way
// back to the registers (128 bytes a clock and SM, broadcast table entries included) is
// the limit where there are many slices per pixel; the latency of dependent loads where
// there are few.
//
// k_fwd_pair: a warp owns the two adjacent bins 2q, 2q + 1 of an angle and 32 VW slices.
// The pixels of the two rays are listed once each (three quarters of the two rays'
// entries) with their detector coordinate t; both hat weights max(0, 1 - |t - i|)
// come from t, so an entry is 8 bytes, and a loaded pixel feeds both bins by packed
// multiply-adds.  Small blocks in order of falling ray length (centre bins first) even out
// the SMs' ends.  256^2 x 60 x 4, 71 angles: 386 -> 333 us against the ray table kernel
// (write-back 84 % busy there); 512^2 x 96 x 4, 141 angles, where the centre-first order
// also keeps the running blocks' pixels in L2: 7795 -> 4404 us with 4 slices per lane.
// Three and four bins per warp load fewer pixels still but took 399 and 530 us: their
// zero-weight products and registers cost more than the loads saved.
//
// k_fwd_pair_flat: a thread owns a pair of bins and 4 slices, threads of a warp run on over
// pairs: 80 to 128 slices do not fill the lanes of a warp per pair.  128^2, 71 angles, 92 slices:
// 53 us (k_fwd_flat 61, k_fwd_pair 61).  With half the threads of k_fwd_flat it gains nothing
// below that: 64 slices 33 us with the image in L2 but 48 us with cold caches (38, 45), 32 (64^2)
// 14.4 us (10.4).
//
// k_fwd_flat: a thread owns one ray and VW slices, threads of a warp run on over rays;
// with few slices a warp holds several rays and no lane idles.  Bound by the latency of its
// loads, 12 in flight.  64^2 x 32, 71 angles: 10.4 us (16.4 with a warp per ray); 177^2 x 16, 45
// angles: 24.4 us (33); 101^2 x 40, 33 angles: 15.3 us.
//
// k_fwd_staged: one, two or four slices.  A thread per ray would read the ray table
// uncoalesced (one sector per lane and entry) in a bare chain of loads; here the warps of a
// block read the entries of 32 rays in runs, gather their pixels into shared memory, and
// one warp adds each ray's products in order.  128^2 x 1, 60 angles: 51 us with a thread per
// ray, 12 us.  (A warp for itself with two rays has less latency and no barrier, but adds with two
// lanes: alone 26.6 -> 22.4 us an iteration, but several problems at once, as in batches, got
// slower, 1052 -> 1312 us for 100 iterations.)
//
// All kernels add each ray's terms in the reference's order (rows, then x) with the
// reference's weights (fused multiply-add), so all shapes give identical iterates.
#include <cuda_runtime.h>

#include "gt_common.cuh"
#include "gt_flat.cuh"
#include "gt_geom.cuh"
#include "gt_vec.cuh"

namespace gt {

namespace {

inline unsigned blocks(long long threads, int bs) { return (unsigned)((threads + bs - 1) / bs); }

// ---------------------------------------------------------------------------
// pair table
// ---------------------------------------------------------------------------
// Entries (pixel, t bits) of the rays 2q and 2q + 1 of one angle: every pixel that either
// ray takes, in the reference's order.  A ray takes a pixel when its weight is positive and
// its x lies in the row's truncated bounds; rounding of those bounds can leave out a pixel
// whose weight is (barely) positive.  The kernel has only t, so a pair with such a pixel
// beside one it shares gets no list (returns 0 entries) and is summed from the ray table.
template <bool FILL>
__device__ int pair_walk(const float4 o, int i0, int N, int nd, int2 *out) {
  int ylo, yhi, ylo1, yhi1;
  ray_rows(o, i0, N, ylo, yhi);
  ray_rows(o, min(i0 + 1, nd - 1), N, ylo1, yhi1);
  ylo = min(ylo, ylo1);
  yhi = max(yhi, yhi1);
  int n = 0;
  for (int y = ylo; y <= yhi; ++y) {
    const float d = __fadd_rn(__fmul_rn((float)y, o.y), o.z);
    int xl[2], xh[2];
#pragma unroll
    for (int r = 0; r < 2; ++r)
      if (i0 + r >= nd || !row_bounds(o, d, i0 + r, N, xl[r], xh[r])) { xl[r] = N; xh[r] = -1; }
    for (int x = min(xl[0], xl[1]); x <= max(xh[0], xh[1]); ++x) {
      const float t = __fadd_rn(__fmul_rn((float)x, o.x), d);
      bool any = false, lost = false;
#pragma unroll
      for (int r = 0; r < 2; ++r) {
        const bool pos = 1.0f - fabsf(__fsub_rn(t, (float)(i0 + r))) > 0.f;
        const bool in = x >= xl[r] && x <= xh[r];
        any = any || (pos && in);
        lost = lost || (pos && !in && i0 + r < nd);
      }
      if (!any) continue;
      if (lost) return 0;
      if (FILL) out[n] = make_int2(y * N + x, __float_as_int(t));
      ++n;
    }
  }
  return n;
}

__global__ void k_pair_count(const float4 *__restrict__ ofs, int N, int nd, int nang, int *__restrict__ count) {
  const int np = (nd + 1) / 2;
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= np * nang) return;
  const int j = t / np, q = t - j * np;
  count[t] = pair_walk<false>(__ldg(ofs + j), 2 * q, N, nd, nullptr);
}

__global__ void k_pair_fill(const float4 *__restrict__ ofs, int N, int nd, int nang, const long long *__restrict__ start,
                            int2 *__restrict__ ent) {
  const int np = (nd + 1) / 2;
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= np * nang || start[t] == start[t + 1]) return;
  const int j = t / np, q = t - j * np;
  pair_walk<true>(__ldg(ofs + j), 2 * q, N, nd, ent + start[t]);
}

// ---------------------------------------------------------------------------
// sums
// ---------------------------------------------------------------------------
// two rays from the pair table; false where a product of a zero weight and an infinity or NaN may
// have reached the wrong ray (looked at after the first group too: once an iterate is NaN
// everywhere, as the nuclear projection's can be, the sums from the ray table follow at once)
template <int VW, int UNR>
__device__ __forceinline__ bool pair_sum(const float *__restrict__ img, size_t S, const int2 *__restrict__ ent, int n,
                                         float fi0, int off2, VecAcc<VW> (&acc)[2]) {
  auto add = [&](float t, const Vec<VW> &v) {
    acc[0].fma(fmaxf(0.f, 1.0f - fabsf(__fsub_rn(t, fi0))), v);
    acc[1].fma(fmaxf(0.f, 1.0f - fabsf(__fsub_rn(t, fi0 + 1.f))), v);
  };
  int2 nx[UNR];
#pragma unroll
  for (int u = 0; u < UNR; ++u) nx[u] = __ldg(ent + min(u, n - 1));
  int e = 0;
  for (; e + UNR <= n; e += UNR) {
    float t[UNR];
    Vec<VW> v[UNR];
#pragma unroll
    for (int u = 0; u < UNR; ++u) {
      v[u].load(img + (size_t)nx[u].x * S, off2);
      t[u] = __int_as_float(nx[u].y);
    }
#pragma unroll
    for (int u = 0; u < UNR; ++u) nx[u] = __ldg(ent + min(e + UNR + u, n - 1));
#pragma unroll
    for (int u = 0; u < UNR; ++u) add(t[u], v[u]);
    if (e == 0 && !(acc[0].finite() && acc[1].finite())) return false;
  }
#pragma unroll
  for (int u = 0; u < UNR - 1; ++u) {
    if (e + u < n) {
      Vec<VW> v;
      v.load(img + (size_t)nx[u].x * S, off2);
      add(__int_as_float(nx[u].y), v);
    }
  }
  return acc[0].finite() && acc[1].finite();
}

// ---------------------------------------------------------------------------
// k_fwd_pair: blocks of AG angles x BG pairs (warps) of one slice chunk
// ---------------------------------------------------------------------------
template <int DISC, int VW, int UNR, int AG, int BG, int MINB>
__global__ void __launch_bounds__(AG *BG * 32, MINB) k_fwd_pair(const IterParams P) {
  const Dims d = P.d;
  const int np = (d.nd + 1) / 2, nb = (np + BG - 1) / BG, na = (d.nang + AG - 1) / AG;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  // groups of pairs from the centre of the detector outwards, angles fastest
  const int k = blockIdx.x / na, ag = blockIdx.x - k * na, h = nb / 2;
  const int bb = (nb & 1) ? ((k & 1) ? h - (k + 1) / 2 : h + k / 2) : ((k & 1) ? h + k / 2 : h - 1 - k / 2);
  const int j = ag * AG + warp / BG, q = bb * BG + warp % BG;
  if (j >= d.nang || q >= np) return;
  const size_t S = d.S;
  constexpr int LW = VW == 8 ? 4 : VW;  // slices of a lane's first run
  const int s0 = blockIdx.y * 32 * VW + lane * LW;
  const bool vb = VW == 8 && s0 + 128 < d.S;
  // lanes past S read the last slices (their sums are not stored)
  const float *__restrict__ img = P.ubar + min(s0, d.S - LW);
  const int off2 = vb ? 128 : 0;
  const int i0 = 2 * q;
  const long long b0 = (long long)j * d.nd + i0;
  const long long e0 = __ldg(P.pair_start + (size_t)j * np + q);
  const int n = (int)(__ldg(P.pair_start + (size_t)j * np + q + 1) - e0);
  VecAcc<VW> acc[2];
  acc[0].zero();
  acc[1].zero();
  bool exact = n == 0;  // no list: from the ray table (no entries there either for rays off the image)
  if (!exact) {
    exact = !pair_sum<VW, UNR>(img, S, P.pair_ent + e0, n, (float)i0, off2, acc);
  }
  if (exact) {
#pragma unroll 1
    for (int r = 0; r < 2 && i0 + r < d.nd; ++r) {
      const long long r0 = __ldg(P.ray_start + b0 + r);
      VecAcc<VW> a;
      a.zero();
      ray_sum<VW, VW == 8 ? 1 : 4>(img, S, P.ray_ent + r0, (int)(__ldg(P.ray_start + b0 + r + 1) - r0), off2, a);
      if (r == 0) acc[0] = a;
      else acc[1] = a;
    }
  }
  if (s0 >= d.S) return;
  data_step<VW>(P, DISC, acc[0], b0, s0, vb);
  if (i0 + 1 < d.nd) data_step<VW>(P, DISC, acc[1], b0 + 1, s0, vb);
}

template <int VW, int UNR, int AG, int BG, int MINB>
void fwd_pair(const IterParams &P, int disc, cudaStream_t st) {
  const int np = (P.d.nd + 1) / 2, nb = (np + BG - 1) / BG, na = (P.d.nang + AG - 1) / AG;
  const dim3 g((unsigned)nb * na, (P.d.S + 32 * VW - 1) / (32 * VW));
  if (disc == KL) k_fwd_pair<KL, VW, UNR, AG, BG, MINB><<<g, AG * BG * 32, 0, st>>>(P);
  else if (disc == L2) k_fwd_pair<L2, VW, UNR, AG, BG, MINB><<<g, AG * BG * 32, 0, st>>>(P);
  else k_fwd_pair<DATA_NONE, VW, UNR, AG, BG, MINB><<<g, AG * BG * 32, 0, st>>>(P);
}

// ---------------------------------------------------------------------------
// k_fwd_flat: thread = (ray, VW slices)
// ---------------------------------------------------------------------------
template <int DISC, int VW, int UNR, int NT>
__global__ void __launch_bounds__(NT, 1) k_fwd_flat(const IterParams P) {
  fwd_flat_body<VW, UNR>(P, DISC, (long long)blockIdx.x * NT + threadIdx.x);
}

template <int VW, int UNR, int NT>
void fwd_flat(const IterParams &P, int disc, cudaStream_t st) {
  const unsigned g = blocks((long long)(P.d.S / VW) * P.d.nd * P.d.nang, NT);
  if (disc == KL) k_fwd_flat<KL, VW, UNR, NT><<<g, NT, 0, st>>>(P);
  else if (disc == L2) k_fwd_flat<L2, VW, UNR, NT><<<g, NT, 0, st>>>(P);
  else k_fwd_flat<DATA_NONE, VW, UNR, NT><<<g, NT, 0, st>>>(P);
}

// ---------------------------------------------------------------------------
// k_fwd_pair_flat: thread = (pair of bins, 4 slices)
// ---------------------------------------------------------------------------
constexpr int PF_G = 4;  // adjacent pairs that stay together; their groups go from the centre outwards

template <int DISC, int UNR>
__global__ void __launch_bounds__(64, 1) k_fwd_pair_flat(const IterParams P) {
  const Dims d = P.d;
  const int ng = d.S / 4, np = (d.nd + 1) / 2, nb = (np + PF_G - 1) / PF_G;
  const long long t = (long long)blockIdx.x * 64 + threadIdx.x, o = div_pos(t, ng);
  const int s0 = (int)(t - o * ng) * 4, b = (int)(o / PF_G), k = b / d.nang, j = b - k * d.nang, h = nb / 2;
  const int bb = (nb & 1) ? ((k & 1) ? h - (k + 1) / 2 : h + k / 2) : ((k & 1) ? h + k / 2 : h - 1 - k / 2);
  const int q = bb * PF_G + (int)(o % PF_G);
  if (k >= nb || q >= np) return;
  const int i0 = 2 * q;
  const long long b0 = (long long)j * d.nd + i0;
  const long long e0 = __ldg(P.pair_start + (size_t)j * np + q);
  const int n = (int)(__ldg(P.pair_start + (size_t)j * np + q + 1) - e0);
  const float *__restrict__ img = P.ubar + s0;
  VecAcc<4> acc[2];
  acc[0].zero();
  acc[1].zero();
  bool exact = n == 0;  // see k_fwd_pair
  if (!exact) {
    exact = !pair_sum<4, UNR>(img, d.S, P.pair_ent + e0, n, (float)i0, 0, acc);
  }
  if (exact) {
#pragma unroll 1
    for (int r = 0; r < 2 && i0 + r < d.nd; ++r) {
      const long long r0 = __ldg(P.ray_start + b0 + r);
      VecAcc<4> a;
      a.zero();
      ray_sum<4, 8>(img, d.S, P.ray_ent + r0, (int)(__ldg(P.ray_start + b0 + r + 1) - r0), 0, a);
      if (r == 0) acc[0] = a;
      else acc[1] = a;
    }
  }
  data_step<4>(P, DISC, acc[0], b0, s0, false);
  if (i0 + 1 < d.nd) data_step<4>(P, DISC, acc[1], b0 + 1, s0, false);
}

template <int UNR>
void fwd_pair_flat(const IterParams &P, int disc, cudaStream_t st) {
  const long long np = (P.d.nd + 1) / 2, pairs = (np + PF_G - 1) / PF_G * PF_G * P.d.nang;
  const unsigned g = blocks(pairs * (P.d.S / 4), 64);
  if (disc == KL) k_fwd_pair_flat<KL, UNR><<<g, 64, 0, st>>>(P);
  else if (disc == L2) k_fwd_pair_flat<L2, UNR><<<g, 64, 0, st>>>(P);
  else k_fwd_pair_flat<DATA_NONE, UNR><<<g, 64, 0, st>>>(P);
}

// ---------------------------------------------------------------------------
// k_fwd_staged: S = VW slices (fwd_staged_body)
// ---------------------------------------------------------------------------
template <int DISC, int VW>
__global__ void __launch_bounds__(256, 1) k_fwd_staged(const IterParams P) {
  __shared__ FwdStage<VW> sh;
  fwd_staged_body<VW>(P, DISC, blockIdx.x, sh);
}

template <int VW>
void fwd_staged(const IterParams &P, int disc, cudaStream_t st) {
  const unsigned g = blocks((long long)P.d.nd * P.d.nang, FS_RAYS);
  if (disc == KL) k_fwd_staged<KL, VW><<<g, 256, 0, st>>>(P);
  else if (disc == L2) k_fwd_staged<L2, VW><<<g, 256, 0, st>>>(P);
  else k_fwd_staged<DATA_NONE, VW><<<g, 256, 0, st>>>(P);
}

}  // namespace

// ---------------------------------------------------------------------------
// host side
// ---------------------------------------------------------------------------
cudaError_t launch_pair_count(const float4 *ofs, int N, int nd, int nang, int *count, cudaStream_t st) {
  k_pair_count<<<blocks((long long)((nd + 1) / 2) * nang, 64), 64, 0, st>>>(ofs, N, nd, nang, count);
  return cudaGetLastError();
}

cudaError_t launch_pair_fill(const float4 *ofs, int N, int nd, int nang, const long long *start, int2 *ent,
                             cudaStream_t st) {
  k_pair_fill<<<blocks((long long)((nd + 1) / 2) * nang, 64), 64, 0, st>>>(ofs, N, nd, nang, start, ent);
  return cudaGetLastError();
}

// k_fwd_pair with vw = 8 or 4 slices per lane (S a multiple of 4)
cudaError_t launch_fwd_pair(const IterParams &P, int disc, int vw, cudaStream_t st) {
  if (vw == 8) fwd_pair<8, 2, 2, 2, 8>(P, disc, st);
  else fwd_pair<4, 8, 1, 4, 6>(P, disc, st);
  return cudaGetLastError();
}

// k_fwd_pair_flat (S a multiple of 4)
cudaError_t launch_fwd_pair_flat(const IterParams &P, int disc, cudaStream_t st) {
  fwd_pair_flat<8>(P, disc, st);
  return cudaGetLastError();
}

// k_fwd_flat with vw slices per thread (4, 2 or 1, a divisor of S)
cudaError_t launch_fwd_flat(const IterParams &P, int disc, int vw, cudaStream_t st) {
  if (vw == 4) fwd_flat<4, 12, 64>(P, disc, st);
  else if (vw == 2) fwd_flat<2, 8, 128>(P, disc, st);
  else fwd_flat<1, 8, 128>(P, disc, st);
  return cudaGetLastError();
}

// k_fwd_staged (S = 1, 2 or 4)
cudaError_t launch_fwd_staged(const IterParams &P, int disc, cudaStream_t st) {
  if (P.d.S == 4) fwd_staged<4>(P, disc, st);
  else if (P.d.S == 2) fwd_staged<2>(P, disc, st);
  else fwd_staged<1>(P, disc, st);
  return cudaGetLastError();
}

}  // namespace gt
