// fss_score_small.cu -- Tanimoto scores of packed pairs of clouds of at most kWidePoints points, with
// the fit side's gradient of the score in the same pass: a warp for a run of pairs up to
// kSmallPoints (atom clouds), a CTA a pair above (surfaces) and for few pairs.
#include <algorithm>

#include "fss_internal.cuh"

namespace fss {
namespace {

constexpr int kWarps = 4;                       // warps of a CTA, independent of one another
constexpr int kRowLanes = 16;                   // lanes that own rows; two halves share the sum
constexpr int kMaxWideWarps = kWidePoints / kSmallPoints;

// A staged cloud: points (2p, 2p + 1) along the f32x2 lanes, negated, so that a difference is one
// packed addition.  F[2p] = -(x, x', y, y'), F[2p + 1] = -(z, z', c, c').  Padded to a multiple of
// four points (one pair to each half) by points so far away that their Gaussian is exactly 0.
struct Cloud {
  float4 *F, *plain;
};
struct SmallCloud {
  float4 F[kSmallPoints];
  float4 plain[kSmallPoints];
};

constexpr float kFar = 3e18f;   // squared distance from any cloud stays finite

__device__ __forceinline__ void put_point(Cloud c, int k, float4 v) {
  float* f = reinterpret_cast<float*>(c.F + (k & ~1)) + (k & 1);
  f[0] = -v.x; f[2] = -v.y; f[4] = -v.z; f[6] = -v.w;
  c.plain[k] = v;
}

// Loads and stages the cloud [begin, begin + n) with `threads` threads.
__device__ __forceinline__ void stage(Cloud c, const float4* __restrict__ pts, int begin, int n,
                                      int thread, int threads) {
  const int padded = (n + 3) & ~3;
  for (int k = thread; k < padded; k += threads)
    put_point(c, k, k < n ? pts[begin + k] : make_float4(kFar, kFar, kFar, 0.f));
}

// R rows per lane against a staged cloud, this half's pairs only: V += sum g (both halves of an
// f32x2 sum kept apart), and with GRAD d[r] = sum g (b_r - y) (w: the charges).
template <bool ESP, bool GRAD, int R>
__device__ __forceinline__ void rows(const float4 (&b)[R], const Cloud c, int n, int half,
                                     float nk, float ne, float2& V, float4 (&d)[R]) {
  const float2 z2 = make_float2(0.f, 0.f);
  const float2 nk2 = make_float2(nk, nk), ne2 = make_float2(ne, ne);
  float2 mx[R], my[R], mz[R], mc[R];
#pragma unroll
  for (int r = 0; r < R; ++r) mx[r] = my[r] = mz[r] = mc[r] = z2;
  const float4* F = c.F + 2 * half;
  const int pairs = (n + 3) / 4;   // pairs of each half
#pragma unroll 2
  for (int p = 0; p < pairs; ++p) {
    const float4 f0 = F[4 * p], f1 = F[4 * p + 1];
#pragma unroll
    for (int r = 0; r < R; ++r) {
      const float2 dx = __fadd2_rn(make_float2(b[r].x, b[r].x), make_float2(f0.x, f0.y));
      const float2 dy = __fadd2_rn(make_float2(b[r].y, b[r].y), make_float2(f0.z, f0.w));
      const float2 dz = __fadd2_rn(make_float2(b[r].z, b[r].z), make_float2(f1.x, f1.y));
      float2 E = __fmul2_rn(nk2, __ffma2_rn(dz, dz, __ffma2_rn(dy, dy, __fmul2_rn(dx, dx))));
      float2 dc = z2;
      if (ESP) {
        dc = __fadd2_rn(make_float2(b[r].w, b[r].w), make_float2(f1.z, f1.w));
        E = __ffma2_rn(__fmul2_rn(ne2, dc), dc, E);
      }
      const float2 g = make_float2(ex2(E.x), ex2(E.y));
      V = __fadd2_rn(V, g);
      if (GRAD) {
        mx[r] = __ffma2_rn(g, dx, mx[r]);
        my[r] = __ffma2_rn(g, dy, my[r]);
        mz[r] = __ffma2_rn(g, dz, mz[r]);
        if (ESP) mc[r] = __ffma2_rn(g, dc, mc[r]);
      }
    }
  }
#pragma unroll
  for (int r = 0; r < R; ++r)
    d[r] = make_float4(mx[r].x + mx[r].y, my[r].x + my[r].y, mz[r].x + mz[r].y,
                       mc[r].x + mc[r].y);
}

__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// Row points j = first + stride r of this lane; rows past the cloud are a far point, whose terms
// are 0.
template <int R>
__device__ __forceinline__ void row_points(const Cloud c, int n, int first, int stride,
                                           float4 (&b)[R]) {
#pragma unroll
  for (int r = 0; r < R; ++r) {
    const int j = first + stride * r;
    b[r] = j < n ? c.plain[j] : make_float4(-kFar, -kFar, -kFar, 0.f);
  }
}

// This lane's part of the self overlap of a staged cloud: 16 rows at a time, their own 16 columns
// once and the later ones twice.  Each warp takes early and late rows in turn.
template <bool ESP>
__device__ __forceinline__ float self_sum(const Cloud c, int n, int lane, int warp, int warps,
                                          float nk, float ne) {
  float2 own = make_float2(0.f, 0.f), later = own;
  const int half = lane / kRowLanes;
#pragma unroll 1
  for (int r = 0; kRowLanes * warps * r < n; ++r) {
    const int j0 = kRowLanes * (warps * r + (r & 1 ? warps - 1 - warp : warp));
    if (j0 >= n) continue;
    float4 b[1], d[1];
    row_points<1>(c, n, j0 + lane % kRowLanes, 0, b);
    rows<ESP, false, 1>(b, Cloud{c.F + j0, nullptr}, min(n - j0, kRowLanes), half, nk, ne, own, d);
    rows<ESP, false, 1>(b, Cloud{c.F + j0 + kRowLanes, nullptr}, max(n - j0 - kRowLanes, 0), half,
                        nk, ne, later, d);
  }
  return fmaf(2.f, later.x + later.y, own.x + own.y);
}

// This lane's part of the overlap of two staged clouds, a lane per point of the larger one (A): for
// a cloud B of too few points to give the warps a row each.
template <bool ESP>
__device__ __forceinline__ float cross_sum(const Cloud A, const Cloud B, int n, int m, int lane,
                                           int warp, int warps, float nk, float ne) {
  float2 v = make_float2(0.f, 0.f);
#pragma unroll 1
  for (int j0 = kRowLanes * warp; j0 < n; j0 += kRowLanes * warps) {
    float4 b[1], d[1];
    row_points<1>(A, n, j0 + lane % kRowLanes, 0, b);
    rows<ESP, false, 1>(b, B, m, lane / kRowLanes, nk, ne, v, d);
  }
  return v.x + v.y;
}

struct SmallArgs {
  const float4* ref;
  const int* roff;
  const float4* fit;
  const int* foff;
  const int *pr, *pf;
  int P, maxN, maxM, run;   // pairs of a warp's run
  float nk, ne, Kc, aKc, cKc;
  float *score, *ov;
  float4* unit;   // (P, maxM): d score / d fit point, GRAD only
};

__device__ __forceinline__ void write_score(const SmallArgs& a, int p, float ab, float aa,
                                            float bb) {
  a.ov[3 * (size_t)p] = ab; a.ov[3 * (size_t)p + 1] = aa; a.ov[3 * (size_t)p + 2] = bb;
  a.score[p] = ab / (aa + bb - ab);
}

__device__ __forceinline__ void write_nan(const SmallArgs& a, int p, int thread) {
  const float nan = __int_as_float(0x7fc00000);
  if (thread < 3) a.ov[3 * (size_t)p + thread] = nan;
  if (thread == 3) a.score[p] = nan;
}

// Unit gradients of this lane's fit rows from their moments against both clouds.
template <bool ESP, int R>
__device__ __forceinline__ void write_unit(const SmallArgs& a, int p, int m, int first, int stride,
                                           int half, float ab, float aa, float bb,
                                           const float4 (&dc)[R], const float4 (&ds)[R]) {
  // d score / d V_AB and d score / d V_BB; d V_XY / d x = -alpha K sum g (x - y), self twice
  const float U = aa + bb, D = U - ab;
  const float dAB = U / (D * D), dSelf = -2.f * ab / (D * D);
  float4* out = a.unit + (size_t)p * a.maxM;
#pragma unroll
  for (int r = 0; r < R; ++r) {
    float x = -a.aKc * fmaf(dAB, dc[r].x, dSelf * ds[r].x);
    float y = -a.aKc * fmaf(dAB, dc[r].y, dSelf * ds[r].y);
    float z = -a.aKc * fmaf(dAB, dc[r].z, dSelf * ds[r].z);
    x += __shfl_xor_sync(0xffffffffu, x, kRowLanes);
    y += __shfl_xor_sync(0xffffffffu, y, kRowLanes);
    z += __shfl_xor_sync(0xffffffffu, z, kRowLanes);
    float c = 0.f;
    if (ESP) {
      c = -a.cKc * fmaf(dAB, dc[r].w, dSelf * ds[r].w);
      c += __shfl_xor_sync(0xffffffffu, c, kRowLanes);
    }
    const int j = first + stride * r;
    if (half == (r & 1) && j < m) out[j] = make_float4(x, y, z, c);
  }
}

// Scores pair p from the staged clouds and the reference's self overlap.
template <bool ESP, bool GRAD, int R>
__device__ __forceinline__ void pair(const SmallArgs& a, const Cloud A, const Cloud B, int n, int m,
                                     int p, int lane, float aa) {
  const int half = lane / kRowLanes, first = lane % kRowLanes;
  float4 b[R], dc[R], ds[R];
  row_points<R>(B, m, first, kRowLanes, b);
  float2 vc = make_float2(0.f, 0.f), vs = vc;
  rows<ESP, GRAD, R>(b, A, n, half, a.nk, a.ne, vc, dc);
  rows<ESP, GRAD, R>(b, B, m, half, a.nk, a.ne, vs, ds);
  const float ab = warp_sum(vc.x + vc.y) * a.Kc, bb = warp_sum(vs.x + vs.y) * a.Kc;
  if (lane == 0) write_score(a, p, ab, aa, bb);
  if (GRAD) write_unit<ESP, R>(a, p, m, first, kRowLanes, half, ab, aa, bb, dc, ds);
}

// Each warp scores `run` consecutive pairs, so a reference shared by them (one query against
// a library) is staged, and its self overlap taken, once; the fit rows give V_AB, V_BB and the fit
// gradient from one evaluation of each Gaussian.  Sixteen lanes own rows (j mod 16, up to four in
// registers) and the two halves share the other cloud's points: 15-60 points fill 82 % of the
// lanes, rows on 32 lanes 73 %.  Differences are taken before they are squared, as everywhere in
// this form: the factored rows of the dense batches would be faster and less exact.  Bound by FP32:
// 11 lane operations a term (3 differences, 4 for the exponent, V and 3 moments).  Loading the next
// pair under this one's loops gave nothing.  One B200, 20 000 pairs of a 60-point query and 15-60
// point molecules, before (a CTA a pair, the Gaussians again in the backward) -> after: forward and
// backward 91 + 64 -> 64 + 7 us, scores alone 92 -> 46; of 15-30 points 52 + 39 -> 28 + 6.
template <bool ESP, bool GRAD>
__global__ void __launch_bounds__(32 * kWarps, 4) score_small_kernel(const SmallArgs a) {
  __shared__ SmallCloud cloud[kWarps][2];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const Cloud A{cloud[warp][0].F, cloud[warp][0].plain}, B{cloud[warp][1].F, cloud[warp][1].plain};
  const long long first = ((long long)blockIdx.x * kWarps + warp) * a.run;
  const int last = (int)min(first + a.run, (long long)a.P);
  int held = -1, n = 0;   // staged reference molecule
  float aa = 0.f;
  for (int p = (int)first; p < last; ++p) {
    const int ri = a.pr[p], fi = a.pf[p];
    const int r0 = a.roff[ri], f0 = a.foff[fi];
    const int nn = a.roff[ri + 1] - r0, m = a.foff[fi + 1] - f0;
    if (nn < 0 || m < 0 || nn > a.maxN || m > a.maxM) {   // outside the staged clouds: NaN
      write_nan(a, p, lane);
      continue;
    }
    __syncwarp();   // the last pair's reads
    stage(B, a.fit, f0, m, lane, 32);
    const bool fresh = ri != held;
    if (fresh) {
      n = nn;
      stage(A, a.ref, r0, n, lane, 32);
    }
    __syncwarp();
    if (fresh) {
      aa = a.Kc * warp_sum(self_sum<ESP>(A, n, lane, 0, 1, a.nk, a.ne));
      held = ri;
    }
    switch ((m + kRowLanes - 1) / kRowLanes) {
      case 0:
      case 1: pair<ESP, GRAD, 1>(a, A, B, n, m, p, lane, aa); break;
      case 2: pair<ESP, GRAD, 2>(a, A, B, n, m, p, lane, aa); break;
      case 3: pair<ESP, GRAD, 3>(a, A, B, n, m, p, lane, aa); break;
      default: pair<ESP, GRAD, 4>(a, A, B, n, m, p, lane, aa); break;
    }
  }
}

// A CTA per pair of larger clouds, up to 64 points a warp, and of few pairs: the same rows, split
// over the warps, and the same bound.  Runs of pairs that share the staged reference were 3 % faster at 400 points and
// 40 % slower at 310 (four pairs on some CTAs, three on the rest).  Shared memory: 32 bytes a point
// of both clouds.  One B200, 1000 charged pairs, before (the Gaussians again in the backward) ->
// after, forward and backward: 100-400 points 161 + 165 -> 186 + 4 us, 100-210 points 70 + 60 ->
// 59 + 3; 30 pairs of 100-310 points 24 + 15 -> 19 + 2; scores alone (100-400) 166 -> 138.
template <bool ESP, bool GRAD, int R>
__device__ __forceinline__ void wide_pair(const SmallArgs& a, const Cloud A, const Cloud B, int n,
                                          int m, int p, float (*red)[3]) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, warps = blockDim.x >> 5;
  const int half = lane / kRowLanes, first = lane % kRowLanes + kRowLanes * warp;
  const int stride = kRowLanes * warps;
  float4 b[R], dc[R], ds[R];
  row_points<R>(B, m, first, stride, b);
  float2 vc = make_float2(0.f, 0.f), vs = vc;
  // Fit points on a quarter of the warps or fewer leave the others idle over a long reference: V_AB
  // then has a lane per reference point (a 512-point reference against 3-16 points, scores alone, 30
  // pairs: 18.7 -> 14.7 us, 300 pairs: 35.3 -> 26.8; a thread per row 16.1 and 33.0); the gradient's
  // moments still need the fit rows.
  float x = 0.f;
  const bool turned = R == 1 && 4 * m <= stride;
  if (turned) x = cross_sum<ESP>(A, B, n, m, lane, warp, warps, a.nk, a.ne);
  if (GRAD || !turned) rows<ESP, GRAD, R>(b, A, n, half, a.nk, a.ne, vc, dc);
  rows<ESP, GRAD, R>(b, B, m, half, a.nk, a.ne, vs, ds);
  const float sab = warp_sum(turned ? x : vc.x + vc.y), sbb = warp_sum(vs.x + vs.y);
  if (lane == 0) { red[warp][0] = sab; red[warp][2] = sbb; }
  __syncthreads();
  float ab = 0.f, aa = 0.f, bb = 0.f;
  for (int w = 0; w < warps; ++w) { ab += red[w][0]; aa += red[w][1]; bb += red[w][2]; }
  ab *= a.Kc; aa *= a.Kc; bb *= a.Kc;
  if (threadIdx.x == 0) write_score(a, p, ab, aa, bb);
  if (GRAD) write_unit<ESP, R>(a, p, m, first, stride, half, ab, aa, bb, dc, ds);
}

template <bool ESP, bool GRAD, int CTAS>
__global__ void __launch_bounds__(32 * kMaxWideWarps, CTAS) score_wide_kernel(const SmallArgs a) {
  extern __shared__ __align__(16) float4 smem[];
  __shared__ float red[kMaxWideWarps][3];
  const int pn = (a.maxN + 3) & ~3, pm = (a.maxM + 3) & ~3;
  const Cloud A{smem, smem + pn}, B{smem + 2 * pn, smem + 2 * pn + pm};
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, stride = blockDim.x / 2;
  const int p = blockIdx.x;
  const int ri = a.pr[p], fi = a.pf[p];
  const int r0 = a.roff[ri], f0 = a.foff[fi];
  const int n = a.roff[ri + 1] - r0, m = a.foff[fi + 1] - f0;
  if (n < 0 || m < 0 || n > a.maxN || m > a.maxM) {
    write_nan(a, p, threadIdx.x);
    return;
  }
  stage(A, a.ref, r0, n, threadIdx.x, blockDim.x);
  stage(B, a.fit, f0, m, threadIdx.x, blockDim.x);
  __syncthreads();
  const float v = warp_sum(self_sum<ESP>(A, n, lane, warp, blockDim.x >> 5, a.nk, a.ne));
  if (lane == 0) red[warp][1] = v;
  switch ((m + stride - 1) / stride) {   // the same for the whole CTA
    case 0:
    case 1: wide_pair<ESP, GRAD, 1>(a, A, B, n, m, p, red); break;
    case 2: wide_pair<ESP, GRAD, 2>(a, A, B, n, m, p, red); break;
    case 3: wide_pair<ESP, GRAD, 3>(a, A, B, n, m, p, red); break;
    default: wide_pair<ESP, GRAD, 4>(a, A, B, n, m, p, red); break;
  }
}

// grad_fit += d loss / d score * the unit gradient, a warp per pair; a molecule of several pairs
// accumulates.  Bound by the bytes of the unit gradients and the L2's additions.
__global__ void __launch_bounds__(128) score_bwd_unit_kernel(
    const int* __restrict__ roff, const int* __restrict__ foff, const int* __restrict__ pr,
    const int* __restrict__ pf, int P, int maxN, int maxM, const float* __restrict__ gs,
    const float4* __restrict__ unit, float4* __restrict__ gfit) {
  const int lane = threadIdx.x & 31;
  const long long p = (long long)blockIdx.x * 4 + (threadIdx.x >> 5);
  if (p >= P) return;
  const int ri = pr[p], fi = pf[p], f0 = foff[fi];
  const int n = roff[ri + 1] - roff[ri], m = foff[fi + 1] - f0;
  if (n < 0 || m < 0 || n > maxN || m > maxM) return;
  const float g = gs[p];
  for (int j = lane; j < m; j += 32) {
    const float4 u = unit[p * maxM + j];
    atomicAdd(gfit + f0 + j, make_float4(g * u.x, g * u.y, g * u.z, g * u.w));
  }
}

}  // namespace

int score_small_launch(const float* ref_pts, const int32_t* ref_off, const float* fit_pts,
                       const int32_t* fit_off, const int32_t* pair_ref, const int32_t* pair_fit,
                       int P, int maxN, int maxM, float nk, float ne, float Kc, float aKc,
                       float cKc, int esp, float* score, float* overlaps, float* unit_fit,
                       cudaStream_t st) {
  const int sms = num_sms();
  SmallArgs a{reinterpret_cast<const float4*>(ref_pts), ref_off,
              reinterpret_cast<const float4*>(fit_pts), fit_off, pair_ref, pair_fit, P, maxN, maxM,
              0, nk, ne, Kc, aKc, cKc, score, overlaps, reinterpret_cast<float4*>(unit_fit)};
  const auto kern = esp ? (unit_fit ? score_small_kernel<true, true> : score_small_kernel<true, false>)
                        : (unit_fit ? score_small_kernel<false, true> : score_small_kernel<false, false>);
  // Few pairs of small clouds leave the SMs to a warp each: they take a CTA with a warp for 16 rows (up
  // to 3 an SM) or 32 (up to 6).  In us, a 60-point query against molecules of 15-60 points, scores
  // alone, a thread per row / a warp per pair / now: 30 pairs 5.8 / 6.7 / 4.2, 300 pairs 6.2 / 7.0 /
  // 4.7, 600 pairs 7.1 / 8.0 / 6.2; 1200 pairs 8.7 / 8.8 (7.7 with 32 rows a warp, but forward and
  // backward of pairs with references of their own 13.7 and 14.5).
  const bool small = maxN <= kSmallPoints && maxM <= kSmallPoints;
  if (!small || P <= 6 * sms) {
    const size_t smem = 2 * sizeof(float4) * (size_t)(((maxN + 3) & ~3) + ((maxM + 3) & ~3));
    const int rows = !small ? kSmallPoints : P <= 3 * sms ? kRowLanes : 2 * kRowLanes;
    const int warps = (std::max({maxN, maxM, 1}) - 1) / rows + 1;
    // With the gradient, four rows a lane want 128 registers, two CTAs an SM; 80 registers and three
    // CTAs are faster where a lane has at most two rows or where many CTAs wait.  In us, forward and
    // backward, 128 and 80 registers (a thread per row): a 400-point reference against 15-60 points,
    // 300 pairs 39.9 and 36.0 (43.8); 100-400 points, 300 pairs 49.1 and 57.9 (101); 15-60 points and
    // one molecule of 512, 2000 pairs 39.8 and 45.5 (61), 20 000 pairs 275 and 217 (237).
    const bool many = maxM <= 2 * kRowLanes * warps || P > 20 * sms;
    const auto wide = !unit_fit ? (esp ? score_wide_kernel<true, false, 4> : score_wide_kernel<false, false, 4>)
                      : many    ? (esp ? score_wide_kernel<true, true, 3> : score_wide_kernel<false, true, 3>)
                                : (esp ? score_wide_kernel<true, true, 2> : score_wide_kernel<false, true, 2>);
    const cudaError_t ce =
        cudaFuncSetAttribute(wide, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (ce != cudaSuccess)
      return set_error(FSS_ERR_CUDA, std::string("fss_score_fwd: ") + cudaGetErrorString(ce));
    wide<<<P, 32 * warps, smem, st>>>(a);
    return check_launch("fss_score_fwd");
  }
  int ctas = 0;
  const cudaError_t ce = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&ctas, kern, 32 * kWarps, 0);
  if (ce != cudaSuccess)
    return set_error(FSS_ERR_CUDA, std::string("fss_score_fwd: ") + cudaGetErrorString(ce));
  const int warps = std::max(1, ctas) * sms * kWarps;
  a.run = (P - 1) / warps + 1;
  const int used = (P - 1) / a.run + 1;
  kern<<<(used - 1) / kWarps + 1, 32 * kWarps, 0, st>>>(a);
  return check_launch("fss_score_fwd");
}

int score_bwd_unit_launch(const int32_t* ref_off, const int32_t* fit_off, const int32_t* pair_ref,
                          const int32_t* pair_fit, int P, int maxN, int maxM,
                          const float* grad_score, const float* unit_fit, float* grad_fit,
                          cudaStream_t st) {
  if (P < 0 || maxN < 0 || maxM < 0)
    return set_error(FSS_ERR_INVALID, "fss_score_bwd_unit: bad sizes");
  if (P == 0) return FSS_OK;
  if (!ref_off || !fit_off || !pair_ref || !pair_fit || !grad_score || !unit_fit || !grad_fit)
    return set_error(FSS_ERR_INVALID, "fss_score_bwd_unit: null pointer");
  score_bwd_unit_kernel<<<(P - 1) / 4 + 1, 128, 0, st>>>(
      ref_off, fit_off, pair_ref, pair_fit, P, maxN, maxM, grad_score,
      reinterpret_cast<const float4*>(unit_fit), reinterpret_cast<float4*>(grad_fit));
  return check_launch("fss_score_bwd_unit");
}

}  // namespace fss
