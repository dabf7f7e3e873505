// fss_seeds.cu -- multi-start seed poses for a batch of pairs, four lanes per pair.
//
// Restates batched_seeds_torch (shepherd_score/accel/drivers/_common.py:281-441):
//   identity, 4 principal-axis alignments (ref axes with the sign flips of :358-362; the
//   fit axis-0 then axis-1 alignment of :369-390), up to 6 structured +-90 degree rotations
//   about the ref axes composed onto the first PCA seed (:401-413), then a Fibonacci fill
//   (given by the caller), every seed with the COM-aligning translation of :425-428, and the
//   fixed fallback rotations for pairs with < 3 points or non-finite coordinates (:430-439).
// The PCA runs in fp64 with the closed-form symmetric 3x3 eigensolver of :207-255.  The
// second fit-axis PCA of the reference is taken on the rotated fit cloud; its inertia tensor
// is R0 I R0^T exactly, so it is formed that way instead of re-reading the points.
#include <cmath>

#include "fss_internal.cuh"

namespace fss {
namespace {

struct M3 {
  double m[3][3];
};

__device__ void sym3x3_axes(const M3& A, M3& out) {
  const double eps = 1e-12;
  const double a00 = A.m[0][0], a11 = A.m[1][1], a22 = A.m[2][2];
  const double a01 = A.m[0][1], a02 = A.m[0][2], a12 = A.m[1][2];
  const double q = (a00 + a11 + a22) / 3.0;
  const double p1 = a01 * a01 + a02 * a02 + a12 * a12;
  const double p2 = (a00 - q) * (a00 - q) + (a11 - q) * (a11 - q) + (a22 - q) * (a22 - q) + 2.0 * p1;
  const double p = sqrt(fmax(p2 / 6.0, eps));
  const double ip = 1.0 / p;
  const double b00 = (a00 - q) * ip, b11 = (a11 - q) * ip, b22 = (a22 - q) * ip;
  const double b01 = a01 * ip, b02 = a02 * ip, b12 = a12 * ip;
  const double detB = b00 * (b11 * b22 - b12 * b12) - b01 * (b01 * b22 - b12 * b02) +
                      b02 * (b01 * b12 - b11 * b02);
  const double r = fmin(fmax(detB * 0.5, -1.0), 1.0);
  const double phi = acos(r) / 3.0;
  const double e1 = q + 2.0 * p * cos(phi);
  const double e3 = q + 2.0 * p * cos(phi + 2.0 * M_PI / 3.0);
  const double e2 = 3.0 * q - e1 - e3;
  auto evec = [&](double lj, double lk, double v[3]) -> double {
    double X[3][3], Y[3][3], P[3][3];
    for (int i = 0; i < 3; ++i)
      for (int j = 0; j < 3; ++j) {
        X[i][j] = A.m[i][j] - (i == j ? lj : 0.0);
        Y[i][j] = A.m[i][j] - (i == j ? lk : 0.0);
      }
    for (int i = 0; i < 3; ++i)
      for (int j = 0; j < 3; ++j)
        P[i][j] = X[i][0] * Y[0][j] + X[i][1] * Y[1][j] + X[i][2] * Y[2][j];
    int idx = 0;
    double best = -1.0;
    for (int j = 0; j < 3; ++j) {  // max-norm column, first index on ties
      const double n = sqrt(P[0][j] * P[0][j] + P[1][j] * P[1][j] + P[2][j] * P[2][j]);
      if (n > best) { best = n; idx = j; }
    }
    const double nrm = best;
    const double inv = 1.0 / fmax(nrm, eps);
#pragma unroll
    for (int i = 0; i < 3; ++i)   // selects: a run-time column would put P in local memory
      v[i] = (idx == 0 ? P[i][0] : idx == 1 ? P[i][1] : P[i][2]) * inv;
    return nrm;
  };
  double v1[3], v2[3], v3[3];
  const double n1 = evec(e2, e3, v1);
  const double n3 = evec(e1, e2, v3);
  auto cross = [](const double a[3], const double b[3], double c[3]) {
    c[0] = a[1] * b[2] - a[2] * b[1];
    c[1] = a[2] * b[0] - a[0] * b[2];
    c[2] = a[0] * b[1] - a[1] * b[0];
  };
  auto normalize = [&](double v[3]) {
    const double n = sqrt(v[0] * v[0] + v[1] * v[1] + v[2] * v[2]);
    const double inv = 1.0 / fmax(n, eps);
    v[0] *= inv; v[1] *= inv; v[2] *= inv;
  };
  cross(v3, v1, v2);
  normalize(v2);
  cross(v2, v3, v1);
  normalize(v1);
  bool bad = n1 < 1e-9 || n3 < 1e-9;
  for (int i = 0; i < 3; ++i)
    bad = bad || !isfinite(v1[i]) || !isfinite(v2[i]) || !isfinite(v3[i]);
  for (int i = 0; i < 3; ++i) {
    out.m[0][i] = bad ? (i == 0 ? 1.0 : 0.0) : v1[i];
    out.m[1][i] = bad ? (i == 1 ? 1.0 : 0.0) : v2[i];
    out.m[2][i] = bad ? (i == 2 ? 1.0 : 0.0) : v3[i];
  }
}

// Lanes that share a pair.  Four: one per PCA seed, and one per coordinate of the float32
// centroid.
constexpr int kLanes = 4;

// A value of lane `src` of the pair's lanes, in all of them.
__device__ __forceinline__ float from_lane(float v, int src) {
  return __shfl_sync(0xffffffffu, v, src, kLanes);
}
__device__ __forceinline__ double from_lane(double v, int src) {
  return __shfl_sync(0xffffffffu, v, src, kLanes);
}
__device__ __forceinline__ double lane_sum(double v) {
  v += __shfl_xor_sync(0xffffffffu, v, 1, kLanes);
  return v + __shfl_xor_sync(0xffffffffu, v, 2, kLanes);
}

// float32 centroid of a cloud (in point order; lane c sums coordinate c), whether every
// coordinate is finite, and the inertia tensor about the fp64 centroid
// (_masked_principal_axes, :258-278) from one pass over the points relative to the float32
// centroid, whose distance from the true one (~1e-7 of the cloud) is taken out of the second
// moments.  Every lane gets all of it.
__device__ __forceinline__ void cloud_moments(const Pts pts, int n, int lane, float c[3],
                                              bool& finite, M3& I) {
  float s = 0.f;
  bool ok = true;
#pragma unroll 8
  for (int i = 0; i < n; ++i) {
    const float4 p = pts[i];
    const float x = lane == 0 ? p.x : lane == 1 ? p.y : p.z;
    s += x;
    ok = ok && isfinite(x);
  }
  __syncwarp();
  const float m = s / (float)(n > 0 ? n : 1);
#pragma unroll
  for (int i = 0; i < 3; ++i) c[i] = from_lane(m, i);
  finite = (__ballot_sync(0xffffffffu, !ok) >> (threadIdx.x & 28) & 15) == 0;
  double sx = 0, sy = 0, sz = 0, xx = 0, xy = 0, xz = 0, yy = 0, yz = 0, zz = 0;
#pragma unroll 2
  for (int i = lane; i < n; i += kLanes) {
    const float4 p = pts[i];
    const double x = (double)p.x - c[0], y = (double)p.y - c[1], z = (double)p.z - c[2];
    sx += x; sy += y; sz += z;
    xx += x * x; xy += x * y; xz += x * z; yy += y * y; yz += y * z; zz += z * z;
  }
  __syncwarp();
  sx = lane_sum(sx); sy = lane_sum(sy); sz = lane_sum(sz);
  xx = lane_sum(xx); xy = lane_sum(xy); xz = lane_sum(xz);
  yy = lane_sum(yy); yz = lane_sum(yz); zz = lane_sum(zz);
  const double inv = 1.0 / (double)(n > 0 ? n : 1);
  const double mx = sx * inv, my = sy * inv, mz = sz * inv;
  xx -= sx * mx; xy -= sx * my; xz -= sx * mz; yy -= sy * my; yz -= sy * mz; zz -= sz * mz;
  I.m[0][0] = yy + zz; I.m[0][1] = -xy; I.m[0][2] = -xz;
  I.m[1][0] = -xy; I.m[1][1] = xx + zz; I.m[1][2] = -yz;
  I.m[2][0] = -xz; I.m[2][1] = -yz; I.m[2][2] = xx + yy;
}

template <typename T>
__device__ void quat_mul(const T a[4], const T b[4], T o[4]) {
  o[0] = a[0] * b[0] - a[1] * b[1] - a[2] * b[2] - a[3] * b[3];
  o[1] = a[0] * b[1] + a[1] * b[0] + a[2] * b[3] - a[3] * b[2];
  o[2] = a[0] * b[2] - a[1] * b[3] + a[2] * b[0] + a[3] * b[1];
  o[3] = a[0] * b[3] + a[1] * b[2] - a[2] * b[1] + a[3] * b[0];
}

// The float32 product of the structured seeds.  Every rounding is written out: a seed's last bit
// decides where its alignment ends.
__device__ __forceinline__ float four_products(float a, float b, float c, float d, float e,
                                               float f, float g, float h) {
  return __fmaf_rn(g, h, __fmaf_rn(e, f, __fmaf_rn(c, d, __fmul_rn(a, b))));
}
__device__ __forceinline__ void quat_mul_f(const float a[4], const float b[4], float o[4]) {
  o[0] = four_products(a[0], b[0], -a[1], b[1], -a[2], b[2], -a[3], b[3]);
  o[1] = four_products(a[0], b[1], a[1], b[0], a[2], b[3], -a[3], b[2]);
  o[2] = four_products(a[0], b[2], -a[1], b[3], a[2], b[0], a[3], b[1]);
  o[3] = four_products(a[0], b[3], a[1], b[2], -a[2], b[1], a[3], b[0]);
}

// rotation matrix of a quaternion after normalising it (quaternion_to_rotation_matrix, :59-97)
template <typename T>
__device__ void quat_rot(const T q_in[4], T R[3][3]) {
  const T n = sqrt(q_in[0] * q_in[0] + q_in[1] * q_in[1] + q_in[2] * q_in[2] + q_in[3] * q_in[3]);
  const T inv = T(1) / (n > T(1e-12) ? n : T(1e-12));
  const T w = q_in[0] * inv, x = q_in[1] * inv, y = q_in[2] * inv, z = q_in[3] * inv;
  R[0][0] = 1 - 2 * (y * y + z * z); R[0][1] = 2 * (x * y - z * w); R[0][2] = 2 * (x * z + y * w);
  R[1][0] = 2 * (x * y + z * w); R[1][1] = 1 - 2 * (x * x + z * z); R[1][2] = 2 * (y * z - x * w);
  R[2][0] = 2 * (x * z - y * w); R[2][1] = 2 * (y * z + x * w); R[2][2] = 1 - 2 * (x * x + y * y);
}

// Four lanes per pair: the points shared out, the two clouds' eigensolves side by side, one
// PCA seed per lane, and the seeds written by turns (64 and 48 consecutive bytes per round).
// Bound by the fp64 chains (eigensolves, acos / sin / cos): a thread per pair ran six
// eigensolves one after the other and wrote 16-byte rows 28 S bytes apart.  One B200: 1 pair
// of 30 atoms, 50 seeds 42 -> 22 us; 100 000 pairs, 20 seeds 226 -> 127 us (80 registers: 6 CTAs;
// 156 us at 96, 175 us at 114); 1024 surface pairs, 50 seeds 188 -> 65 us.
__global__ void __launch_bounds__(128, 6) seeds_kernel(
    const float4* __restrict__ rp, const int* __restrict__ roff, const Pts fp,
    const int* __restrict__ foff, const int* __restrict__ pair_ref,
    const int* __restrict__ pair_fit, int P, int S, const float* __restrict__ fibo, int n_fibo,
    float* __restrict__ sq, float* __restrict__ st) {
  const int lane = threadIdx.x % kLanes;
  const long long at = ((long long)blockIdx.x * blockDim.x + threadIdx.x) / kLanes;
  const bool active = at < P;   // lanes past the last pair shadow it
  const int pi = active ? (int)at : P - 1;
  float* oq = sq + (size_t)pi * S * 4;
  float* ot = st + (size_t)pi * S * 3;
  if (S == 1) {
    if (active) {
      oq[lane] = lane == 0 ? 1.f : 0.f;
      if (lane < 3) ot[lane] = 0.f;
    }
    return;
  }
  const int ri = pair_ref[pi], fi = pair_fit[pi];
  const Pts A(rp + roff[ri]);
  const Pts B = fp + foff[fi];
  const int N = roff[ri + 1] - roff[ri], M = foff[fi + 1] - foff[fi];
  // centroids are the COM of the translations
  float rc[3], fc[3];
  bool ref_ok, fit_ok;
  M3 Ir, If;
  cloud_moments(A, N, lane, rc, ref_ok, Ir);
  cloud_moments(B, M, lane, fc, fit_ok, If);
  const bool valid = N >= 3 && M >= 3 && ref_ok && fit_ok;
  M3 axes;   // reference axes on even lanes, fit axes (before any rotation) on odd ones
  {
    M3 own;
#pragma unroll
    for (int i = 0; i < 3; ++i)
#pragma unroll
      for (int j = 0; j < 3; ++j) own.m[i][j] = lane % 2 ? If.m[i][j] : Ir.m[i][j];
    sym3x3_axes(own, axes);
  }
  float raxf[3][3];   // reference axes, float32
  float pq[4];        // this lane's PCA seed
  {
    double rax[2][3], fax0[3];
#pragma unroll
    for (int a = 0; a < 3; ++a)
#pragma unroll
      for (int c = 0; c < 3; ++c) {
        const double s = from_lane(axes.m[a][c], 0);
        raxf[a][c] = (float)s;
        // sign flips of seed v = lane: axis 0 for v = 1, axis 1 for v = 2, both for v = 3
        if (a < 2) rax[a][c] = (lane == a + 1 || lane == 3) ? -s : s;
        if (a == 0) fax0[c] = from_lane(axes.m[0][c], 1);
      }
    double qo[2][4];
    M3 Irot;
#pragma unroll
    for (int ax = 0; ax < 2; ++ax) {
      double v1[3];
      if (ax == 0) {
        v1[0] = fax0[0]; v1[1] = fax0[1]; v1[2] = fax0[2];
      } else {
        M3 cur;   // fit axes of the rotated fit cloud
        sym3x3_axes(Irot, cur);
        v1[0] = cur.m[1][0]; v1[1] = cur.m[1][1]; v1[2] = cur.m[1][2];
      }
      const double* v2 = rax[ax];
      double cs = v1[0] * v2[0] + v1[1] * v2[1] + v1[2] * v2[2];
      cs = fmin(fmax(cs, -1.0), 1.0);
      const double ang = acos(cs);
      double axis[3] = {v1[1] * v2[2] - v1[2] * v2[1], v1[2] * v2[0] - v1[0] * v2[2],
                        v1[0] * v2[1] - v1[1] * v2[0]};
      const double an = sqrt(axis[0] * axis[0] + axis[1] * axis[1] + axis[2] * axis[2]);
      if (an < 1e-8) {
        axis[0] = 1.0; axis[1] = 0.0; axis[2] = 0.0;
      } else {
        const double inv = 1.0 / fmax(an, 1e-12);
        axis[0] *= inv; axis[1] *= inv; axis[2] *= inv;
      }
      const double h = ang * 0.5, sh = sin(h);
      qo[ax][0] = cos(h); qo[ax][1] = axis[0] * sh; qo[ax][2] = axis[1] * sh; qo[ax][3] = axis[2] * sh;
      if (ax == 0) {  // inertia of the rotated cloud: R I R^T
        double R[3][3];
        quat_rot<double>(qo[0], R);
        double T[3][3];
#pragma unroll
        for (int i = 0; i < 3; ++i)
#pragma unroll
          for (int j = 0; j < 3; ++j)
            T[i][j] = R[i][0] * If.m[0][j] + R[i][1] * If.m[1][j] + R[i][2] * If.m[2][j];
#pragma unroll
        for (int i = 0; i < 3; ++i)
#pragma unroll
          for (int j = 0; j < 3; ++j)
            Irot.m[i][j] = T[i][0] * R[j][0] + T[i][1] * R[j][1] + T[i][2] * R[j][2];
      }
    }
    double qq[4];
    quat_mul<double>(qo[1], qo[0], qq);
#pragma unroll
    for (int c = 0; c < 4; ++c) pq[c] = (float)qq[c];
  }
  float p0[4];   // the first PCA seed, which the structured seeds turn
#pragma unroll
  for (int c = 0; c < 4; ++c) p0[c] = from_lane(pq[c], 0);
  if (!active) return;

  const int n_struct = min(max(S - 5, 0), 6);
  const bool wide = (reinterpret_cast<size_t>(sq) & 15) == 0;   // every row is 16 S bytes on
  // normalise seed n and write it with its COM-aligning translation
  auto write = [&](int n, float q[4]) {
    const float nn = sqrtf(q[0] * q[0] + q[1] * q[1] + q[2] * q[2] + q[3] * q[3]);
    const float inv = 1.f / fmaxf(nn, 1e-12f);
#pragma unroll
    for (int c = 0; c < 4; ++c) q[c] *= inv;
    if (wide) {
      reinterpret_cast<float4*>(oq)[n] = make_float4(q[0], q[1], q[2], q[3]);
    } else {
#pragma unroll
      for (int c = 0; c < 4; ++c) oq[n * 4 + c] = q[c];
    }
    if (valid) {
      float R[3][3];
      quat_rot<float>(q, R);
#pragma unroll
      for (int r = 0; r < 3; ++r)
        ot[n * 3 + r] = rc[r] - (R[r][0] * fc[0] + R[r][1] * fc[1] + R[r][2] * fc[2]);
    } else {
#pragma unroll
      for (int r = 0; r < 3; ++r) ot[n * 3 + r] = rc[r] - fc[r];
    }
  };
  for (int n = lane; n < S; n += kLanes) {
    float q[4] = {1.f, 0.f, 0.f, 0.f};   // seed 0, and fill beyond the Fibonacci table
    const int s = n - 5;
    if (!valid) {
      // fixed fallback rotations (_common.py:189-204), cycled
      const float s2 = 0.70710678118654757f;
      const int f = n % 10;
      q[0] = f == 0 ? 1.f : f >= 4 && f <= 6 ? s2 : 0.f;
      q[1] = f == 1 ? 1.f : f == 4 || f == 7 || f == 8 ? s2 : 0.f;
      q[2] = f == 2 ? 1.f : f == 5 || f == 7 || f == 9 ? s2 : 0.f;
      q[3] = f == 3 ? 1.f : f == 6 || f == 8 || f == 9 ? s2 : 0.f;
    } else if (s >= 0 && s < n_struct) {
      const int a = s / 2;
      const float ch = 0.70710678118654757f, sg = (s % 2 == 0) ? ch : -ch;
      float qa[4] = {ch, 0.f, 0.f, 0.f};
#pragma unroll
      for (int c = 0; c < 3; ++c)
        qa[1 + c] = sg * (a == 0 ? raxf[0][c] : a == 1 ? raxf[1][c] : raxf[2][c]);
      quat_mul_f(qa, p0, q);
    } else if (s >= n_struct && s - n_struct < n_fibo) {
#pragma unroll
      for (int c = 0; c < 4; ++c) q[c] = fibo[(s - n_struct) * 4 + c];
    } else if (n >= 1 && n <= 4) {
      continue;   // the PCA seeds, below
    }
    write(n, q);
  }
  if (valid) write(1 + lane, pq);
}

}  // namespace

int seeds_launch(const float* ref_pts, const int32_t* ref_off, const float* fit_pts,
                 const int32_t* fit_off, const int32_t* pair_ref, const int32_t* pair_fit,
                 int P, int S, const float* fibo, int n_fibo, int fit_f16, float* sq, float* st,
                 cudaStream_t stream) {
  if (P < 0 || S < 1 || S > 64 || (S > 1 && S < 5))
    return set_error(FSS_ERR_INVALID, "fss_seeds: n_seeds must be 1 or in [5, 64]");
  if (n_fibo < 0 || (n_fibo > 0 && !fibo))
    return set_error(FSS_ERR_INVALID, "fss_seeds: bad Fibonacci table");
  if (P == 0) return FSS_OK;
  if (!ref_pts || !ref_off || !fit_pts || !fit_off || !pair_ref || !pair_fit || !sq || !st)
    return set_error(FSS_ERR_INVALID, "fss_seeds: null pointer");
  // one-warp CTAs spread a small batch over the SMs
  const long long lanes = (long long)P * kLanes;
  const int threads = lanes <= 32LL * 8 * num_sms() ? 32 : 128;
  seeds_kernel<<<(unsigned)((lanes + threads - 1) / threads), threads, 0, stream>>>(
      reinterpret_cast<const float4*>(ref_pts), ref_off, Pts(fit_pts, fit_f16 ? 1 : 0), fit_off,
      pair_ref, pair_fit, P, S, fibo, n_fibo, sq, st);
  return check_launch("fss_seeds");
}

}  // namespace fss
