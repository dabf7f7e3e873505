// fss_eval.cu -- single-evaluation kernels on the reference's padded (K, N_pad, 3) layout,
// and the per-step Tanimoto/Adam kernel.  These back the reference-compatible kernel API
// (overlap value + SE(3) gradient per pose) used by parity tests, the step-by-step
// (graph-capturable) driver and the one-launch-per-pair comparator.  The arithmetic is the
// same device code the fused kernel runs (fss_device.cuh).
#include <algorithm>
#include <cmath>

#include "fss_align_spread.cuh"

namespace fss {

namespace {

constexpr int kFewLanes = 8;   // lanes of a pharmacophore pose with a small stage

// Component c (0: V, 1-3: dV/dt, 4-7: dV/dq) of pose `row`.
__device__ __forceinline__ void eval_write(int c, float x, size_t row, int need_grad, float* V,
                                           float* dQ, float* dT) {
  if (c == 0) V[row] = x;
  else if (need_grad && c < 4) dT[row * 3 + c - 1] = x;
  else if (need_grad) dQ[row * 4 + c - 4] = x;
}

// Expanded reference point (stage_ref).
template <bool ESP>
__device__ __forceinline__ void expand_point(float ax, float ay, float az, float ci, float k,
                                             float e, float4* P, float2* Q) {
  float w = -k * (ax * ax + ay * ay + az * az);
  if (ESP) {
    w = fmaf(-e * ci, ci, w);
    *Q = make_float2(2.f * e * ci, 2.f * e * ci);
  }
  const float px = 2.f * k * ax, py = 2.f * k * ay, pz = 2.f * k * az;
  P[0] = make_float4(px, px, py, py);
  P[1] = make_float4(pz, pz, w, w);
}

}  // namespace

// A pose to a CTA of one warp (atom clouds) or two (surfaces, few poses).  A surface is bound by the
// pairwise loop's ex2 and FP32 and wants more warps than one per pose; an atom cloud by the
// instructions and latency around a short loop, where a second warp, or several poses to a warp, gave
// nothing.  The reduction halves the components with the lanes (LanePose), 13 shuffles for 40.  One B200, before
// (a warp a pose, full butterflies) -> after: 1600 poses of 200-400 charged points 129 -> 87 us, 20
// of them 72 -> 35; 12 800 poses of 15-50 atoms 20.3 -> 19.7, 100 of them 4.5 -> 4.2.
template <bool ESP, int WARPS, int UNR>
__global__ void __launch_bounds__(32 * WARPS) overlap_eval_kernel(
    const float* __restrict__ A, const float* __restrict__ B, const float* __restrict__ CA,
    const float* __restrict__ CB, const float* __restrict__ q, const float* __restrict__ t,
    const int* __restrict__ Nr, const int* __restrict__ Mr, int Npad, int Mpad, float k, float e,
    float inv2k, float Kc, float aKc, int need_grad, float* V, float* dQ, float* dT) {
  constexpr int kThreads = 32 * WARPS;
  extern __shared__ __align__(16) float4 smem[];
  __shared__ float red[96];
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const size_t row = blockIdx.x;
  const int N = Nr ? min(max(Nr[row], 0), Npad) : Npad;
  const int M = Mr ? min(max(Mr[row], 0), Mpad) : Mpad;
  float4* sP = smem;
  float4* sB = sP + 2 * Npad;
  float2* sQ = reinterpret_cast<float2*>(sB + Mpad);
  const float* a = A + row * Npad * 3;
  const float* b = B + row * Mpad * 3;
  for (int j = tid; j < M; j += kThreads)
    sB[j] = make_float4(b[3 * j], b[3 * j + 1], b[3 * j + 2], ESP ? CB[row * Mpad + j] : 0.f);
  float3 s = make_float3(0.f, 0.f, 0.f);
  for (int i = tid; i < N; i += kThreads) {
    s.x += a[3 * i]; s.y += a[3 * i + 1]; s.z += a[3 * i + 2];
  }
  s = block_sum3(s, red);
  const float inv = 1.f / (float)(N > 0 ? N : 1);
  const float3 c = make_float3(s.x * inv, s.y * inv, s.z * inv);
  for (int i = tid; i < N; i += kThreads)
    expand_point<ESP>(a[3 * i] - c.x, a[3 * i + 1] - c.y, a[3 * i + 2] - c.z,
                      ESP ? CA[row * Npad + i] : 0.f, k, e, sP + 2 * i, sQ + i);
  __syncthreads();
  float qq[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) qq[i] = q[row * 4 + i];
  const Rot R = quat_to_rot(qq);
  Moments acc;
  acc.zero();
  shape_pose<kThreads, ESP, 2, UNR>(sP, sQ, sB, N, M, tid, R, t[row * 3] - c.x, t[row * 3 + 1] - c.y,
                                  t[row * 3 + 2] - c.z, k, e, inv2k, acc);
  Reduced r;
  r.from(acc, qq);
  float own[1];
  LanePose<32>::reduce(r, lane, own);
  const int id = LanePose<32>::comp(lane, 0);
  const float f = id == 0 ? Kc : aKc;
  if (WARPS == 1) {
    if (lane % 4 == 0) eval_write(id, own[0] * f, row, need_grad, V, dQ, dT);
    return;
  }
  // red was last read before the barrier above
  if (lane % 4 == 0) red[warp * 8 + id] = own[0];
  __syncthreads();
  if (tid < 8) {
    float x = 0.f;
#pragma unroll
    for (int w = 0; w < WARPS; ++w) x += red[w * 8 + tid];
    eval_write(tid, x * (tid == 0 ? Kc : aKc), row, need_grad, V, dQ, dT);
  }
}

// LANES lanes a pose, 32 / LANES poses to a warp: a few features leave most of a warp idle.  Fit
// features visit the reference features of their own type only.  Bound by the latency around short
// loops.  One B200, before (a warp a pose, every reference feature looked at) -> after: 13 000
// poses of 3-20 features 20.9 -> 14.7 us (8 lanes), of 3-70 features 71.1 -> 41.4 (32 lanes).
template <int LANES>
__global__ void __launch_bounds__(32) pharm_eval_kernel(
    const float* __restrict__ A, const float* __restrict__ B, const float* __restrict__ RV,
    const float* __restrict__ FV, const int* __restrict__ At, const int* __restrict__ Bt,
    const float* __restrict__ q, const float* __restrict__ t, const int* __restrict__ Nr,
    const int* __restrict__ Mr, int K, int Npad, int Mpad, int words, PharmTables tab,
    int need_grad, float* O, float* dQ, float* dT) {
  extern __shared__ __align__(16) float4 smem[];
  constexpr int kPoses = 32 / LANES;   // poses of a warp
  const int lane = threadIdx.x % LANES, grp = threadIdx.x / LANES;
  const size_t first = (size_t)blockIdx.x * kPoses;
  const bool active = first + grp < (size_t)K;   // groups past the last pose shadow it
  const size_t row = active ? first + grp : (size_t)K - 1;
  const int N = Nr ? min(max(Nr[row], 0), Npad) : Npad;
  const int M = Mr ? min(max(Mr[row], 0), Mpad) : Mpad;
  float4* sRA = smem + 2 * ((size_t)Npad + Mpad) * grp;
  float4* sRV = sRA + Npad;
  float4* sFA = sRV + Npad;
  float4* sFV = sFA + Mpad;
  // Reference features grouped by type, in their order: bit i of sM[type] marks feature i, so a
  // feature's place is the marks of earlier types and those below its own.  words = 0: left as
  // they are (no room for the marks).
  unsigned* sM = reinterpret_cast<unsigned*>(smem + 2 * ((size_t)Npad + Mpad) * kPoses) +
                 (9 * words + 10) * grp;
  int* off = reinterpret_cast<int*>(sM + 9 * words);
  auto type_of = [](const int* ty, size_t i) {
    const int u = ty[i];
    return (u < 0 || u > 8) ? 8 : u;  // out-of-table types are treated as Dummy
  };
  if (words) {
    for (int i = lane; i < 9 * words; i += LANES) sM[i] = 0;
    __syncwarp();
    for (int i = lane; i < N; i += LANES)
      atomicOr(&sM[type_of(At, row * Npad + i) * words + i / 32], 1u << (i % 32));
    __syncwarp();
    for (int y = lane; y < 10; y += LANES) {
      int n = 0;
      for (int w = 0; w < y * words; ++w) n += __popc(sM[w]);
      off[y] = n;
    }
    __syncwarp();
  }
  auto put = [&](const float* x, const float* v, int u, float4* a, float4* d) {
    *a = make_float4(x[0], x[1], x[2], __int_as_float(u));
    *d = v ? unit4(v[0], v[1], v[2]) : make_float4(0.f, 0.f, 0.f, 0.f);
  };
  for (int i = lane; i < N; i += LANES) {
    const size_t g = row * Npad + i;
    const int u = type_of(At, g);
    int at = i;
    if (words) {
      const unsigned* m = sM + u * words;
      at = off[u] + __popc(m[i / 32] & ((1u << (i % 32)) - 1));
      for (int w = 0; w < i / 32; ++w) at += __popc(m[w]);
    }
    put(A + 3 * g, RV ? RV + 3 * g : nullptr, u, sRA + at, sRV + at);
  }
  for (int j = lane; j < M; j += LANES) {
    const size_t g = row * Mpad + j;
    put(B + 3 * g, FV ? FV + 3 * g : nullptr, type_of(Bt, g), sFA + j, sFV + j);
  }
  __syncwarp();
  float qq[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) qq[i] = q[row * 4 + i];
  const Rot R = quat_to_rot(qq);
  Moments acc;
  acc.zero();
  pharm_pose<LANES>(sRA, sRV, sFA, sFV, N, M, lane, R, t[row * 3], t[row * 3 + 1],
                    t[row * 3 + 2], tab, acc, words ? off : nullptr);
  __syncwarp();
  Reduced r;
  r.from(acc, qq);
  float own[1];
  LanePose<LANES>::reduce(r, lane, own);
  if (active && lane % (LANES / 8) == 0)
    eval_write(LanePose<LANES>::comp(lane, 0), own[0], row, need_grad, O, dQ, dT);
}

__global__ void tanimoto_adam_kernel(const float* __restrict__ V, const float* __restrict__ dQ,
                                     const float* __restrict__ dT, const float* __restrict__ U,
                                     float* q, float* t, float* mq, float* vq, float* mt,
                                     float* vt, float* best, float* bq, float* bt, int K,
                                     float lr) {
  const int r = blockIdx.x * blockDim.x + threadIdx.x;
  if (r >= K) return;
  PoseState s;
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    s.q[i] = q[(size_t)r * 4 + i]; s.mq[i] = mq[(size_t)r * 4 + i];
    s.vq[i] = vq[(size_t)r * 4 + i]; s.bq[i] = bq[(size_t)r * 4 + i];
  }
#pragma unroll
  for (int i = 0; i < 3; ++i) {
    s.t[i] = t[(size_t)r * 3 + i]; s.mt[i] = mt[(size_t)r * 3 + i];
    s.vt[i] = vt[(size_t)r * 3 + i]; s.bt[i] = bt[(size_t)r * 3 + i];
  }
  s.best = best[r];
  float score, scale;
  tanimoto(V[r], U[r], score, scale);
  float gq[4], gt[3];
#pragma unroll
  for (int i = 0; i < 4; ++i) gq[i] = -scale * dQ[(size_t)r * 4 + i];
#pragma unroll
  for (int i = 0; i < 3; ++i) gt[i] = -scale * dT[(size_t)r * 3 + i];
  adam_tail(s, score, gq, gt, lr);
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    q[(size_t)r * 4 + i] = s.q[i]; mq[(size_t)r * 4 + i] = s.mq[i];
    vq[(size_t)r * 4 + i] = s.vq[i]; bq[(size_t)r * 4 + i] = s.bq[i];
  }
#pragma unroll
  for (int i = 0; i < 3; ++i) {
    t[(size_t)r * 3 + i] = s.t[i]; mt[(size_t)r * 3 + i] = s.mt[i];
    vt[(size_t)r * 3 + i] = s.vt[i]; bt[(size_t)r * 3 + i] = s.bt[i];
  }
  best[r] = s.best;
}

int overlap_eval_launch(const float* A, const float* B, const float* CA, const float* CB,
                        const float* q, const float* t, const int32_t* Nr, const int32_t* Mr,
                        int K, int Npad, int Mpad, float alpha, float inv_lam, int need_grad,
                        float* V, float* dQ, float* dT, cudaStream_t st) {
  if (K < 0 || Npad < 0 || Mpad < 0 || !(alpha > 0.f))
    return set_error(FSS_ERR_INVALID, "fss_overlap_grad: bad sizes or alpha");
  if (K == 0) return FSS_OK;
  if (!A || !B || !q || !t || !V || (need_grad && (!dQ || !dT)))
    return set_error(FSS_ERR_INVALID, "fss_overlap_grad: null pointer");
  if ((CA == nullptr) != (CB == nullptr))
    return set_error(FSS_ERR_INVALID, "fss_overlap_grad: give both charge arrays or neither");
  if (Npad > kMaxPoints || Mpad > kMaxPoints)
    return set_error(FSS_ERR_UNSUPPORTED, "fss_overlap_grad: more than fss_max_points() points");
  const bool esp = CA != nullptr;
  const double a = alpha;
  const float k = (float)(0.5 * a * 1.4426950408889634);
  const float e = esp ? (float)((double)inv_lam * 1.4426950408889634) : 0.f;
  const float inv2k = (float)(1.0 / (a * 1.4426950408889634));
  const double Kd = std::pow(M_PI, 1.5) / std::pow(2.0 * a, 1.5);
  const size_t smem = sizeof(float4) * (2 * (size_t)Npad + Mpad + (esp ? (Npad + 1) / 2 : 0));
  // Two warps from 256 fit points on, where each lane has whole register tiles, if the reference is
  // no small one, and above 64 points (below, lanes of the second would have none) while the poses
  // are few.  In us with one and with two: 148 poses of 65 points 4.5 and 3.8, 13 000 of them 24.3
  // and 35.4; of 100 points 6.5 and 5.1, 47.4 and 58.4; 600 charged poses of 200 points 19.1 and
  // 16.5, 6000 72 and 88; 3000 of 300 points 92 and 77; 13 000 of 400 against 30 points 48.8 and 55.3.
  const bool wide = Mpad > 64 && ((Mpad >= 256 && Npad > 64) || K <= 12 * num_sms());
  // One warp: the loop unrolled twice instead of four times needs fewer registers (more poses on
  // an SM) and pays for small clouds in large batches (four times, twice): 13 000 poses of 30 points
  // 14.7 and 14.1 us,
  // charged 17.1 and 16.0; 600 of 50 points 4.7 and 4.9.
  const bool few = K <= (esp ? 16 : 24) * num_sms() || Npad > 100;
  const auto kern = esp ? (wide ? overlap_eval_kernel<true, 2, 4>
                           : few ? overlap_eval_kernel<true, 1, 4> : overlap_eval_kernel<true, 1, 2>)
                        : (wide ? overlap_eval_kernel<false, 2, 4>
                           : few ? overlap_eval_kernel<false, 1, 4> : overlap_eval_kernel<false, 1, 2>);
  const cudaError_t ce =
      cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (ce != cudaSuccess)
    return set_error(FSS_ERR_CUDA, std::string("fss_overlap_grad: ") + cudaGetErrorString(ce));
  kern<<<K, wide ? 64 : 32, smem, st>>>(A, B, CA, CB, q, t, Nr, Mr, Npad, Mpad, k, e, inv2k,
                                        (float)Kd, (float)(a * Kd), need_grad, V, dQ, dT);
  return check_launch("fss_overlap_grad");
}

int pharm_eval_launch(const float* A, const float* B, const float* RV, const float* FV,
                      const int32_t* At, const int32_t* Bt, const float* q, const float* t,
                      const int32_t* Nr, const int32_t* Mr, int K, int Npad, int Mpad,
                      int directional, int need_grad, float* O, float* dQ, float* dT,
                      cudaStream_t st) {
  if (K < 0 || Npad < 0 || Mpad < 0) return set_error(FSS_ERR_INVALID, "fss_pharm_grad: bad sizes");
  if (K == 0) return FSS_OK;
  if (!A || !B || !At || !Bt || !q || !t || !O || (need_grad && (!dQ || !dT)))
    return set_error(FSS_ERR_INVALID, "fss_pharm_grad: null pointer");
  if (directional && (!RV || !FV))
    return set_error(FSS_ERR_INVALID, "fss_pharm_grad: directional scoring needs vectors");
  if (Npad > kMaxPoints || Mpad > kMaxPoints)
    return set_error(FSS_ERR_UNSUPPORTED, "fss_pharm_grad: more than fss_max_points() features");
  int dev = 0, optin = 0, sms = 0;
  cudaError_t ce = cudaGetDevice(&dev);
  if (ce == cudaSuccess)
    ce = cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
  if (ce == cudaSuccess) ce = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  if (ce != cudaSuccess)
    return set_error(FSS_ERR_CUDA, std::string("fss_pharm_grad: ") + cudaGetErrorString(ce));
  // the largest feature lists leave no room to group them by type
  int words = (Npad + 31) / 32;
  auto bytes = [&] {
    return sizeof(float4) * 2 * ((size_t)Npad + Mpad) +
           (words ? sizeof(int) * (9 * (size_t)words + 10) : 0);
  };
  if (bytes() > (size_t)optin) words = 0;
  const size_t stage = bytes();
  // Eight lanes a pose up to four fit features per lane and from one full wave of one-warp CTAs
  // on; in us with 8 and with 32 lanes: 13 000 poses of 3-20 features 14.7 and 22.3, 3-30 19.9 and
  // 23.2, 3-45 42.9 and 31.0; 100 poses of 3-20 10.4 and 5.5.
  constexpr int kPoses = 32 / kFewLanes;
  const bool small = Npad <= 32 && Mpad <= 32 && K > 32 * sms;
  const int per_cta = small ? kPoses : 1;
  const size_t smem = per_cta * stage;
  const auto kern = small ? pharm_eval_kernel<kFewLanes> : pharm_eval_kernel<32>;
  ce = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (ce != cudaSuccess)
    return set_error(FSS_ERR_CUDA, std::string("fss_pharm_grad: ") + cudaGetErrorString(ce));
  kern<<<(K - 1) / per_cta + 1, 32, smem, st>>>(
      A, B, directional ? RV : nullptr, directional ? FV : nullptr, At, Bt, q, t, Nr, Mr, K, Npad,
      Mpad, words, make_pharm_tables(directional != 0), need_grad, O, dQ, dT);
  return check_launch("fss_pharm_grad");
}

int tanimoto_adam_launch(const float* V, const float* dQ, const float* dT, const float* U,
                         float* q, float* t, float* mq, float* vq, float* mt, float* vt,
                         float* best, float* bq, float* bt, int K, float lr, cudaStream_t st) {
  if (K < 0) return set_error(FSS_ERR_INVALID, "fss_tanimoto_adam_step: K < 0");
  if (K == 0) return FSS_OK;
  if (!V || !dQ || !dT || !U || !q || !t || !mq || !vq || !mt || !vt || !best || !bq || !bt)
    return set_error(FSS_ERR_INVALID, "fss_tanimoto_adam_step: null pointer");
  tanimoto_adam_kernel<<<(K + 127) / 128, 128, 0, st>>>(V, dQ, dT, U, q, t, mq, vq, mt, vt,
                                                        best, bq, bt, K, lr);
  return check_launch("fss_tanimoto_adam_step");
}

}  // namespace fss
