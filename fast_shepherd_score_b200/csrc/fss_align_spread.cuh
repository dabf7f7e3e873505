// fss_align_spread.cuh -- the fused persistent alignment kernel for poses of 4 or more lanes.
//
// Same work items, staging and arithmetic as align_kernel (fss_align_kernel.cuh), which keeps
// what launch_align lists.  Two things differ:
//
//  * A pose's optimiser state is spread over its lanes (LanePose) instead of being replicated
//    in every lane and parked in shared memory: per step one Adam update per component instead
//    of seven in each lane, 19 shuffles instead of 24, and none of the 44 shared-memory
//    accesses.
//  * The fit points left over after the full register tiles share the last tile's loop over the
//    reference points (pose_tile) instead of running loops of their own: 5 points per lane are
//    one loop, not one of four points and one of a single point with nothing to overlap.
//
// A tile's results are the bits align_kernel gives: an alignment amplifies one last bit to another
// optimum within some thirty steps, and one oversized molecule changes the kernel for all pairs of
// a launch.  The pairwise sums, the reduction, the rotation and the update of each component have
// their roundings written out (__fmaf_rn and the like).  The rest is plain arithmetic as in
// align_kernel: the sums of four products in update, the scores and gradients of combo and
// esp_combo, and what both kernels share (quat_grad_from_moment, pharm_pose, esp_side).  There the
// equality rests on the compiler contracting the same expressions alike; it holds for nvcc 12.9 and
// is what tests/test_gpu_spread.py and test_gpu_spread_far.py compare.
#pragma once
#include "fss_align_kernel.cuh"

namespace fss {

// quat_to_rot with its roundings written out.
__device__ __forceinline__ Rot quat_to_rot_rn(const float q[4]) {
  const float qr = q[0], qi = q[1], qj = q[2], qk = q[3];
  const float jj = __fmul_rn(qj, qj), kk = __fmul_rn(qk, qk), kr = __fmul_rn(qk, qr),
              ik = __fmul_rn(qi, qk), ir = __fmul_rn(qi, qr);
  Rot R;
  R.r[0] = __fmaf_rn(-2.f, __fadd_rn(jj, kk), 1.f);
  R.r[1] = 2.f * __fmaf_rn(qi, qj, -kr);
  R.r[2] = 2.f * __fmaf_rn(qj, qr, ik);
  R.r[3] = 2.f * __fmaf_rn(qi, qj, kr);
  R.r[4] = __fmaf_rn(-2.f, __fmaf_rn(qi, qi, kk), 1.f);
  R.r[5] = 2.f * __fmaf_rn(qj, qk, -ir);
  R.r[6] = 2.f * __fmaf_rn(-qj, qr, ik);
  R.r[7] = 2.f * __fmaf_rn(qj, qk, ir);
  R.r[8] = __fmaf_rn(-2.f, __fmaf_rn(qi, qi, jj), 1.f);
  return R;
}

// ---------------------------------------------------------------------------------------
// Pose state spread over a pose's lanes.
//
// The eight reduced values of a step (0: V, 1-3: dV/dt, 4-7: dV/dq) and the pose's seven
// parameters (t as 1-3, q as 4-7) share one numbering, and lane l owns component
// l / (LPP / 8) (LPP = 4: components 2 l and 2 l + 1): its Adam moments, its current and its
// best parameter live in that lane's registers.  A step reduces by halves -- 7 shuffles for
// the 8 values, in the butterfly's pairing -- and q and t are gathered back for the next
// rotation.
// ---------------------------------------------------------------------------------------
template <int LPP>
struct LanePose {
  static_assert(LPP >= 4 && LPP <= 32, "replicated state below 4 lanes a pose");
  static constexpr int NV = LPP >= 8 ? 1 : 8 / LPP;   // components a lane owns
  float q[4], t[3];                                   // every lane: the pose of this step
  float par[NV], m[NV], v[NV], bpar[NV], best;

  static __device__ __forceinline__ int comp(int lane, int k) {
    return LPP >= 8 ? lane / (LPP >= 8 ? LPP / 8 : 1) : lane * NV + k;
  }
  // component c of a lane-owned array, in every lane of the pose
  static __device__ __forceinline__ float gather(const float (&a)[NV], int c) {
    return __shfl_sync(0xffffffffu, a[c % NV], LPP >= 8 ? c * (LPP / 8) : c / NV, LPP);
  }
  // totals of the lane's components over the pose's lanes, from each lane's partial sums
  static __device__ __forceinline__ void reduce(const Reduced& r, int lane, float (&own)[NV]) {
    float a[8] = {r.v, r.f[0], r.f[1], r.f[2], r.dq[0], r.dq[1], r.dq[2], r.dq[3]};
    int n = 8;
#pragma unroll
    for (int o = LPP / 2; o > 0; o >>= 1) {
      if (n > NV) {
        n /= 2;
        const bool hi = lane & o;
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          if (k < n) {
            const float send = hi ? a[k] : a[k + n];
            const float keep = hi ? a[k + n] : a[k];
            a[k] = __fadd_rn(keep, __shfl_xor_sync(0xffffffffu, send, o));
          }
        }
      } else {
#pragma unroll
        for (int k = 0; k < NV; ++k)
          a[k] = __fadd_rn(a[k], __shfl_xor_sync(0xffffffffu, a[k], o));
      }
    }
#pragma unroll
    for (int k = 0; k < NV; ++k) own[k] = a[k];
  }
  // value by sv, forces and quaternion gradient by sf
  static __device__ __forceinline__ void scale(float (&own)[NV], int lane, float sv, float sf) {
#pragma unroll
    for (int k = 0; k < NV; ++k) own[k] = __fmul_rn(own[k], comp(lane, k) == 0 ? sv : sf);
  }
  __device__ __forceinline__ void init(const float* seed_q, const float* seed_t, float3 c,
                                       int lane) {
#pragma unroll
    for (int i = 0; i < 4; ++i) q[i] = seed_q[i];
    t[0] = __fsub_rn(seed_t[0], c.x);
    t[1] = __fsub_rn(seed_t[1], c.y);
    t[2] = __fsub_rn(seed_t[2], c.z);
#pragma unroll
    for (int k = 0; k < NV; ++k) {
      const int id = comp(lane, k);
      float p = 0.f;
#pragma unroll
      for (int i = 0; i < 4; ++i) p = id == 4 + i ? q[i] : p;
#pragma unroll
      for (int i = 0; i < 3; ++i) p = id == 1 + i ? t[i] : p;
      par[k] = bpar[k] = p;
      m[k] = 0.f; v[k] = 0.f;
    }
    best = -INFINITY;
  }
  // adam_tail on the lane's components: best tracking with the pre-update pose, tangent
  // projection, Adam, renormalisation, and the new q and t in every lane.  g: the gradient of
  // the loss by component.  SPLIT: a translation's step is rounded before it is subtracted.
  template <bool SPLIT = false>
  __device__ __forceinline__ void update(float score, const float (&g)[NV], int lane, float lr) {
    if (score > best) {  // NaN never replaces the best
      best = score;
#pragma unroll
      for (int k = 0; k < NV; ++k) bpar[k] = par[k];
    }
    float gq[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) gq[i] = gather(g, 4 + i);
    const float radial = gq[0] * q[0] + gq[1] * q[1] + gq[2] * q[2] + gq[3] * q[3];
    const float c1 = 1.f - kBeta1, c2 = 1.f - kBeta2;
#pragma unroll
    for (int k = 0; k < NV; ++k) {
      const bool rot = comp(lane, k) >= 4;
      const float d = rot ? __fmaf_rn(-par[k], radial, g[k]) : g[k];
      const float cd = __fmul_rn(c2, d);
      m[k] = rot ? __fmaf_rn(kBeta1, m[k], __fmul_rn(c1, d))
                 : __fmaf_rn(c1, d, __fmul_rn(kBeta1, m[k]));
      v[k] = rot ? __fmaf_rn(kBeta2, v[k], __fmul_rn(cd, d))
                 : __fmaf_rn(cd, d, __fmul_rn(kBeta2, v[k]));
      const float x = __fmul_rn(lr, m[k]), r = __frsqrt_rn(__fadd_rn(v[k], kAdamEps));
      par[k] = SPLIT && !rot ? __fsub_rn(par[k], __fmul_rn(x, r)) : __fmaf_rn(-x, r, par[k]);
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) q[i] = gather(par, 4 + i);
#pragma unroll
    for (int i = 0; i < 3; ++i) t[i] = gather(par, 1 + i);
    const float n2 = q[0] * q[0] + q[1] * q[1] + q[2] * q[2] + q[3] * q[3];
    const float inv = __frsqrt_rn(fmaxf(n2, 1e-24f));
#pragma unroll
    for (int i = 0; i < 4; ++i) q[i] = __fmul_rn(q[i], inv);
#pragma unroll
    for (int k = 0; k < NV; ++k)
      if (comp(lane, k) >= 4) par[k] = __fmul_rn(par[k], inv);
  }
  // Tanimoto V / (U - V) and its derivative's scale
  static __device__ __forceinline__ void tanimoto_rn(float V, float U, float& score, float& scl) {
    float denom = __fsub_rn(U, V);
    if (denom == 0.f) denom = 1e-12f;
    const float r = __frcp_rn(denom);
    score = __fmul_rn(V, r);
    scl = __fmul_rn(__fmul_rn(U, r), r);
  }
  // step_single, step_tversky, step_combo and step_esp_combo of the replicated form
  template <bool SPLIT = false>
  __device__ __forceinline__ void single(const float (&own)[NV], int lane, float U, float lr) {
    float score, scl, g[NV];
    tanimoto_rn(gather(own, 0), U, score, scl);
#pragma unroll
    for (int k = 0; k < NV; ++k) g[k] = __fmul_rn(-scl, own[k]);
    update<SPLIT>(score, g, lane, lr);
  }
  template <bool SPLIT = false>
  __device__ __forceinline__ void tversky(const float (&own)[NV], int lane, float D, float lr) {
    const float V = gather(own, 0);
    const float score = D > 1e-8f ? fminf(V / D, 1.f) : 0.f;
    const float scl = V < D ? 1.f / D : 0.f;
    float g[NV];
#pragma unroll
    for (int k = 0; k < NV; ++k) g[k] = __fmul_rn(-scl, own[k]);
    update<SPLIT>(score, g, lane, lr);
  }
  __device__ __forceinline__ void combo(const float (&os)[NV], float Us, const float (&oc)[NV],
                                        float Uc, float w, int lane, float lr) {
    float ss, scs, sc, scc, g[NV];
    tanimoto_rn(gather(os, 0), Us, ss, scs);
    tanimoto_rn(gather(oc, 0), Uc, sc, scc);
    const float score = (1.f - w) * ss + w * sc;
    const float cs = -(1.f - w) * scs, cc = -w * scc;
#pragma unroll
    for (int k = 0; k < NV; ++k) g[k] = cs * os[k] + cc * oc[k];
    update(score, g, lane, lr);
  }
  __device__ __forceinline__ void esp_combo(const float (&own)[NV], int lane, float U,
                                            float esp_sum, float n_surf, float w, bool scored,
                                            float lr) {
    float vs, scl, g[NV];
    tanimoto_rn(gather(own, 0), U, vs, scl);
    const float score = scored ? w * (esp_sum / n_surf) + (1.f - w) * vs : -INFINITY;
    const float c = -scl * (1.f - w);
#pragma unroll
    for (int k = 0; k < NV; ++k) g[k] = __fmul_rn(c, own[k]);
    update(score, g, lane, lr);
  }
  // best score and pose; c: the centroid the poses were moved to
  __device__ __forceinline__ void write(int lane, float3 c, float* score, float* oq,
                                        float* ot) const {
    if (lane == 0) *score = best;
    if (LPP > 8 && lane % (LPP >= 8 ? LPP / 8 : 1) != 0) return;
#pragma unroll
    for (int k = 0; k < NV; ++k) {
      const int id = comp(lane, k);
      if (id >= 4) oq[id - 4] = bpar[k];
      else if (id >= 1) ot[id - 1] = __fadd_rn(bpar[k], id == 1 ? c.x : id == 2 ? c.y : c.z);
    }
  }
};

// ---------------------------------------------------------------------------------------
// Shape / ESP sums of a pose
// ---------------------------------------------------------------------------------------
struct ShapeArgs {
  const float4* sPd;   // staged reference cloud (stage_ref)
  const float2* sQd;
  const float4* sB;    // fit cloud, body frame
  int N, M;
  float tx, ty, tz, k, e, inv2k;
};

// One fit point in the reference frame, and its part of the exponent (positive).
template <bool ESP>
__device__ __forceinline__ void pose_point(const ShapeArgs& a, const Rot& R, int j, float4& b,
                                           float& x, float& y, float& z, float& w) {
  b = j < a.M ? a.sB[j] : make_float4(0.f, 0.f, 0.f, 0.f);
  const float3 p = rot_apply(R, b.x, b.y, b.z);
  x = __fadd_rn(p.x, a.tx); y = __fadd_rn(p.y, a.ty); z = __fadd_rn(p.z, a.tz);
  w = __fmul_rn(a.k, __fmaf_rn(z, z, __fmaf_rn(x, x, __fmul_rn(y, y))));
  if (ESP) w = __fmaf_rn(__fmul_rn(a.e, b.w), b.w, w);
}

// A point's sums into the pose's moments (scaled by 2^-w unless the exponent was unfactored).
__device__ __forceinline__ void add_point(Moments& acc, float inv2k, float4 b, float x, float y,
                                          float z, float g, float gx, float gy, float gz) {
  acc.v = __fadd_rn(acc.v, g);
  acc.add_force(__fmaf_rn(gx, inv2k, __fmul_rn(-x, g)), __fmaf_rn(gy, inv2k, __fmul_rn(-y, g)),
                __fmaf_rn(gz, inv2k, __fmul_rn(-z, g)), b.x, b.y, b.z);
}

// COUNT points per lane (j0 + u * LPP) with the unfactored exponent.
template <int LPP, bool ESP, int COUNT, int UNR>
__device__ __forceinline__ void far_points(const ShapeArgs& a, const Rot& R, int j0,
                                           Moments& acc) {
  float4 b[COUNT];
  float x[COUNT], y[COUNT], z[COUNT], w[COUNT], sg[COUNT], sx[COUNT], sy[COUNT], sz[COUNT];
#pragma unroll
  for (int u = 0; u < COUNT; ++u) {
    pose_point<ESP>(a, R, j0 + u * LPP, b[u], x[u], y[u], z[u], w[u]);
    sg[u] = sx[u] = sy[u] = sz[u] = 0.f;
  }
#pragma unroll UNR
  for (int i = 0; i < a.N; ++i) {
    const float4 p = a.sPd[2 * i], r = a.sPd[2 * i + 1];
    float qc = 0.f;
    if (ESP) qc = a.sQd[i].x;
#pragma unroll
    for (int u = 0; u < COUNT; ++u) {
      float E = __fmaf_rn(p.x, x[u],
                          __fmaf_rn(p.z, y[u], __fmaf_rn(r.x, z[u], __fsub_rn(r.z, w[u]))));
      if (ESP) E = __fmaf_rn(qc, b[u].w, E);
      const float g = ex2(E);
      sg[u] = __fadd_rn(sg[u], g);
      sx[u] = __fmaf_rn(g, p.x, sx[u]);
      sy[u] = __fmaf_rn(g, p.z, sy[u]);
      sz[u] = __fmaf_rn(g, r.x, sz[u]);
    }
  }
#pragma unroll
  for (int u = 0; u < COUNT; ++u)
    if (j0 + u * LPP < a.M)
      add_point(acc, a.inv2k, b[u], x[u], y[u], z[u], sg[u], sx[u], sy[u], sz[u]);
}

// Fit points of a lane in the reference frame: NP f32x2 pairs and an odd one.
template <int NP>
struct TilePoints {
  static constexpr int kPairs = NP > 0 ? NP : 1;
  float2 x[kPairs], y[kPairs], z[kPairs], c[kPairs], w[kPairs];
  float ox, oy, oz, oc, ow;
};

// One loop over the reference points for pairs V0 .. V0 + NP of a tile with the factored
// exponent, and (PL) its odd point with the unfactored one, which needs no 2^-w.
template <int LPP, bool ESP, int V0, int NP, bool PL, int UNR, int TP>
__device__ __forceinline__ void near_points(const ShapeArgs& a, const TilePoints<TP>& t, int j0,
                                            Moments& acc) {
  constexpr int T = 2 * NP + (PL ? 1 : 0);
  float2 sg[NP > 0 ? NP : 1], sx[NP > 0 ? NP : 1], sy[NP > 0 ? NP : 1], sz[NP > 0 ? NP : 1];
  float og = 0.f, ogx = 0.f, ogy = 0.f, ogz = 0.f;
#pragma unroll
  for (int v = 0; v < NP; ++v) sg[v] = sx[v] = sy[v] = sz[v] = f2(0.f, 0.f);
#pragma unroll UNR
  for (int i = 0; i < a.N; ++i) {
    const float4 p = a.sPd[2 * i], r = a.sPd[2 * i + 1];
    const float2 PX = f2(p.x, p.y), PY = f2(p.z, p.w), PZ = f2(r.x, r.y), PW = f2(r.z, r.w);
    float2 QC;
    if (ESP) QC = a.sQd[i];
#pragma unroll
    for (int v = 0; v < NP; ++v) {
      float2 E = __ffma2_rn(PX, t.x[V0 + v],
                            __ffma2_rn(PY, t.y[V0 + v], __ffma2_rn(PZ, t.z[V0 + v], PW)));
      if (ESP) E = __ffma2_rn(QC, t.c[V0 + v], E);
      const float2 g = f2(ex2(E.x), ex2(E.y));
      sg[v] = __fadd2_rn(sg[v], g);
      sx[v] = __ffma2_rn(g, PX, sx[v]);
      sy[v] = __ffma2_rn(g, PY, sy[v]);
      sz[v] = __ffma2_rn(g, PZ, sz[v]);
    }
    if (PL) {
      float E = __fmaf_rn(PX.x, t.ox,
                          __fmaf_rn(PY.x, t.oy, __fmaf_rn(PZ.x, t.oz, __fsub_rn(PW.x, t.ow))));
      if (ESP) E = __fmaf_rn(QC.x, t.oc, E);
      const float g = ex2(E);
      og = __fadd_rn(og, g);
      ogx = __fmaf_rn(g, PX.x, ogx);
      ogy = __fmaf_rn(g, PY.x, ogy);
      ogz = __fmaf_rn(g, PZ.x, ogz);
    }
  }
#pragma unroll
  for (int u = 0; u < T; ++u) {
    const int j = j0 + (2 * V0 + u) * LPP;
    if (j < a.M) {
      const float4 b = a.sB[j];
      if (PL && u == T - 1) {
        add_point(acc, a.inv2k, b, t.ox, t.oy, t.oz, og, ogx, ogy, ogz);
      } else {
        const int v = u / 2, f = V0 + v;
        const bool h = u % 2;
        const float s = ex2(-(h ? t.w[f].y : t.w[f].x));
        add_point(acc, a.inv2k, b, h ? t.x[f].y : t.x[f].x, h ? t.y[f].y : t.y[f].x,
                  h ? t.z[f].y : t.z[f].x, __fmul_rn(h ? sg[v].y : sg[v].x, s),
                  __fmul_rn(h ? sx[v].y : sx[v].x, s), __fmul_rn(h ? sy[v].y : sy[v].x, s),
                  __fmul_rn(h ? sz[v].y : sz[v].x, s));
      }
    }
  }
}

// A register tile: NP pairs of fit points per lane and an odd point (PL).  GROUP points are voted
// together: a group with a far point (k |b'|^2 beyond kFactorMax in any lane of the pose) is
// unfactored as a whole.  Molecules and surfaces longer than about 25 A have such poses at every
// step, so this path runs as many points as the tile has, inline.  A tile of one group takes
// far_points with all its points; in a tile of two groups the poses of a warp can be far in the
// one, the other or both, so as soon as one is, the groups run one after the other: a warp then has
// two ways to go at a time, not four.  One B200, molecules of 15-50 atoms stretched to 31 A, 50 x
// 100, align_kernel -> here: 1024 pairs 4.88 -> 4.29 ms (8 lanes), 5.10 -> 4.30 (16 lanes); 2048 ESP
// pairs 11.4 -> 10.6 ms (4 lanes).  An out-of-line function for four points, padded to that many
// and taken by the whole tile, ran them in 6.92, 9.51 and 13.7 ms.
template <int LPP, bool ESP, int NP, bool PL, int GROUP, int UNR, int FAR>
__device__ __forceinline__ void pose_tile(const ShapeArgs& a, const Rot& R, int j0, Moments& acc) {
  constexpr int T = 2 * NP + (PL ? 1 : 0);
  constexpr int NG = (2 * NP + GROUP - 1) / GROUP;
  static_assert(NG <= 2, "one or two groups a tile");
  TilePoints<NP> t;
  bool far[NG > 0 ? NG : 1] = {};
#pragma unroll
  for (int v = 0; v < NP; ++v) {
    float x[2], y[2], z[2], c[2], w[2];
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const int j = j0 + (2 * v + h) * LPP;
      float4 b;
      pose_point<ESP>(a, R, j, b, x[h], y[h], z[h], w[h]);
      c[h] = b.w;
      far[2 * v / GROUP] = far[2 * v / GROUP] || (j < a.M && w[h] > kFactorMax);
    }
    t.x[v] = f2(x[0], x[1]); t.y[v] = f2(y[0], y[1]); t.z[v] = f2(z[0], z[1]);
    t.c[v] = f2(c[0], c[1]); t.w[v] = f2(w[0], w[1]);
  }
  if (PL) {
    float4 b;
    const int j = j0 + 2 * NP * LPP;
    pose_point<ESP>(a, R, j, b, t.ox, t.oy, t.oz, t.ow);
    t.oc = b.w;
    t.ow = j < a.M ? t.ow : INFINITY;
  }
  if constexpr (NG > 0) {
    // vote of this pose's lanes only: its path must not depend on the poses it shares a warp with
    const unsigned own = LPP >= 32 ? 0xffffffffu
                                   : ((1u << (LPP & 31)) - 1u) << ((threadIdx.x & 31) & ~(LPP - 1));
    unsigned any = 0;   // in any pose of the warp
#pragma unroll
    for (int g = 0; g < NG; ++g) {
      const unsigned vote = __ballot_sync(0xffffffffu, far[g]);
      far[g] = (vote & own) != 0;
      any |= vote;
    }
    if constexpr (NG == 1) {
      if (far[0]) {
        far_points<LPP, ESP, T, FAR>(a, R, j0, acc);
        return;
      }
    } else if (any) {
      constexpr int kRest = 2 * NP - GROUP;
      if (far[0]) far_points<LPP, ESP, GROUP, FAR>(a, R, j0, acc);
      else near_points<LPP, ESP, 0, GROUP / 2, false, UNR>(a, t, j0, acc);
      __syncwarp();
      if (far[1]) far_points<LPP, ESP, kRest, FAR>(a, R, j0 + GROUP * LPP, acc);
      else near_points<LPP, ESP, GROUP / 2, kRest / 2, false, UNR>(a, t, j0, acc);
      if (PL) far_points<LPP, ESP, 1, FAR>(a, R, j0 + 2 * NP * LPP, acc);
      return;
    }
  }
  near_points<LPP, ESP, 0, NP, PL, UNR>(a, t, j0, acc);
}

// All fit points of a pose: register tiles of GROUP points per lane, the last of them together
// with points left over (TAIL at most).
template <int LPP, bool ESP, int GROUP, int TAIL, int UNR, int FAR>
__device__ __forceinline__ void pose_sums(const ShapeArgs& a, const Rot& R, int lane,
                                          Moments& acc) {
  int left = (a.M + LPP - 1) / LPP;   // points per lane
  int j = lane;
  for (; left > TAIL; left -= GROUP, j += GROUP * LPP)
    pose_tile<LPP, ESP, GROUP / 2, false, GROUP, UNR, FAR>(a, R, j, acc);
  switch (left) {
    case 1: pose_tile<LPP, ESP, 0, true, GROUP, UNR, FAR>(a, R, j, acc); break;
    case 2: pose_tile<LPP, ESP, 1, false, GROUP, UNR, FAR>(a, R, j, acc); break;
    case 3: pose_tile<LPP, ESP, 1, true, GROUP, UNR, FAR>(a, R, j, acc); break;
    case 4: pose_tile<LPP, ESP, 2, false, GROUP, UNR, FAR>(a, R, j, acc); break;
    case 5: if (TAIL >= 5) pose_tile<LPP, ESP, 2, true, GROUP, UNR, FAR>(a, R, j, acc); break;
    case 6: if (TAIL >= 6) pose_tile<LPP, ESP, 3, false, GROUP, UNR, FAR>(a, R, j, acc); break;
    case 7: if (TAIL >= 7) pose_tile<LPP, ESP, 3, true, GROUP, UNR, FAR>(a, R, j, acc); break;
    case 8: if (TAIL >= 8) pose_tile<LPP, ESP, 4, false, GROUP, UNR, FAR>(a, R, j, acc); break;
    default: break;
  }
}

// Registers, the largest last tile and the unroll of a tile's loop.  168 registers keep 12 warps
// on an SM, 128 keep 16, 96 keep 20.
//  * shape, ESP: 168 -- with a few rounds of CTAs the largest pair's serial chain of steps decides
//    the time, and runs faster beside 11 warps than beside 15 (256 pairs of 15-50 atoms, 8 lanes:
//    1.56 ms, 2.0 ms at 128 registers);
//  * ESP combo: 128 -- its field points are spread over all lanes and wait for each other's rsqrt
//    and ex2, so warps count, but 20 of them (96 registers) gain nothing over 16 (calls of 8 x 60,
//    16 lanes, at 168 / 128 / 96 registers: 64 pairs 1.62 / 1.53 / 1.58 ms, 1024 pairs 3.86 / 3.48
//    / 3.81, 4096 pairs 12.8 / 12.0 / 11.8; 50 x 60, 512 pairs 10.2 / 9.5 / 10.3; align_kernel
//    1.75, 3.88, 12.3 and 10.5);
//  * two channels: 128 (16 384 pairs of 20 x 100: 24.8 ms, 25.9 ms at 168);
//  * pharmacophores: 96 from 8 lanes on, where warps hide the feature loops (1000 pairs, 128 / 96
//    registers: 3-20 features, 32 x 50, 8 lanes 512 / 481 us; 150-300 features, 20 x 30, 8 lanes
//    15.7 / 12.7 ms, 16 lanes 14.5 / 12.5, align_kernel at 96 13.3 and 13.4), 128 at 4 lanes
//    (437 / 465 us; 18.1 / 19.9 ms);
//  * last tiles of up to 5 points, 4 with a second channel beside them: the warps of ragged pairs
//    run different tiles, and more of them, or longer loops, miss the instruction cache (8192
//    shape + pharm pairs, 8 lanes: 34.5 ms with up to 4 points unrolled twice, 35.4 unrolled
//    four times, 41.0 with up to 5 points; align_kernel 38.0).  A few pairs of 4 lanes (ALONE:
//    their warps have a scheduler each) take up to 8: one pair of 30 atoms 553 us, 617 with 5.
//    With last tiles of 8 points in every launch (GROUP 8) the loop is unrolled twice: 1024 pairs
//    of 50 x 100, 4 lanes: 3.26 ms, 3.71 unrolled four times.  The loop of far points is unrolled
//    where latency bounds it (ALONE, 16 and 32 lanes) and not in the many warps of 4 or 8 lanes
//    (1024 stretched pairs, 4 lanes: 4.93 ms, 5.51 unrolled twice); two channels at 8 lanes unroll
//    it for the compact molecules beside it (16 384 pairs of 20 x 100: 27.5 ms, 28.0 without).
template <int LPP, int MODE, int GROUP, bool ALONE>
struct SpreadTile {
  static constexpr bool kTwo = MODE == FSS_MODE_SHAPE_PHARM || MODE == FSS_MODE_SHAPE_COLOR ||
                               MODE == FSS_MODE_PHARM;
  static constexpr int kRegs =
      MODE == FSS_MODE_PHARM ? (LPP >= 8 ? 96 : 128)
      : kTwo || MODE == FSS_MODE_ESP_COMBO ? 128 : 168;
  static constexpr int kTail = GROUP == 8 || ALONE ? 8 : kTwo || MODE == FSS_MODE_ESP_COMBO ? 4 : 5;
  static constexpr int kUnroll = kTwo || GROUP == 8 ? 2 : 4;
  static constexpr int kFarUnroll = LPP <= (kTwo ? 4 : 8) && !ALONE ? 1 : 2;
};

template <int LPP, int MODE, int GROUP, int EXT, bool ALONE>
__global__ void __maxnreg__((SpreadTile<LPP, MODE, GROUP, ALONE>::kRegs))
    spread_kernel(const AlignParams p) {
  using Tile = SpreadTile<LPP, MODE, GROUP, ALONE>;
  constexpr bool kCombo = MODE == FSS_MODE_ESP_COMBO;
  constexpr bool kShape = MODE != FSS_MODE_PHARM;
  constexpr bool kEsp = MODE == FSS_MODE_ESP;
  constexpr bool kPharm = MODE == FSS_MODE_PHARM || MODE == FSS_MODE_SHAPE_PHARM ||
                          MODE == FSS_MODE_SHAPE_COLOR;
  extern __shared__ __align__(16) float4 smem[];
  float4* sP = smem;
  float4* sB = sP + 2 * p.maxN;
  float4* sRA = sB + p.maxM;
  float4* sRV = sRA + p.maxNp;
  float4* sFA = sRV + p.maxNp;
  float4* sFV = sFA + p.maxMp;
  float2* sQc = reinterpret_cast<float2*>(sFV + p.maxMp);
  // vol_and_surf_esp channel, as align_kernel
  float4* sSA = sFV + p.maxMp;
  float4* sSB = sSA + p.maxNs;
  float4* sAA = sSB + p.maxMs;
  float4* sAB = sAA + 2 * p.maxNa;
  float2* sRA2 = reinterpret_cast<float2*>(sAB + 2 * p.maxMa);
  float2* sRB2 = sRA2 + p.maxNa;
  __shared__ float red[96];
  __shared__ int s_item;
  __shared__ int s_toff[10];   // first reference pharmacophore of each type

  const int tid = threadIdx.x;
  const int grp = tid / LPP, lane = tid % LPP;
  const int ppc = blockDim.x / LPP;  // poses per CTA
  constexpr int kGroupsPerWarp = 32 / LPP;

  for (;;) {
    if (tid == 0) s_item = atomicAdd(p.counter, 1);
    __syncthreads();
    const int item = s_item;
    if (item >= p.n_items) break;
    const int pidx = p.order ? p.order[item / p.chunks] : item / p.chunks;
    const int chunk = item % p.chunks;
    const int ri = p.pair_ref[pidx], fi = p.pair_fit[pidx];

    int N = 0, M = 0, Np = 0, Mp = 0, r0 = 0, f0 = 0, rp0 = 0, fp0 = 0;
    if (kShape) {
      r0 = p.ref_off[ri]; f0 = p.fit_off[fi];
      N = p.ref_off[ri + 1] - r0;
      M = p.fit_off[fi + 1] - f0;
    }
    if (kPharm) {
      rp0 = p.ref_ph_off[ri]; fp0 = p.fit_ph_off[fi];
      Np = p.ref_ph_off[ri + 1] - rp0;
      Mp = p.fit_ph_off[fi + 1] - fp0;
    }
    int Na = 0, Ma = 0, Ns = 0, Ms = 0, ra0 = 0, fa0 = 0, rs0 = 0, fs0 = 0;
    if (kCombo) {
      ra0 = p.ref_atom_off[ri]; fa0 = p.fit_atom_off[fi];
      rs0 = p.ref_surf_off[ri]; fs0 = p.fit_surf_off[fi];
      Na = p.ref_atom_off[ri + 1] - ra0; Ma = p.fit_atom_off[fi + 1] - fa0;
      Ns = p.ref_surf_off[ri + 1] - rs0; Ms = p.fit_surf_off[fi + 1] - fs0;
    }
    if (N < 0 || M < 0 || Np < 0 || Mp < 0 || N > p.maxN || M > p.maxM || Np > p.maxNp ||
        Mp > p.maxMp || Na < 0 || Ma < 0 || Ns < 0 || Ms < 0 || Na > p.maxNa ||
        Ma > p.maxMa || Ns > p.maxNs || Ms > p.maxMs) {
      // larger than the tiles this launch was sized for: flag it, leave its rows untouched
      if (tid == 0) atomicOr(p.counter + 1, 1);
      __syncthreads();
      continue;
    }
    float3 c = make_float3(0.f, 0.f, 0.f);
    if (kShape) {
      c = block_centroid(p.ref_pts + r0, N, red);
      stage_ref<kEsp>(p.ref_pts + r0, N, c, p.k, p.e, sP, sQc);
      stage_copy(Pts(p.fit_pts, p.fit_f16) + f0, M, sB);
    }
    if (kCombo) {
      // reference-side arrays move into the centred frame of the shape channel
      for (int i = tid; i < Ns; i += blockDim.x) {
        const float4 v = p.ref_surf[rs0 + i];
        sSA[i] = make_float4(v.x - c.x, v.y - c.y, v.z - c.z, v.w);
      }
      stage_copy(p.fit_surf + fs0, Ms, sSB);
      for (int i = tid; i < Na; i += blockDim.x) {
        const float4 v = p.ref_atoms[ra0 + i];
        const float x = c.x - v.x, y = c.y - v.y, z = c.z - v.z;
        sAA[2 * i] = make_float4(x, x, y, y);
        sAA[2 * i + 1] = make_float4(z, z, v.w, v.w);
        const float r = p.ref_radii[ra0 + i] + p.probe;
        sRA2[i] = make_float2(-r * r, -r * r);
      }
      for (int i = tid; i < Ma; i += blockDim.x) {
        const float4 v = p.fit_atoms[fa0 + i];
        sAB[2 * i] = make_float4(-v.x, -v.x, -v.y, -v.y);
        sAB[2 * i + 1] = make_float4(-v.z, -v.z, v.w, v.w);
        const float r = p.fit_radii[fa0 + i] + p.probe;
        sRB2[i] = make_float2(-r * r, -r * r);
      }
    }
    if (kPharm) {
      if (!kShape) c = block_centroid(p.ref_anc + rp0, Np, red);
      stage_ref_pharm(p.ref_anc + rp0, p.ref_vec ? p.ref_vec + rp0 : nullptr, Np, c, sRA, sRV,
                      s_toff);
      stage_fit_pharm(Pts(p.fit_anc, p.fit_f16) + fp0, Pts(p.fit_vec, p.fit_f16) + fp0, Mp, sFA,
                      sFV);
    }
    __syncthreads();

    const float Us = p.ref_self[ri] + p.fit_self[fi];
    const float Dtv = p.sigma * p.ref_self[ri] + (1.f - p.sigma) * p.fit_self[fi];
    const float Uc = kShape && kPharm ? p.ref_self_ph[ri] + p.fit_self_ph[fi] : 0.f;
    const int start = chunk * ppc + grp;
    const int warp_first = chunk * ppc + (tid >> 5) * kGroupsPerWarp;
    if (warp_first < p.n_starts) {  // whole idle warps skip the loop; idle groups shadow one
      const bool active = start < p.n_starts;
      const size_t row = (size_t)pidx * p.n_starts + (active ? start : p.n_starts - 1);
      using S = LanePose<LPP>;
      S s;
      s.init(p.seed_q + row * 4, p.seed_t + row * 3, c, lane);
      for (int step = 0; step < p.steps; ++step) {
        const Rot R = quat_to_rot_rn(s.q);
        Reduced rs, rc;
        float os[S::NV], oc[S::NV];
        if (kShape) {
          const ShapeArgs a{sP, sQc, sB, N, M, s.t[0], s.t[1], s.t[2], p.k, p.e, p.inv2k};
          Moments ms;
          ms.zero();
          pose_sums<LPP, kEsp, GROUP, Tile::kTail, Tile::kUnroll, Tile::kFarUnroll>(a, R, lane, ms);
          rs.from(ms, s.q);
          S::reduce(rs, lane, os);
          S::scale(os, lane, p.Kc, p.aKc);
        }
        if (kPharm) {
          Moments mc;
          mc.zero();
          pharm_pose<LPP, EXT>(sRA, sRV, sFA, sFV, Np, Mp, lane, R, s.t[0], s.t[1], s.t[2], p.tab,
                               mc, s_toff);
          rc.from(mc, s.q);
          S::reduce(rc, lane, oc);
        }
        if (kShape && kPharm) {
          s.combo(os, Us, oc, Uc, p.w, lane, p.lr);
        } else if (kPharm) {
          if (p.sigma >= 0.f) s.template tversky<true>(oc, lane, Dtv, p.lr);
          else s.template single<true>(oc, lane, Us, p.lr);
        } else if (kCombo) {
          const bool scored = step % p.esp_stride == 0 || step == p.steps - 1;
          float esp = 0.f;
          if (scored) {
            esp = esp_side<LPP, true>(sSA, Ns, sAB, sRB2, Ma, lane, R, s.t[0], s.t[1], s.t[2],
                                      p.coulomb, p.nkl) +
                  esp_side<LPP, false>(sSB, Ms, sAA, sRA2, Na, lane, R, s.t[0], s.t[1], s.t[2],
                                       p.coulomb, p.nkl);
#pragma unroll
            for (int o = LPP / 2; o > 0; o >>= 1) esp += __shfl_xor_sync(0xffffffffu, esp, o);
          }
          s.esp_combo(os, lane, Us, esp, (float)(Ns + Ms), p.esp_w, scored, p.lr);
        } else {
          s.single(os, lane, Us, p.lr);
        }
      }
      if (active) {
        const size_t r = (size_t)pidx * p.n_starts + start;
        s.write(lane, c, p.row_score + r, p.row_q + r * 4, p.row_t + r * 3);
      }
    }
    __syncthreads();  // shared memory is restaged for the next item
  }
}

}  // namespace fss
