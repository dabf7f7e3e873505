// fss_prep.cu -- what an alignment call computes around its fused kernel: the pairs' index check and
// cost keys, the centring of pharmacophore sets and the fold of the centroids into the poses.  Each
// was a chain of elementwise launches (about 110 a call of 1000 pharmacophore pairs, with a hidden
// synchronisation in two of them) whose host time exceeded the alignment's; each is bound by the
// latency of one small launch.  One B200, with no free-memory query before them either (run_chunked in
// memory.py), a call of 1000 pharmacophore pairs 2.0 -> 0.63 ms, of one atom pair 1.05 -> 0.93.
#include <algorithm>

#include "fss_internal.cuh"

namespace fss {
namespace {

constexpr int kThreads = 256;

// key[p] = -(reference size x fit size), clamped to int32: an ascending stable sort gives the
// costliest pairs first.  A pair outside the molecule tables sets *bad and gets key 0.
__global__ void __launch_bounds__(kThreads) pair_cost_kernel(
    const int* __restrict__ roff, const int* __restrict__ foff, const int* __restrict__ pr,
    const int* __restrict__ pf, int P, int n_ref, int n_fit, int* key, int* bad) {
  const int p = blockIdx.x * kThreads + threadIdx.x;
  if (p >= P) return;
  const int r = pr[p], f = pf[p];
  if (r < 0 || f < 0 || r >= n_ref || f >= n_fit) {
    if (bad) atomicOr(bad, 1);
    key[p] = 0;
    return;
  }
  const long long cost = (long long)(roff[r + 1] - roff[r]) * (foff[f + 1] - foff[f]);
  key[p] = -(int)min(cost, 0x7fffffffLL);
}

// out[(mol L + i) 3 + c] = anchor i of molecule mol, 0 past its last: the padded cloud whose
// per-molecule sums give the centroids.
__global__ void __launch_bounds__(kThreads) pad_anchors_kernel(const float4* __restrict__ anc,
                                                               const int* __restrict__ off,
                                                               long long total, int L, float* out) {
  const long long k = (long long)blockIdx.x * kThreads + threadIdx.x;
  if (k >= total) return;
  const int mol = (int)(k / L), i = (int)(k - (long long)mol * L);
  const int a = off[mol];
  const float4 v = i < off[mol + 1] - a ? anc[a + i] : make_float4(0.f, 0.f, 0.f, 0.f);
  out[3 * k] = v.x; out[3 * k + 1] = v.y; out[3 * k + 2] = v.z;
}

// A warp per molecule: centroid = sum / size, anchors moved to it (types kept), and the same
// positions as a plain cloud.
__global__ void __launch_bounds__(kThreads) centre_anchors_kernel(
    const float4* __restrict__ anc, const int* __restrict__ off, int n_mol,
    const float* __restrict__ sum, float4* centred, float4* cloud, float* centroid) {
  const long long mol = ((long long)blockIdx.x * kThreads + threadIdx.x) / 32;
  const int lane = threadIdx.x % 32;
  if (mol >= n_mol) return;
  const int a = off[mol], b = off[mol + 1];
  const float n = (float)max(b - a, 1);
  const float x = __fdiv_rn(sum[3 * mol], n), y = __fdiv_rn(sum[3 * mol + 1], n),
              z = __fdiv_rn(sum[3 * mol + 2], n);
  for (int k = a + lane; k < b; k += 32) {
    const float4 v = anc[k];
    const float4 w = make_float4(v.x - x, v.y - y, v.z - z, v.w);
    centred[k] = w;
    cloud[k] = make_float4(w.x, w.y, w.z, 0.f);
  }
  if (lane < 3) centroid[3 * mol + lane] = lane == 0 ? x : lane == 1 ? y : z;
}

// t = t - R(q) c_fit + c_ref: poses of centred clouds as poses of the clouds themselves.
__global__ void __launch_bounds__(kThreads) fold_centroids_kernel(
    const float* __restrict__ q, const float* __restrict__ t, const int* __restrict__ pr,
    const int* __restrict__ pf, const float* __restrict__ cr, const float* __restrict__ cf, int P,
    float* out) {
  const int p = blockIdx.x * kThreads + threadIdx.x;
  if (p >= P) return;
  float v[4], s = 0.f;
#pragma unroll
  for (int i = 0; i < 4; ++i) { v[i] = q[4 * (size_t)p + i]; s = fmaf(v[i], v[i], s); }
  const float norm = fmaxf(sqrtf(s), 1e-12f);
#pragma unroll
  for (int i = 0; i < 4; ++i) v[i] /= norm;
  const Rot R = quat_to_rot(v);
  const float* f = cf + 3 * (size_t)pf[p];
  const float* r = cr + 3 * (size_t)pr[p];
  const float3 y = rot_apply(R, f[0], f[1], f[2]);
  out[3 * (size_t)p] = t[3 * (size_t)p] - y.x + r[0];
  out[3 * (size_t)p + 1] = t[3 * (size_t)p + 1] - y.y + r[1];
  out[3 * (size_t)p + 2] = t[3 * (size_t)p + 2] - y.z + r[2];
}

unsigned blocks(long long n) { return (unsigned)((n + kThreads - 1) / kThreads); }

}  // namespace

int pair_cost_launch(const int32_t* roff, const int32_t* foff, const int32_t* pr,
                     const int32_t* pf, int P, int n_ref, int n_fit, int32_t* key, int32_t* bad,
                     cudaStream_t st) {
  if (P < 0 || n_ref < 0 || n_fit < 0) return set_error(FSS_ERR_INVALID, "fss_pair_cost: bad sizes");
  if (P == 0) return FSS_OK;
  if (!roff || !foff || !pr || !pf || !key)
    return set_error(FSS_ERR_INVALID, "fss_pair_cost: null pointer");
  pair_cost_kernel<<<blocks(P), kThreads, 0, st>>>(roff, foff, pr, pf, P, n_ref, n_fit, key, bad);
  return check_launch("fss_pair_cost");
}

int pad_anchors_launch(const float* anc, const int32_t* off, int n_mol, int L, float* out,
                       cudaStream_t st) {
  if (n_mol < 0 || L < 1) return set_error(FSS_ERR_INVALID, "fss_pad_anchors: bad sizes");
  if (n_mol == 0) return FSS_OK;
  if (!off || !out) return set_error(FSS_ERR_INVALID, "fss_pad_anchors: null pointer");
  const long long total = (long long)n_mol * L;
  pad_anchors_kernel<<<blocks(total), kThreads, 0, st>>>(reinterpret_cast<const float4*>(anc), off,
                                                         total, L, out);
  return check_launch("fss_pad_anchors");
}

int centre_anchors_launch(const float* anc, const int32_t* off, int n_mol, const float* sum,
                          float* centred, float* cloud, float* centroid, cudaStream_t st) {
  if (n_mol < 0) return set_error(FSS_ERR_INVALID, "fss_centre_anchors: bad sizes");
  if (n_mol == 0) return FSS_OK;
  if (!off || !sum || !centroid)
    return set_error(FSS_ERR_INVALID, "fss_centre_anchors: null pointer");
  centre_anchors_kernel<<<blocks(32LL * n_mol), kThreads, 0, st>>>(
      reinterpret_cast<const float4*>(anc), off, n_mol, sum, reinterpret_cast<float4*>(centred),
      reinterpret_cast<float4*>(cloud), centroid);
  return check_launch("fss_centre_anchors");
}

int fold_centroids_launch(const float* q, const float* t, const int32_t* pr, const int32_t* pf,
                          const float* cr, const float* cf, int P, float* out, cudaStream_t st) {
  if (P < 0) return set_error(FSS_ERR_INVALID, "fss_fold_centroids: bad sizes");
  if (P == 0) return FSS_OK;
  if (!q || !t || !pr || !pf || !cr || !cf || !out)
    return set_error(FSS_ERR_INVALID, "fss_fold_centroids: null pointer");
  fold_centroids_kernel<<<blocks(P), kThreads, 0, st>>>(q, t, pr, pf, cr, cf, P, out);
  return check_launch("fss_fold_centroids");
}

}  // namespace fss
