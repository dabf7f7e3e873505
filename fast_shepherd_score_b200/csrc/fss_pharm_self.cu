// fss_pharm_self.cu -- self overlaps of packed pharmacophore sets at the identity pose.
//
// A molecule has 3-20 features and a library 10^5-10^6 molecules: a warp takes one molecule
// after another, a feature per lane, and a lane visits the features of its own type (found with
// one warp match) instead of testing all of them.  Bound by the instructions issued around 2-3
// terms a lane.  One B200, 100 000 molecules, a 32-thread CTA per molecule that tested every
// pair of types -> this form: 126 -> 52 us; 16 384: 23.7 -> 13 us.
//
// Sums keep the order and arithmetic of pharm_pose with every rounding written out: a self
// overlap's last bit reaches every score and gradient of an alignment.
#include <algorithm>
#include <cmath>

#include "fss_internal.cuh"

namespace fss {
namespace {

constexpr int kSelfWarps = 4;   // warps per CTA at most; each works alone
constexpr unsigned kAll = 0xffffffffu;

__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(kAll, v, o);
  return v;
}

// |p|^2 rounded with y before z, or with x before z.
__device__ __forceinline__ float sq_yz(float x, float y, float z) {
  return __fmaf_rn(z, z, __fmaf_rn(y, y, __fmul_rn(x, x)));
}
__device__ __forceinline__ float sq_xz(float x, float y, float z) {
  return __fmaf_rn(z, z, __fmaf_rn(x, x, __fmul_rn(y, y)));
}

// One lane per feature, against the same-type features of its molecule.  EXT as pharm_pose:
// 0 cosine weights, 1 extended points and anchors, 2 extended points only.
template <int EXT>
__global__ void __launch_bounds__(32 * kSelfWarps) pharm_self_kernel(
    const Pts anc, const Pts vec, const int* __restrict__ off, int n_mol, int max_n,
    const PharmTables tab, float* __restrict__ out) {
  extern __shared__ __align__(16) float4 smem[];
  __shared__ float4 types[kSelfWarps][9];   // (-alpha log2(e) / 2, K, category, 0) of each type
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int warps = gridDim.x * (blockDim.x >> 5);
  float4* type = types[warp];
  if (lane < 9)
    type[lane] = make_float4(-0.5f * tab.alpha[lane] * kLog2e, tab.K[lane],
                             __int_as_float(tab.cat[lane]), 0.f);
  float4* sA = smem + 2 * (size_t)max_n * warp;   // anchors (type bits in w)
  float4* sV = sA + max_n;                        // unit vectors
  int m = blockIdx.x * (blockDim.x >> 5) + warp;
  if (m >= n_mol) return;
  int o0 = off[m], o1 = off[m + 1];
  for (; m < n_mol;) {
    const int first = o0, n = o1 - o0;
    const bool more = n_mol - m > warps;
    const int next = more ? m + warps : n_mol;
    o0 = more ? off[next] : 0;
    o1 = more ? off[next + 1] : 0;
    if (n < 0 || n > max_n) {
      if (lane == 0) out[m] = __int_as_float(0x7fc00000);
      m = next;
      continue;
    }
    float3 t = make_float3(0.f, 0.f, 0.f);
    for (int i = lane; i < n; i += 32) {
      const float4 a = anc.anchor(first + i);
      const float4 v = vec ? vec[first + i] : make_float4(0.f, 0.f, 0.f, 0.f);
      const float l = sqrtf(sq_xz(v.x, v.y, v.z));
      const float inv = 1.f / (l > 1e-12f ? l : 1e-12f);
      sA[i] = make_float4(a.x, a.y, a.z, clamp_type(a.w));
      sV[i] = make_float4(v.x * inv, v.y * inv, v.z * inv, 0.f);
      t.x += a.x; t.y += a.y; t.z += a.z;
    }
    const float inv = 1.f / (float)(n > 0 ? n : 1);
    const float3 c = make_float3(__fmul_rn(warp_sum(t.x), inv), __fmul_rn(warp_sum(t.y), inv),
                                 __fmul_rn(warp_sum(t.z), inv));
    for (int i = lane; i < n; i += 32) {
      const float4 a = sA[i];
      sA[i] = make_float4(__fsub_rn(a.x, c.x), __fsub_rn(a.y, c.y), __fsub_rn(a.z, c.z), a.w);
    }
    __syncwarp();
    float v = 0.f;
    for (int j0 = 0; j0 < n; j0 += 32) {
      const int j = j0 + lane;
      const bool on = j < n;
      const float4 f = on ? sA[j] : make_float4(0.f, 0.f, 0.f, __int_as_float(8));
      const int ityp = __float_as_int(f.w);
      const float4 ty = type[ityp], fv = on ? sV[j] : f;
      const int icat = __float_as_int(ty.z);
      const bool ext = EXT != 0 && (ityp == 0 || ityp == 1);   // acceptor, donor
      float o = 0.f;
      for (int i0 = 0; i0 < n; i0 += 32) {
        // the features i0.. of this lane's type, one bit each
        const int at = i0 == j0 ? ityp : i0 + lane < n ? __float_as_int(sA[i0 + lane].w) : 8;
        unsigned mine = 0;
        if (i0 == j0) {
          mine = __match_any_sync(kAll, ityp);
        } else {
#pragma unroll
          for (int k = 0; k < 8; ++k) {
            const unsigned b = __ballot_sync(kAll, at == k);
            mine = ityp == k ? b : mine;
          }
        }
        for (unsigned b = on && icat != 3 ? mine : 0u; b; b &= b - 1) {
          const int i = i0 + __ffs(b) - 1;
          const float4 p = sA[i];
          const float dx = __fsub_rn(p.x, f.x), dy = __fsub_rn(p.y, f.y),
                      dz = __fsub_rn(p.z, f.z);
          const float KE = __fmul_rn(ty.y, ex2(__fmul_rn(ty.x, sq_yz(dx, dy, dz))));
          float w = 1.f;
          if (icat != 0) {
            const float4 rv = sV[i];
            if (ext) {
              w = EXT == 1 ? 1.f : 0.f;
              const float gx = __fsub_rn(__fadd_rn(dx, rv.x), fv.x);
              const float gy = __fsub_rn(__fadd_rn(dy, rv.y), fv.y);
              const float gz = __fsub_rn(__fadd_rn(dz, rv.z), fv.z);
              o = __fadd_rn(o, __fmul_rn(ty.y, ex2(__fmul_rn(ty.x, sq_xz(gx, gy, gz)))));
            } else {
              const float D = __fmaf_rn(fv.z, rv.z, __fmaf_rn(fv.x, rv.x, __fmul_rn(fv.y, rv.y)));
              w = __fmul_rn(__fadd_rn(icat == 1 ? fminf(fmaxf(D, 0.f), 1.f) : fabsf(D), 2.f),
                            1.f / 3.f);
            }
          }
          o = __fadd_rn(o, __fmul_rn(KE, w));
        }
      }
      if (on) v = __fadd_rn(v, o);
    }
    v = warp_sum(v);
    if (lane == 0) out[m] = v;
    __syncwarp();
    m = next;
  }
}

// Warps per CTA: four while they stage into 32 KB, one for larger molecules.
int self_warps(size_t bytes_per_warp) {
  return bytes_per_warp * kSelfWarps <= (32 << 10) ? kSelfWarps : 1;
}

// CTAs of a launch: what is resident at most, so that a warp takes several molecules.
template <class Kern>
int self_grid(Kern kern, int n_mol, int warps, size_t smem) {
  int occ = 0;
  if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, kern, 32 * warps, smem) != cudaSuccess ||
      occ <= 0) {
    (void)cudaGetLastError();
    occ = 1;
  }
  return (int)std::min<long long>(((long long)n_mol + warps - 1) / warps,
                                  (long long)occ * num_sms());
}

}  // namespace

int pharm_self_launch(const float* anc, const float* vec, const int32_t* off, int n_mol, int max_n,
                      int directional, int extended, int f16, float* out, cudaStream_t st) {
  if (n_mol < 0 || !anc || !off || !out || (directional && !vec))
    return set_error(FSS_ERR_INVALID, "fss_pharm_self_overlap: bad arguments");
  if (extended < 0 || extended > 2 || (extended && !directional))
    return set_error(FSS_ERR_INVALID, "fss_pharm_self_overlap: extended must be 0, 1 or 2 "
                                      "(directional tables)");
  if (max_n > kMaxPoints) return set_error(FSS_ERR_UNSUPPORTED, "fss_pharm_self_overlap: molecule too large");
  if (n_mol == 0) return FSS_OK;
  if (max_n < 0) return set_error(FSS_ERR_INVALID, "fss_pharm_self_overlap: negative extent");
  // An alignment stages the anchors and vectors of both sides: a molecule it could not take against
  // itself (more than 3631 features) is refused here too, although this kernel stages it once.
  if (4 * sizeof(float4) * (size_t)max_n + 16 > (227u << 10))
    return set_error(FSS_ERR_CUDA, "fss_pharm_self_overlap: molecule too large for shared memory");
  const size_t per = 2 * sizeof(float4) * (size_t)max_n;
  const int warps = self_warps(per);
  const size_t smem = per * warps;
  auto kern = extended == 1 ? pharm_self_kernel<1>
              : extended == 2 ? pharm_self_kernel<2> : pharm_self_kernel<0>;
  cudaError_t ce = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (ce != cudaSuccess) return set_error(FSS_ERR_CUDA, std::string("fss_pharm_self_overlap: ") + cudaGetErrorString(ce));
  kern<<<self_grid(kern, n_mol, warps, smem), 32 * warps, smem, st>>>(
      Pts(anc, f16), Pts(vec, f16), off, n_mol, max_n, make_pharm_tables(directional != 0), out);
  return check_launch("fss_pharm_self_overlap");
}

}  // namespace fss
