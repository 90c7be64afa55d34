// Producers of the statistics the fused prologues of gemm read: per-voxel PixelNorm factors for conv3's `pn` (pixstats,
// src/ops/video.js:301-318) and the GroupNorm scale / offset per channel for conv's `gn` (gnPartial + gnFinalize,
// src/ops/misc.js:50-120).  Bandwidth kernels: the tensor is read once (a 64-pixel chunk stays in registers
// for the exact two-pass variance).
#include "common.cuh"
#include "ctx.h"
#include "sync.cuh"

using namespace p0p;

namespace {

// ---- pixstats: R[ro + v] = rsqrt(sum_c x[v][c]^2 / C + eps), x fp16 [V][C].  L lanes share a voxel (16-byte loads).
__global__ void __launch_bounds__(256) k_pixstats(const __half* X, uint32_t V, uint32_t C, uint32_t L, float eps, float* R, uint32_t vec) {
  const uint32_t gt = blockIdx.x * blockDim.x + threadIdx.x, sub = gt % L;
  const uint32_t v = gt / L;
  float s = 0.0f;
  grid_dependency_wait();
  grid_launch_dependents();
  if (v < V) {
    const __half* x = X + (size_t)v * C;
    if (vec) {
      for (uint32_t c = sub * 8u; c < C; c += L * 8u) {
        const uint4 q = ld_now(reinterpret_cast<const uint4*>(x + c));
        const __half2* h = reinterpret_cast<const __half2*>(&q);
#pragma unroll
        for (int i = 0; i < 4; i++) { const float2 f = __half22float2(h[i]); s = fmaf(f.x, f.x, s); s = fmaf(f.y, f.y, s); }
      }
    } else {
      for (uint32_t c = sub; c < C; c += L) { const float f = __half2float(x[c]); s = fmaf(f, f, s); }
    }
  }
  for (uint32_t o = L >> 1; o > 0u; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);      // L is a power of two <= 32: partners stay inside the voxel's lanes
  if (v < V && sub == 0u) R[v] = rsqrtf(s / (float)C + eps);
}

// ---- GroupNorm partial statistics: one block per 64 pixels of an HWC fp16 tensor [pix][C], 32 groups of C / 32 channels.
// PT[(wgOff + block) * 32 + g] = (count, mean, M2, 0) of the block's own chunk, by an exact two-pass (src/ops/misc.js:50-73).
// C is a power of two (32..512), so a thread's eight consecutive elements are the same eight channels in every round of 2048
// elements: per-thread channel sums -> per-channel sums over the threads that share channels -> per-group sums, all in a
// fixed order (deterministic).  NI = C / 32 rounds make the chunk (NI is a template argument): all of a thread's 16-byte loads are
// issued before the first is used and the values stay in registers for the second pass.  (128 x 128 x 512: 10.5 -> 8.3 us)
template <int NI>
__global__ void __launch_bounds__(256) k_gn_partial(const __half* X, uint32_t pix, uint32_t wgOff, float4* PT) {
  constexpr uint32_t C = 32u * NI, cpg = NI, reps = 2048u / C, per = C / 8u;
  __shared__ float part[256][9];      // per thread, per element of its 8 (padded against bank conflicts)
  __shared__ float chs[C];            // per channel
  __shared__ float mg[32], m2[32];    // group means, group M2
  const uint32_t t = threadIdx.x, wg = blockIdx.x, px0 = wg * 64u, npx = min(64u, pix - min(px0, pix));
  const uint32_t n = npx * C, c0 = (t * 8u) % C;
  const __half* x = X + (size_t)px0 * C;
  const float cnt = (float)(npx * cpg);
  grid_dependency_wait();
  grid_launch_dependents();
  uint4 v[NI];
#pragma unroll
  for (uint32_t i = 0; i < (uint32_t)NI; i++) { const uint32_t e = i * 2048u + t * 8u; v[i] = e < n ? ld_now(reinterpret_cast<const uint4*>(x + e)) : make_uint4(0u, 0u, 0u, 0u); }
  float acc[8];
  auto reduce_groups = [&](float* out32) {      // acc[] of all threads -> out32[g]; ends with a barrier
#pragma unroll
    for (int j = 0; j < 8; j++) part[t][j] = acc[j];
    __syncthreads();
    for (uint32_t c = t; c < C; c += 256u) {
      float s = 0.0f;
#pragma unroll 8
      for (uint32_t r = 0; r < reps; r++) s += part[c / 8u + r * per][c % 8u];
      chs[c] = s;
    }
    __syncthreads();
    if (t < 32u) {
      float s = 0.0f;
#pragma unroll
      for (uint32_t j = 0; j < cpg; j++) s += chs[t * cpg + j];
      out32[t] = s;
    }
    __syncthreads();
  };
#pragma unroll
  for (int j = 0; j < 8; j++) acc[j] = 0.0f;
#pragma unroll
  for (int i = 0; i < NI; i++) {
    const __half* h = reinterpret_cast<const __half*>(&v[i]);
#pragma unroll
    for (int j = 0; j < 8; j++) acc[j] += __half2float(h[j]);
  }
  reduce_groups(mg);
  if (t < 32u) mg[t] = mg[t] / fmaxf(cnt, 1.0f);
  __syncthreads();
  float mean[8];
#pragma unroll
  for (int j = 0; j < 8; j++) { mean[j] = mg[(c0 + j) / cpg]; acc[j] = 0.0f; }
#pragma unroll
  for (uint32_t i = 0; i < (uint32_t)NI; i++) {
    if (i * 2048u + t * 8u >= n) break;
    const __half* h = reinterpret_cast<const __half*>(&v[i]);
#pragma unroll
    for (int j = 0; j < 8; j++) { const float d = __half2float(h[j]) - mean[j]; acc[j] = fmaf(d, d, acc[j]); }
  }
  reduce_groups(m2);
  if (t < 32u) PT[((size_t)wgOff + wg) * 32u + t] = make_float4(cnt, mg[t], m2[t], 0.0f);
}

// ---- merge of the partial rows with Chan's parallel formula (src/ops/misc.js:75-104) -> per channel a = gamma * rstd,
// b = beta - mean * a.  One block per group: a thread merges every 256th row in order (its next rows already loading), then the
// warp's lanes and the eight warps merge pairwise (the formula is symmetric).  Bound by latency: one block for all 32 groups, a warp
// to each, was a chain of nwg / 32 dependent merges per lane on one SM (256 rows: 10.9 us, 5.4 now)
struct Chan { float n, mean, m2; };
__device__ __forceinline__ Chan chan_merge(Chan a, Chan b) {
  if (!(b.n > 0.0f)) return a;
  if (!(a.n > 0.0f)) return b;
  const float nn = a.n + b.n, d = b.mean - a.mean;
  Chan r; r.n = nn; r.mean = a.mean + d * (b.n / nn); r.m2 = a.m2 + b.m2 + d * d * (a.n * b.n / nn);
  return r;
}
__global__ void __launch_bounds__(256) k_gn_finalize(const float4* PT, uint32_t nwg, uint32_t C, float eps, const float* GB, uint32_t gOff, uint32_t bOff,
                                                     float* AB) {
  __shared__ Chan sh[8];
  const uint32_t g = blockIdx.x, t = threadIdx.x, l = t & 31u, cpg = C / 32u;
  grid_dependency_wait();
  grid_launch_dependents();
  Chan s{0.0f, 0.0f, 0.0f};
#pragma unroll 4
  for (uint32_t w = t; w < nwg; w += 256u) { const float4 q = ld_now(PT + (size_t)w * 32u + g); s = chan_merge(s, Chan{q.x, q.y, q.z}); }
#pragma unroll
  for (uint32_t o = 1; o < 32u; o <<= 1) {
    Chan b; b.n = __shfl_xor_sync(0xffffffffu, s.n, o); b.mean = __shfl_xor_sync(0xffffffffu, s.mean, o); b.m2 = __shfl_xor_sync(0xffffffffu, s.m2, o);
    s = (l & o) ? chan_merge(b, s) : chan_merge(s, b);      // both partners merge (lower, upper): the same value on both
  }
  if (l == 0u) sh[t >> 5] = s;
  __syncthreads();
  if (t >= cpg) return;
  s = sh[0];
#pragma unroll
  for (int w = 1; w < 8; w++) s = chan_merge(s, sh[w]);
  const float rs = rsqrtf(s.m2 / fmaxf(s.n, 1.0f) + eps);
  const uint32_t c = g * cpg + t;
  const float a = ld_now(GB + gOff + c) * rs;
  AB[c] = a; AB[C + c] = ld_now(GB + bOff + c) - s.mean * a;
}

inline bool live(const p0p_ctx* c, const p0p_buf* b) { return b && c->bufs.count(const_cast<p0p_buf*>(b)); }

}  // namespace

extern "C" int p0p_pixstats(p0p_ctx* c, const p0p_buf* x, uint64_t x_off, uint32_t V, uint32_t C, float eps, p0p_buf* r, uint32_t ro) {
  P0P_ALIVE(c);
  if (!live(c, x) || !live(c, r)) return fail(c, -4, "pixstats: missing binding");
  if (!V || !C) return 0;
  if (C % 4u) return fail(c, -5, "pixstats: C must be a multiple of 4");                  // the reference reads vec4<f16>
  if (x_off & 7u) return fail(c, -5, "pixstats: x.off must be a multiple of 8 bytes");
  const uint64_t xb = (uint64_t)V * C * 2ull, rb = ((uint64_t)ro + V) * 4ull;
  if (x_off > x->size || xb > x->size - x_off || rb > r->size) return fail(c, -7, "pixstats: a range is outside its buffer");
  DeviceGuard g(c->device);
  const __half* X = reinterpret_cast<const __half*>((const char*)x->ptr + x_off);
  const uint32_t vec = (C % 8u == 0u && ((uintptr_t)X & 15u) == 0u) ? 1u : 0u;
  uint32_t L = 1u; while (L < 32u && L * (vec ? 8u : 1u) < C) L <<= 1;                     // lanes per voxel: enough for one load each, at most a warp
  const uint64_t threads = (uint64_t)V * L;
  cudaError_t e = launch_chained(k_pixstats, dim3((unsigned)((threads + 255u) / 256u)), dim3(256), 0, c->stream, X, V, C, L, eps != 0.0f ? eps : 1e-8f, (float*)r->ptr + ro, vec);
  if (e != cudaSuccess) return cuda_fail(c, e, "pixstats launch");
  c->launches += 1;
  return 0;
}

extern "C" int p0p_gn_partial(p0p_ctx* c, const p0p_buf* x, uint64_t x_off, uint32_t pix, uint32_t C, p0p_buf* part, uint32_t wgOff, uint32_t* nwg_out) {
  P0P_ALIVE(c);
  const uint32_t nwg = (pix + 63u) / 64u;
  if (nwg_out) *nwg_out = nwg;
  if (!live(c, x) || !live(c, part)) return fail(c, -4, "gnPartial: missing binding");
  if (!pix) return 0;
  if (C < 32u || C > 512u || (C & (C - 1u))) return fail(c, -5, "gnPartial: C must be a power of two from 32 to 512");      // src/ops/misc.js:110
  if (x_off & 15u) return fail(c, -5, "gnPartial: x.off must be a multiple of 16 bytes");
  const uint64_t xb = (uint64_t)pix * C * 2ull, pb = ((uint64_t)wgOff + nwg) * 512ull;
  if (x_off > x->size || xb > x->size - x_off || pb > part->size) return fail(c, -7, "gnPartial: a range is outside its buffer");
  DeviceGuard g(c->device);
  cudaError_t e = launch_chained(C == 32u ? k_gn_partial<1> : C == 64u ? k_gn_partial<2> : C == 128u ? k_gn_partial<4> : C == 256u ? k_gn_partial<8> : k_gn_partial<16>,
                                 dim3(nwg), dim3(256), 0, c->stream, reinterpret_cast<const __half*>((const char*)x->ptr + x_off), pix, wgOff, (float4*)part->ptr);
  if (e != cudaSuccess) return cuda_fail(c, e, "gnPartial launch");
  c->launches += 1;
  return 0;
}

extern "C" int p0p_gn_finalize(p0p_ctx* c, const p0p_buf* part, uint32_t nwg, uint32_t C, float eps, const p0p_buf* gb, uint32_t g_off, uint32_t b_off,
                               p0p_buf* ab, uint32_t ab_off) {
  P0P_ALIVE(c);
  if (!live(c, part) || !live(c, gb) || !live(c, ab)) return fail(c, -4, "gnFinalize: missing binding");
  if (C < 32u || C > 512u || (C & (C - 1u))) return fail(c, -5, "gnFinalize: C must be a power of two from 32 to 512");
  if ((uint64_t)nwg * 512ull > part->size || ((uint64_t)std::max(g_off, b_off) + C) * 4ull > gb->size || ((uint64_t)ab_off + 2ull * C) * 4ull > ab->size)
    return fail(c, -7, "gnFinalize: a range is outside its buffer");
  DeviceGuard g(c->device);
  cudaError_t e = launch_chained(k_gn_finalize, dim3(32), dim3(256), 0, c->stream, (const float4*)part->ptr, nwg, C, eps != 0.0f ? eps : 1e-6f, (const float*)gb->ptr, g_off, b_off,
                                 (float*)ab->ptr + ab_off);
  if (e != cudaSuccess) return cuda_fail(c, e, "gnFinalize launch");
  c->launches += 1;
  return 0;
}
