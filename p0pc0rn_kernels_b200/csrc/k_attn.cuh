// Attention of few query rows over a long key / value sequence (decoding steps), head_dim 128 (src/ops/attention.js):
// Q [Hq][Lq][128] f16, K / V [Hkv][Lk][128] f16 (head-major, as the GEMM's 'heads' epilogue writes them), O [Lq][ldo] f16
// token-major at column h * 128.  fp32 scores, online-softmax statistics and accumulators.
//   mask 0 = none; 1 = causal + valid length (key j visible to query i iff j <= min(i, nvalid - 1)); 2 = valid length (j < nvalid)
//   GQA: query head h reads kv head h / (Hq / Hkv)                                            (attention.js:8-10, 64, 93-99)
// Bound: one pass over K and V, so the work is cut where those bytes are.  The query rows of all heads that share a kv head
// are one contiguous matrix of (Hq / Hkv) * Lq rows: every K / V tile is read once for all of them, and the keys are cut into
// S splits until the blocks cover the SMs (a block per (head, 64 queries) left 116 of 148 SMs without work at 32 heads and
// read every K / V byte once per query head).  The partial (maximum, sum, O) of the splits are merged by the block that
// finishes last (one counter per kv head and row block; it resets the counter), in split order: deterministic, one launch.
// Block = 4 warps: WM row tiles of 16 x (4 / WM) shares of each 64-key tile; K / V tiles arrive by cp.async through three
// stages in an XOR swizzle (conflict-free ldmatrix); both products are mma.sync m16n8k16.
// Measured: 32:8 heads, 1 query, 4000 of 4096 keys (16.4 MB): 8.9 us a call, host call included (a block per head and 64 queries,
// the earlier kernel: 135 us).
#pragma once
#include <cuda_fp16.h>
#include <stdint.h>

#include "sync.cuh"

namespace p0p {

struct AttnP {
  const __half* Q; const __half* K; const __half* V; __half* O;
  uint32_t Lq, Lk, ldo, Hq, Hkv, mode, nvalid;
  float scale_log2;      // scale * log2(e): the softmax runs on exp2
  uint32_t rows;         // query rows that share a kv head: (Hq / Hkv) * Lq
  uint32_t S, tps;       // splits of the keys, and key tiles of 64 per split
  float* part;           // [kv head][row block][split][16 WM rows][128] unnormalised O, then the same without 128: (maximum, sum)
  float2* part_ml;
  uint32_t* count;       // [kv head][row block] arrivals, zero between calls
};

constexpr uint32_t AT_STAGES = 3u, AT_TILE_B = 64u * 256u;               // bytes of one K or V tile of 64 keys
constexpr uint32_t AT_SMEM = AT_STAGES * 2u * AT_TILE_B;

__device__ __forceinline__ void at_mma(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
               : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3]) : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
// 16 bytes, or 16 zero bytes when `on` is 0 (the source is then not read)
__device__ __forceinline__ void at_cp16(uint32_t dst, const void* src, uint32_t on) { asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(on ? 16u : 0u) : "memory"); }
__device__ __forceinline__ void at_cp_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N> __device__ __forceinline__ void at_cp_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }
__device__ __forceinline__ uint32_t at_pack(float lo, float hi) { __half2 h = __floats2half2_rn(lo, hi); return *reinterpret_cast<uint32_t*>(&h); }
__device__ __forceinline__ float at_ex2(float x) { float y; asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x)); return y; }
__device__ __forceinline__ void at_ldsm(uint32_t (&r)[4], uint32_t a) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(a) : "memory");
}
__device__ __forceinline__ void at_ldsm_t(uint32_t (&r)[4], uint32_t a) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(a) : "memory");
}

// (Every row sees at least key 0, nvalid being >= 1, so the sums that are divided by are positive.)
template <int WM>
__global__ void __launch_bounds__(128) k_attn_split(const AttnP p) {
  extern __shared__ __align__(128) unsigned char at_smem[];
  constexpr uint32_t WK = 4u / WM, KPW = 64u / WK, NB = KPW / 8u, RB = 16u * WM;      // key shares, keys per warp and tile, 8-key blocks of them, rows per block
  __shared__ float sm_m[4][16], sm_l[4][16];
  __shared__ uint32_t sm_last;
  const uint32_t tid = threadIdx.x, warp = tid >> 5, lane = tid & 31u, g = lane >> 2, t4 = lane & 3u, wm = warp % WM, wk = warp / WM;
  const uint32_t rb = blockIdx.x, hk = blockIdx.y, split = blockIdx.z, r0 = rb * RB, grp = p.Hq / p.Hkv;
  const __half* Kg = p.K + (size_t)hk * p.Lk * 128u; const __half* Vg = p.V + (size_t)hk * p.Lk * 128u;
  const __half* Qg = p.Q + (size_t)hk * grp * p.Lq * 128u;
  const uint32_t base = (uint32_t)__cvta_generic_to_shared(at_smem);
  // keys that any row of this block sees                                                     (attention.js:64)
  uint32_t kEnd = p.Lk;
  if (p.mode == 1u) {
    const uint32_t rl = min(r0 + RB, p.rows) - 1u, imax = r0 / p.Lq == rl / p.Lq ? rl % p.Lq : p.Lq - 1u;
    kEnd = min(p.Lk, min(imax, p.nvalid - 1u) + 1u);
  }
  if (p.mode == 2u) kEnd = min(p.Lk, p.nvalid);
  const uint32_t nt = (kEnd + 63u) >> 6, tb = min(split * p.tps, nt), te = min(tb + p.tps, nt);
  auto load = [&](uint32_t t, uint32_t st) {
    const uint32_t kk = t * 64u, dst = base + st * 2u * AT_TILE_B;
#pragma unroll
    for (uint32_t i = 0; i < 8u; i++) {
      const uint32_t e = i * 128u + tid, r = e >> 4, c = e & 15u, key = kk + r, on = key < kEnd ? 1u : 0u, o = r * 256u + ((c ^ (r & 7u)) << 4);
      const size_t src = (size_t)min(key, p.Lk - 1u) * 128u + c * 8u;
      at_cp16(dst + o, Kg + src, on);
      at_cp16(dst + AT_TILE_B + o, Vg + src, on);
    }
  };
  grid_dependency_wait();
  grid_launch_dependents();
#pragma unroll
  for (uint32_t s = 0; s < AT_STAGES - 1u; s++) { if (tb + s < te) load(tb + s, s); at_cp_commit(); }
  // this thread's two rows (rows past the end repeat the last one; they are not stored)
  const uint32_t ra = min(r0 + wm * 16u + g, p.rows - 1u), rc = min(r0 + wm * 16u + g + 8u, p.rows - 1u);
  uint32_t qa[8][4];
#pragma unroll
  for (int ks = 0; ks < 8; ks++) {
    const uint32_t* a = reinterpret_cast<const uint32_t*>(Qg + (size_t)ra * 128u + ks * 16) + t4; const uint32_t* b = reinterpret_cast<const uint32_t*>(Qg + (size_t)rc * 128u + ks * 16) + t4;
    qa[ks][0] = ld_now(a); qa[ks][1] = ld_now(b); qa[ks][2] = ld_now(a + 4); qa[ks][3] = ld_now(b + 4);
  }
  uint32_t lim[2] = {kEnd, kEnd};
  if (p.mode == 1u) { lim[0] = min(p.Lk, min(ra % p.Lq, p.nvalid - 1u) + 1u); lim[1] = min(p.Lk, min(rc % p.Lq, p.nvalid - 1u) + 1u); }
  float o[16][4];
#pragma unroll
  for (int d = 0; d < 16; d++) { o[d][0] = o[d][1] = o[d][2] = o[d][3] = 0.0f; }
  float m[2] = {-INFINITY, -INFINITY}, l[2] = {0.0f, 0.0f};
  for (uint32_t t = tb; t < te; t++) {
    const uint32_t st = (t - tb) % AT_STAGES;
    at_cp_wait<AT_STAGES - 2>();
    __syncthreads();                                     // tile t is complete, and everyone is past tile t - 1, whose stage is refilled now
    if (t + AT_STAGES - 1u < te) load(t + AT_STAGES - 1u, (t - tb + AT_STAGES - 1u) % AT_STAGES);
    at_cp_commit();
    const uint32_t ks_ = base + st * 2u * AT_TILE_B, vs_ = ks_ + AT_TILE_B, k0 = wk * KPW;
    float s[NB][4];
#pragma unroll
    for (uint32_t n = 0; n < NB; n++) { s[n][0] = s[n][1] = s[n][2] = s[n][3] = 0.0f; }
#pragma unroll
    for (uint32_t n = 0; n < NB; n += 2u) {
      const uint32_t key = k0 + n * 8u + ((lane >> 4) << 3) + (lane & 7u), row = ks_ + key * 256u, x = key & 7u, c0 = (lane >> 3) & 1u;
#pragma unroll
      for (uint32_t ks = 0; ks < 8u; ks++) {
        uint32_t b[4];
        at_ldsm(b, row + (((ks * 2u + c0) ^ x) << 4));
        at_mma(s[n], qa[ks], b[0], b[1]);
        at_mma(s[n + 1], qa[ks], b[2], b[3]);
      }
    }
    const uint32_t kk = t * 64u + k0;
    float mx[2] = {-INFINITY, -INFINITY};
#pragma unroll
    for (uint32_t n = 0; n < NB; n++)
#pragma unroll
      for (uint32_t e = 0; e < 4u; e++) {
        const uint32_t key = kk + n * 8u + 2u * t4 + (e & 1u);
        s[n][e] = key < lim[e >> 1] ? s[n][e] * p.scale_log2 : -INFINITY;
        mx[e >> 1] = fmaxf(mx[e >> 1], s[n][e]);
      }
#pragma unroll
    for (int h = 0; h < 2; h++) { mx[h] = fmaxf(mx[h], __shfl_xor_sync(0xffffffffu, mx[h], 1)); mx[h] = fmaxf(mx[h], __shfl_xor_sync(0xffffffffu, mx[h], 2)); }
    if (__any_sync(0xffffffffu, mx[0] > m[0] || mx[1] > m[1])) {
      const float n0 = fmaxf(m[0], mx[0]), n1 = fmaxf(m[1], mx[1]);
      const float a0 = n0 == -INFINITY ? 1.0f : at_ex2(m[0] - n0), a1 = n1 == -INFINITY ? 1.0f : at_ex2(m[1] - n1);
      m[0] = n0; m[1] = n1; l[0] *= a0; l[1] *= a1;
#pragma unroll
      for (int d = 0; d < 16; d++) { o[d][0] *= a0; o[d][1] *= a0; o[d][2] *= a1; o[d][3] *= a1; }
    }
    const float e0 = m[0] == -INFINITY ? 0.0f : m[0], e1 = m[1] == -INFINITY ? 0.0f : m[1];
#pragma unroll
    for (uint32_t n = 0; n < NB; n += 2u) {
      uint32_t pa[4];
#pragma unroll
      for (uint32_t h = 0; h < 2u; h++) {
        const float p0 = at_ex2(s[n + h][0] - e0), p1 = at_ex2(s[n + h][1] - e0), p2 = at_ex2(s[n + h][2] - e1), p3 = at_ex2(s[n + h][3] - e1);
        l[0] += p0 + p1; l[1] += p2 + p3;
        pa[2u * h] = at_pack(p0, p1); pa[2u * h + 1u] = at_pack(p2, p3);
      }
      const uint32_t key = k0 + n * 8u + (((lane >> 3) & 1u) << 3) + (lane & 7u), row = vs_ + key * 256u, x = key & 7u, c0 = lane >> 4;
#pragma unroll
      for (uint32_t d = 0; d < 8u; d++) {
        uint32_t b[4];
        at_ldsm_t(b, row + (((d * 2u + c0) ^ x) << 4));
        at_mma(o[2u * d], pa, b[0], b[1]);
        at_mma(o[2u * d + 1u], pa, b[2], b[3]);
      }
    }
  }
  // ---- the warps' shares of the keys, merged through shared memory (in warp order)
#pragma unroll
  for (int h = 0; h < 2; h++) { l[h] += __shfl_xor_sync(0xffffffffu, l[h], 1); l[h] += __shfl_xor_sync(0xffffffffu, l[h], 2); }
  if (t4 == 0u) { sm_m[warp][g] = m[0]; sm_m[warp][g + 8u] = m[1]; sm_l[warp][g] = l[0]; sm_l[warp][g + 8u] = l[1]; }
  at_cp_wait<0>();
  __syncthreads();                                       // every warp is past its last tile: the stages become the merge buffer
  constexpr uint32_t LD = 132u;
  float* ob = reinterpret_cast<float*>(at_smem);
#pragma unroll
  for (uint32_t d = 0; d < 16u; d++) {
    *reinterpret_cast<float2*>(ob + (warp * 16u + g) * LD + d * 8u + 2u * t4) = make_float2(o[d][0], o[d][1]);
    *reinterpret_cast<float2*>(ob + (warp * 16u + g + 8u) * LD + d * 8u + 2u * t4) = make_float2(o[d][2], o[d][3]);
  }
  __syncthreads();
  const uint32_t nrows = min(RB, p.rows - r0);
  auto store = [&](uint32_t r, float4 v) {               // columns 4 lane .. of packed row r
    const uint32_t h = hk * grp + r / p.Lq, i = r % p.Lq;
    __half2* d = reinterpret_cast<__half2*>(p.O + (size_t)i * p.ldo + h * 128u + 4u * lane);
    d[0] = __floats2half2_rn(v.x, v.y); d[1] = __floats2half2_rn(v.z, v.w);
  };
  const size_t slab = ((size_t)hk * gridDim.x + rb) * p.S;
  for (uint32_t r = warp; r < nrows; r += 4u) {
    const uint32_t w0 = r >> 4, rr = r & 15u;
    float M = -INFINITY, L = 0.0f;
#pragma unroll
    for (uint32_t k = 0; k < WK; k++) M = fmaxf(M, sm_m[k * WM + w0][rr]);
    float4 acc = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
#pragma unroll
    for (uint32_t k = 0; k < WK; k++) {
      const uint32_t w = k * WM + w0;
      const float f = M == -INFINITY ? 0.0f : at_ex2(sm_m[w][rr] - M);
      const float4 v = *reinterpret_cast<const float4*>(ob + (w * 16u + rr) * LD + 4u * lane);
      L += f * sm_l[w][rr];
      acc.x += f * v.x; acc.y += f * v.y; acc.z += f * v.z; acc.w += f * v.w;
    }
    if (p.S == 1u) { const float inv = 1.0f / L; store(r0 + r, make_float4(acc.x * inv, acc.y * inv, acc.z * inv, acc.w * inv)); }
    else {
      *reinterpret_cast<float4*>(p.part + ((slab + split) * RB + r) * 128u + 4u * lane) = acc;
      if (lane == 0u) p.part_ml[(slab + split) * RB + r] = make_float2(M, L);
    }
  }
  if (p.S == 1u) return;
  // ---- the last block of this kv head and row block merges the splits
  __threadfence();
  __syncthreads();
  if (tid == 0u) {
    uint32_t* c = p.count + hk * gridDim.x + rb;
    const uint32_t last = atomicAdd(c, 1u) == p.S - 1u ? 1u : 0u;
    if (last) *c = 0u;
    sm_last = last;
  }
  __syncthreads();
  if (!sm_last) return;
  __threadfence();
  for (uint32_t r = warp; r < nrows; r += 4u) {
    float M = -INFINITY;
    for (uint32_t s = lane; s < p.S; s += 32u) M = fmaxf(M, __ldcg(&p.part_ml[(slab + s) * RB + r]).x);
#pragma unroll
    for (uint32_t x = 16; x > 0; x >>= 1) M = fmaxf(M, __shfl_xor_sync(0xffffffffu, M, x));
    float4 acc = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    float L = 0.0f;
    for (uint32_t s0 = 0; s0 < p.S; s0 += 8u) {
      float4 v[8]; float2 ml[8];
#pragma unroll
      for (uint32_t i = 0; i < 8u; i++) {
        const size_t at = (slab + min(s0 + i, p.S - 1u)) * RB + r;
        v[i] = __ldcg(reinterpret_cast<const float4*>(p.part + at * 128u) + lane); ml[i] = __ldcg(&p.part_ml[at]);
      }
#pragma unroll
      for (uint32_t i = 0; i < 8u; i++) {
        const float f = s0 + i < p.S ? at_ex2(ml[i].x - M) : 0.0f;      // (a split that saw no key of this row has maximum -inf: weight 0)
        L += f * ml[i].y;
        acc.x += f * v[i].x; acc.y += f * v[i].y; acc.z += f * v[i].z; acc.w += f * v[i].w;
      }
    }
    const float inv = 1.0f / L;
    store(r0 + r, make_float4(acc.x * inv, acc.y * inv, acc.z * inv, acc.w * inv));
  }
}

}  // namespace p0p
