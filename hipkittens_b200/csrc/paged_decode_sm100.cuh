// Paged-KV GQA decode for sm_100a: one query token per sequence, KV cache in 16-token pages that are
// reached through a block table. The reference has no such kernel; the math is the forward's
// (kernels/attn/gqa/kernel.cpp:569-573 for L) applied to one query row that sees its whole context.
//
// Split-K layout: a CTA owns part of the context of one (sequence, kv head) and all G = H / H_KV query heads of that kv
// head, so every K/V byte of the context is read exactly once. Inside the CTA each of the 4 or 8 warps streams its own
// pages through a private cp.async ring of 16-byte copies; scores and the PV product run on mma.sync m16n8k16 (bf16,
// fp32 accumulate) with the G heads in the 16-row M dimension, which is far more than an HBM-bound kernel needs and keeps
// the CUDA cores free for address generation and the exponentials.
// The CTAs of one (sequence, kv head) are a cluster, which splits the context evenly whatever its length and merges the
// partial results through distributed shared memory: one launch, nothing in the workspace. Where that would leave the GPU
// to a few CTAs (decode_pick_shape), a CTA takes a chunk of 512 or 1024 consecutive tokens instead; contexts of one chunk
// are finished in place, longer ones leave per-chunk (O, m, l) partials in the workspace, which
// `paged_decode_combine_kernel` merges.
#pragma once

#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include "dependent_launch.cuh"
#include "sm100_ptx.cuh"

namespace hk {

constexpr int kPageTokens = 16;
constexpr int kDecodeD = 128;
constexpr int kChunkPagesMin = 32;                    // pages per CTA: 32 (512 tokens) or 64 (1024 tokens),
constexpr int kChunkPagesMax = 64;                    // chosen per launch by decode_pick_chunk_pages
constexpr int kDecodeStages = 3;                      // pages in flight per warp
constexpr int kSlabBytes = kPageTokens * kDecodeD * 2;   // one page of one kv head: 4 KB
constexpr int kStageBytes = 2 * kSlabBytes;           // K slab + V slab
constexpr int decode_smem_bytes(int warps) { return warps * kDecodeStages * kStageBytes; }  // 96 or 192 KB
constexpr int kMaxCombineSplits = 256;

enum : int { kStatusBadPage = 2, kStatusBadLen = 4 };  // 3 is the backward kernels' kStatusSmemAlign

struct DecodeParams {
  const __nv_bfloat16* q;        // [S,1,H,128]
  const __nv_bfloat16* k_pages;  // [P,16,H_KV,128]
  const __nv_bfloat16* v_pages;
  const int32_t* block_table;    // [S,max_pages]
  const int32_t* ctx_lens;       // [S]
  __nv_bfloat16* o;              // [S,1,H,128]
  float* lse;                    // [S,H,1,1]
  int S, H, H_KV, max_pages, num_pages;
  int chunk_pages;               // pages per CTA (kChunkPagesMin or kChunkPagesMax)
  float scale, scale_log2;
  void* workspace;
  int* status;
};

// The workspace is laid out for the smaller chunk size (the larger split count), whichever size a launch uses.
__host__ __device__ inline int decode_max_splits(int max_pages) {
  return (max_pages + kChunkPagesMin - 1) / kChunkPagesMin;
}
// Chunks: 1024-token chunks halve the partial results and were measured 4-5 % faster on the 64-sequence workload
// (94.5 % vs 90.7 % of the copy bandwidth); 512-token chunks keep more CTAs in flight when the batch is
// small. Take the large chunk when it still gives every SM two rounds of two CTAs.
inline int decode_pick_chunk_pages(int S, int H_KV, int max_pages, int sm_count) {
  const long long ctas = 1ll * S * H_KV * ((max_pages + kChunkPagesMax - 1) / kChunkPagesMax);
  return ctas >= 4ll * sm_count ? kChunkPagesMax : kChunkPagesMin;
}
// What the device holds at once of the split kernel, by the size of its clusters (filled by prepare_decode_kernels).
struct DecodeLimits {
  int sm_count = 0;
  int clusters4[kMaxCluster + 1] = {};  // clusters of so many CTAs of 4 warps (two per SM)
  int clusters8 = 0;                    // clusters of kMaxCluster CTAs of 8 warps (one per SM)
};

// How the context of one (sequence, kv head), a unit, is spread: over a cluster of CTAs of 4 or 8 warps, or, with
// cluster = 0, over chunks that a second kernel combines. The host knows the block table's width and not the contexts;
// clusters spread each context evenly, so the width matters only for the most that one CTA may meet.
//  * Clusters as large as keeps all units in one wave, and no larger: a cluster behind the first wave starts when a whole
//    one fits, and one size too many costs more than it gives. us, chunks / clusters of that size / of another, H_KV 8 unless
//    said: 1 x 3250 tokens 10.4 / 7.6 (16) / 8.0 (8); 4 x 750 10.1 / 6.3 (8) / 6.7 (4), 11.4 (16); 8 x 2500 20.6 / 17.0
//    (4) / 22.6 (2), 19.0 (8); 40 x 1650 of H_KV 1 13.3 / 10.9 (6) / 14.1 (7).
//  * How much of one context a CTA may meet is bounded: the table may be as wide as it is for one long context among short
//    ones, which its own cluster then reads alone (12.5 us per 1000 tokens of a CTA of 4 warps, 5.5 with 8), where chunks
//    would spread it over the GPU. The lines are where that costs the one long context about as much as batches of equal
//    lengths gain. us, chunks / this, one context as long as the table beside others of 100 tokens, then all that long, then
//    all a quarter of that:
//    CTAs of 4 warps in clusters, 64 pages each: 8 x 3072 tokens of H_KV 8 (48 pages each) 10.8 / 10.4, 22.3 / 16.6, 11.7 / 6.7; 8 x
//    4096 10.8 / 12.4, 30.5 / 25.3, 11.9 / 7.2; 64 x 4096 of H_KV 1 9.8 / 11.9, 30.2 / 25.1, 12.3 / 7.3; behind the line 8 x 8192
//    12.3 / 19.8, 53.7 / 45.2, 14.0 / 10.0.
//    CTAs of their own of 8 warps (units for more than a wave in clusters of 3), 96 pages: 16 x 1408 10.8 / 10.7, 20.1 /
//    15.3, 9.1 / 5.6; 32 x 1536 11.1 / 11.4, 43.2 / 36.7, 10.6 / 10.4; behind the line 12 x 2560 10.4 / 16.5, 29.1 / 24.5, 12.3 /
//    7.2, 32 x 2048 10.3 / 14.0, 52.7 / 45.9, 12.5 / 11.9.
//    Of 4 warps, while one wave of those with 8 is not enough, 64 pages: 24 x 1024 10.6 / 11.2, 22.8 / 19.7, 8.1 / 6.3; 32 x 1024
//    10.6 / 12.5, 30.7 / 24.8, 8.6 / 6.3 (8 warps 8.9, 27.6, 9.1).
//    With units for more than two waves of those of 8 they are the better ones throughout, and the chunks are slower with the one
//    long context too: 80 pages, 64 x 1152 15.2 / 12.8, 57.6 / 49.9, 16.3 / 12.9 (8 warps 13.4, 55.2, 19.0).
//    One wave of CTAs of 8 warps also serves 160 pages where the chunks need more than two waves: then all but the one long
//    context gain most (18 x 2560 10.8 / 16.5, 40.9 / 32.6, 13.7 / 7.1, lengths evenly up to 2560 21.5 / 18.4).
//  * Clusters of several waves gain up to 5 % on long contexts (64 x 4350: 182 / 174 in clusters of 4), but where most of the
//    table's width is empty their idle CTAs cost more than those of the chunks (64 x 300 tokens in tables for 8192: 24 / 47),
//    so those stay in chunks.
//  * Few units with long contexts: 16 CTAs of 4 warps fall behind the chunks from some 700 tokens each on (1 x 14000 13.5 /
//    14.7); up to 6 units the CTAs can have 8 warps (H_KV 1, 1 x 16000: 11.7 / 11.0, 4 warps 12.5; below 4096 tokens 4
//    warps are better, 1 x 2000: 9.4 / 5.4, 8 warps 6.2).
struct DecodeShape {
  int cluster, warps;
};
inline DecodeShape decode_pick_shape(int S, int H_KV, int max_pages, const DecodeLimits& lim) {
  const long long units = 1ll * S * H_KV;
  constexpr DecodeShape kChunks{0, 4};
  int cluster = kMaxCluster, warps = 4;
  while (cluster > 1 && lim.clusters4[cluster] < units) --cluster;
  if (cluster < 3) {
    cluster = 1;
    const bool one_wave = units <= lim.sm_count, two_waves = units <= 2ll * lim.sm_count;
    const bool many_chunks = units * max_pages > 4ll * lim.sm_count * kChunkPagesMin;
    warps = one_wave || (two_waves && max_pages > 64) ? 8 : 4;
    if (max_pages > (one_wave && many_chunks ? 160 : two_waves ? 96 : 80)) return kChunks;
  } else if (max_pages > 256 && units <= lim.clusters8) {
    cluster = kMaxCluster;
    warps = 8;
    if (max_pages > 64 * cluster) return kChunks;
  } else if (max_pages > (cluster == kMaxCluster ? 44 : 64) * cluster) {
    return kChunks;
  }
  const int useful = (max_pages + warps - 1) / warps;  // a page per warp
  return {cluster < useful ? cluster : useful, warps};
}
// Workspace: partial O as fp32 [S][H][splits][128], then (m, l) pairs as fp32 [S][H][splits][2].
// Shapes the two kernels can be launched for: the combine kernel holds one weight per split in shared memory
// (kMaxCombineSplits of them, counted for the smaller chunk size so that either chunk choice fits), and sequences
// and kv heads are grid dimensions y and z.
inline bool decode_shape_supported(int S, int H_KV, int max_pages) {
  return S > 0 && S <= 65535 && H_KV > 0 && H_KV <= 65535 && max_pages > 0 &&
         decode_max_splits(max_pages) <= kMaxCombineSplits;
}
inline size_t decode_workspace_bytes(int S, int H, int D, int max_pages, int page_size) {
  if (S <= 0 || S > 65535 || H <= 0 || D != kDecodeD || page_size != kPageTokens || max_pages <= 0) return 0;
  if (decode_max_splits(max_pages) > kMaxCombineSplits) return 0;
  const size_t splits = decode_max_splits(max_pages);
  const size_t o_bytes = size_t(S) * H * splits * kDecodeD * sizeof(float);
  const size_t ml_bytes = size_t(S) * H * splits * 2 * sizeof(float);
  return ((o_bytes + 255) & ~size_t(255)) + ((ml_bytes + 255) & ~size_t(255));
}

namespace dec {

__device__ __forceinline__ void cp_async16(uint32_t dst, const void* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() {
  asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}
__device__ __forceinline__ void ldmatrix_x4(uint32_t addr, uint32_t& r0, uint32_t& r1, uint32_t& r2, uint32_t& r3) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];"
               : "=r"(r0), "=r"(r1), "=r"(r2), "=r"(r3)
               : "r"(addr));
}
__device__ __forceinline__ void ldmatrix_x4_trans(uint32_t addr, uint32_t& r0, uint32_t& r1, uint32_t& r2,
                                                  uint32_t& r3) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];"
               : "=r"(r0), "=r"(r1), "=r"(r2), "=r"(r3)
               : "r"(addr));
}
// D = A(16x16, row) * B(16x8, col) + D, bf16 inputs, fp32 accumulate.
__device__ __forceinline__ void mma_16816(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3,
                                          uint32_t b0, uint32_t b1) {
  asm volatile(
      "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
      : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
      : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

}  // namespace dec

// grid = (max_splits, H_KV, S), or (cluster size, H_KV, S) in clusters along x; block = 32 W threads, dynamic smem =
// decode_smem_bytes(W).
template <int G, bool CLUSTER, int W>
__global__ void __launch_bounds__(W * 32, W == 8 ? 1 : 2) paged_decode_split_kernel(const DecodeParams p) {
  using namespace dec;
  extern __shared__ __align__(128) uint8_t dsmem[];
  ptx::grid_dep_wait();
  ptx::grid_dep_launch();
  const int split = blockIdx.x, kvh = blockIdx.y, seq = blockIdx.z;
  // A length beyond what the block-table row can address is clamped to the row's capacity and reported; nothing
  // past the row is read.
  int ctx = p.ctx_lens[seq];
  if (ctx > p.max_pages * kPageTokens) {
    ctx = p.max_pages * kPageTokens;
    if (threadIdx.x == 0) atomicCAS(p.status, 0, kStatusBadLen);
  }
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int g = lane >> 2, t = lane & 3;
  const int total_pages = (ctx + kPageTokens - 1) / kPageTokens;
  // This warp's pages: page_first, page_first + page_step, ... below page_end. A CTA of a cluster takes every n_used-th
  // group of W pages, so that whatever the length the live CTAs of a cluster differ by a page per warp at most.
  int n_used, page_first, page_step, page_end;
  if constexpr (CLUSTER) {
    if (ctx <= 0) {  // defined output for an empty context
      if (split == 0) {
        for (int i = threadIdx.x; i < G * kDecodeD; i += W * 32)
          p.o[(size_t(seq) * p.H + kvh * G) * kDecodeD + i] = __float2bfloat16(0.f);
        if (threadIdx.x < G) p.lse[size_t(seq) * p.H + kvh * G + threadIdx.x] = -INFINITY;
      }
      return;
    }
    n_used = min(static_cast<int>(gridDim.x), (total_pages + W - 1) / W);  // a page for every warp of a live CTA
    if (split >= n_used) return;  // the cluster's barriers count the threads that are left
    page_first = split * W + warp;
    page_step = n_used * W;
    page_end = total_pages;
  } else {
    if (split * p.chunk_pages * kPageTokens >= ctx) return;
    n_used = 1;
    page_first = split * p.chunk_pages + warp;
    page_step = W;
    page_end = min(split * p.chunk_pages + p.chunk_pages, total_pages);
  }
  const float c = p.scale_log2;

  // page ids of this warp, one per lane: no warp has more than 32 pages (decode_pick_shape and the chunk sizes see to it)
  int my_id = 0;
  if (const int page = page_first + lane * page_step; page < page_end) {
    my_id = p.block_table[size_t(seq) * p.max_pages + page];
    if (my_id < 0 || my_id >= p.num_pages) {
      atomicCAS(p.status, 0, kStatusBadPage);  // never dereference an id outside the pool
      my_id = 0;
    }
  }

  // Q fragments: row g = head kvh*G+g (rows >= G are zero), 8 k-steps of 16 columns
  uint32_t qa[8][2];
  {
    const __nv_bfloat16* qrow = p.q + (size_t(seq) * p.H + kvh * G + (g < G ? g : 0)) * kDecodeD;
#pragma unroll
    for (int ks = 0; ks < 8; ++ks) {
      uint32_t lo = *reinterpret_cast<const uint32_t*>(qrow + ks * 16 + 2 * t);
      uint32_t hi = *reinterpret_cast<const uint32_t*>(qrow + ks * 16 + 8 + 2 * t);
      qa[ks][0] = (g < G) ? lo : 0u;
      qa[ks][1] = (g < G) ? hi : 0u;
    }
  }

  const uint32_t ring = ptx::smem_u32(dsmem) + warp * (kDecodeStages * kStageBytes);
  const size_t row_elems = size_t(p.H_KV) * kDecodeD;  // elements between consecutive tokens of a page

  // 16-byte gather of one page of this kv head: lane copies chunks lane, lane+32, ... of the 256
  // chunks (16 tokens x 16 chunks) of K and of V; chunk index is XOR-swizzled with the token so that
  // ldmatrix reads are bank-conflict free.
  auto fetch = [&](int i) {
    if (page_first + i * page_step < page_end) {
      const int id = __shfl_sync(0xffffffffu, my_id, i);
      const size_t base = (size_t(id) * kPageTokens) * row_elems + size_t(kvh) * kDecodeD;
      const uint32_t st = ring + (i % kDecodeStages) * kStageBytes;
#pragma unroll
      for (int r = 0; r < 8; ++r) {
        const int ch_lin = r * 32 + lane;
        const int tok = ch_lin >> 4, ch = ch_lin & 15;
        const size_t src = base + size_t(tok) * row_elems + ch * 8;
        const uint32_t dst = tok * 256 + ((ch ^ (tok & 7)) << 4);
        cp_async16(st + dst, p.k_pages + src);
        cp_async16(st + kSlabBytes + dst, p.v_pages + src);
      }
    }
    cp_async_commit();
  };

  float oacc[16][4];
#pragma unroll
  for (int j = 0; j < 16; ++j) oacc[j][0] = oacc[j][1] = oacc[j][2] = oacc[j][3] = 0.f;
  float m = -INFINITY, l = 0.f;

#pragma unroll
  for (int i = 0; i < kDecodeStages - 1; ++i) fetch(i);

  for (int i = 0, page = page_first; page < page_end; ++i, page += page_step) {
    fetch(i + kDecodeStages - 1);
    cp_async_wait<kDecodeStages - 1>();
    __syncwarp();
    const uint32_t sK = ring + (i % kDecodeStages) * kStageBytes;
    const uint32_t sV = sK + kSlabBytes;

    // ---- S[16 x 16 tokens] = Q K^T, in two halves of the head dimension: a warp has one page at a time, and with one
    // accumulator per 8 tokens the eight products on it wait for one another
    float sc[2][4] = {{0.f, 0.f, 0.f, 0.f}, {0.f, 0.f, 0.f, 0.f}};
    {
      float sd[2][4] = {{0.f, 0.f, 0.f, 0.f}, {0.f, 0.f, 0.f, 0.f}};
      const int mi = lane >> 3, r = lane & 7;
      const int tok = r + 8 * (mi >> 1);
#pragma unroll
      for (int ks = 0; ks < 8; ++ks) {
        const int ch = ks * 2 + (mi & 1);
        uint32_t b0, b1, b2, b3;
        ldmatrix_x4(sK + tok * 256 + ((ch ^ (tok & 7)) << 4), b0, b1, b2, b3);
        mma_16816(ks & 1 ? sd[0] : sc[0], qa[ks][0], 0u, qa[ks][1], 0u, b0, b1);
        mma_16816(ks & 1 ? sd[1] : sc[1], qa[ks][0], 0u, qa[ks][1], 0u, b2, b3);
      }
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        sc[0][e] += sd[0][e];
        sc[1][e] += sd[1][e];
      }
    }
    // ---- online softmax over this page (row g, tokens nt*8 + 2t + {0,1})
    const int tok_base = page * kPageTokens;
    float sv[4] = {sc[0][0], sc[0][1], sc[1][0], sc[1][1]};
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const int tok = tok_base + (e >> 1) * 8 + 2 * t + (e & 1);
      if (tok >= ctx) sv[e] = -INFINITY;
    }
    float pm = fmaxf(fmaxf(sv[0], sv[1]), fmaxf(sv[2], sv[3]));
    pm = fmaxf(pm, __shfl_xor_sync(0xffffffffu, pm, 1));
    pm = fmaxf(pm, __shfl_xor_sync(0xffffffffu, pm, 2));
    const float m_new = fmaxf(m, pm);
    if (__any_sync(0xffffffffu, (m_new - m) * c > kRescaleThresholdLog2)) {
      const float alpha = ptx::ex2_approx((m - m_new) * c);  // m = -inf on the first page gives 0
      l *= alpha;
#pragma unroll
      for (int j = 0; j < 16; ++j) {
        oacc[j][0] *= alpha;
        oacc[j][1] *= alpha;
      }
      m = m_new;
    }
    const float mc = m * c;
    float pv[4];
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      pv[e] = ptx::ex2_approx(fmaf(sv[e], c, -mc));
      l += pv[e];
    }
    const uint32_t pa0 = ptx::pack_bf16x2(pv[0], pv[1]);
    const uint32_t pa2 = ptx::pack_bf16x2(pv[2], pv[3]);
    // ---- O[16 x 128] += P[16 x 16 tokens] V[16 tokens x 128]
    {
      const int mi = lane >> 3, r = lane & 7;
      const int tok = r + 8 * (mi & 1);
#pragma unroll
      for (int jp = 0; jp < 8; ++jp) {
        const int ch = jp * 2 + (mi >> 1);
        uint32_t b0, b1, b2, b3;
        ldmatrix_x4_trans(sV + tok * 256 + ((ch ^ (tok & 7)) << 4), b0, b1, b2, b3);
        mma_16816(oacc[2 * jp], pa0, 0u, pa2, 0u, b0, b1);
        mma_16816(oacc[2 * jp + 1], pa0, 0u, pa2, 0u, b2, b3);
      }
    }
    __syncwarp();
  }
  cp_async_wait<0>();
  l += __shfl_xor_sync(0xffffffffu, l, 1);
  l += __shfl_xor_sync(0xffffffffu, l, 2);

  // ---- merge the W warps through shared memory (the ring is idle now)
  __syncthreads();
  float* sm_o = reinterpret_cast<float*>(dsmem);  // [W][8][128]
  float* sm_m = sm_o + W * 8 * kDecodeD;          // [W][8]
  float* sm_l = sm_m + W * 8;                     // [W][8]
#pragma unroll
  for (int j = 0; j < 16; ++j) {
    float2 v2 = make_float2(oacc[j][0], oacc[j][1]);
    *reinterpret_cast<float2*>(sm_o + (warp * 8 + g) * kDecodeD + j * 8 + 2 * t) = v2;
  }
  if (t == 0) {
    sm_m[warp * 8 + g] = m;
    sm_l[warp * 8 + g] = l;
  }
  __syncthreads();
  // 128 threads <-> 128 output columns; with 8 warps each half of them takes every other head of the group
  constexpr int kHalves = W / 4, kHeads = (G + kHalves - 1) / kHalves;
  const int d = threadIdx.x & (kDecodeD - 1), h0 = threadIdx.x / kDecodeD;
  // per head of this thread: reference maximum, row sum and this thread's column of the CTA's share
  float M[kHeads], L[kHeads], acc[kHeads];
#pragma unroll
  for (int i = 0; i < kHeads; ++i) {
    const int h = min(i * kHalves + h0, G - 1);
    M[i] = sm_m[h];
#pragma unroll
    for (int w = 1; w < W; ++w) M[i] = fmaxf(M[i], sm_m[w * 8 + h]);
    acc[i] = L[i] = 0.f;
#pragma unroll
    for (int w = 0; w < W; ++w) {
      const float wgt = ptx::ex2_approx((sm_m[w * 8 + h] - M[i]) * c);
      acc[i] += wgt * sm_o[(w * 8 + h) * kDecodeD + d];
      L[i] += wgt * sm_l[w * 8 + h];
    }
  }
  if constexpr (CLUSTER) {
    if (n_used > 1) {
      // ---- merge the CTAs of the cluster: each leaves its share in its own shared memory, and CTA r reads all of
      // head r, r + n_used, ... in the order of the ranks
      float* cl_o = sm_l + W * 8;          // [G][128]
      float* cl_ml = cl_o + 8 * kDecodeD;  // [G][2]
#pragma unroll
      for (int i = 0; i < kHeads; ++i) {
        const int h = i * kHalves + h0;
        if (h >= G) break;
        cl_o[h * kDecodeD + d] = acc[i];
        if (d == 0) {
          cl_ml[2 * h] = M[i];
          cl_ml[2 * h + 1] = L[i];
        }
      }
      ptx::cluster_arrive();
      ptx::cluster_wait();
      for (int h = split * kHalves + h0; h < G; h += n_used * kHalves) {
        float m_r[kMaxCluster], l_r[kMaxCluster], o_r[kMaxCluster];
        const uint32_t a_ml = ptx::smem_u32(cl_ml + 2 * h), a_o = ptx::smem_u32(cl_o + h * kDecodeD + d);
#pragma unroll
        for (int r = 0; r < kMaxCluster; ++r) {
          m_r[r] = -INFINITY;
          l_r[r] = o_r[r] = 0.f;
          if (r < n_used) {
            const uint32_t ml = ptx::map_to_rank(a_ml, r);
            m_r[r] = ptx::ld_cluster(ml);
            l_r[r] = ptx::ld_cluster(ml + 4);
            o_r[r] = ptx::ld_cluster(ptx::map_to_rank(a_o, r));
          }
        }
        float Mc = m_r[0];
#pragma unroll
        for (int r = 1; r < kMaxCluster; ++r) Mc = fmaxf(Mc, m_r[r]);
        float sum = 0.f, out = 0.f;
#pragma unroll
        for (int r = 0; r < kMaxCluster; ++r) {
          const float wgt = ptx::ex2_approx((m_r[r] - Mc) * c);
          sum += wgt * l_r[r];
          out += wgt * o_r[r];
        }
        const size_t row = size_t(seq) * p.H + kvh * G + h;
        p.o[row * kDecodeD + d] = __float2bfloat16(out / sum);
        if (d == 0) p.lse[row] = Mc * p.scale + __logf(sum);
      }
      ptx::cluster_arrive();  // nobody leaves while its shared memory is being read
      ptx::cluster_wait();
      return;
    }
  }
  const int n_splits = CLUSTER ? 1 : (total_pages + p.chunk_pages - 1) / p.chunk_pages;
  const int max_splits = decode_max_splits(p.max_pages);
  float* ws_o = reinterpret_cast<float*>(p.workspace);
  const size_t o_bytes = (size_t(p.S) * p.H * max_splits * kDecodeD * sizeof(float) + 255) & ~size_t(255);
  float* ws_ml = reinterpret_cast<float*>(reinterpret_cast<uint8_t*>(p.workspace) + o_bytes);
#pragma unroll
  for (int i = 0; i < kHeads; ++i) {
    const int h = i * kHalves + h0;
    if (h >= G) break;
    const size_t row = size_t(seq) * p.H + kvh * G + h;
    if (n_splits == 1) {
      p.o[row * kDecodeD + d] = __float2bfloat16(acc[i] / L[i]);
      if (d == 0) p.lse[row] = M[i] * p.scale + __logf(L[i]);
    } else {
      const size_t slot = row * max_splits + split;
      ws_o[slot * kDecodeD + d] = acc[i];
      if (d == 0) {
        ws_ml[slot * 2] = M[i];
        ws_ml[slot * 2 + 1] = L[i];
      }
    }
  }
}

// grid = (H, S), block = 128 threads (one per output column). Merges the per-chunk partials of
// sequences that span more than one chunk.
__global__ void __launch_bounds__(kDecodeD) paged_decode_combine_kernel(const DecodeParams p) {
  ptx::grid_dep_wait();  // from here on the split grid has completed and its partials are visible
  ptx::grid_dep_launch();
  const int head = blockIdx.x, seq = blockIdx.y;
  const int ctx = min(p.ctx_lens[seq], p.max_pages * kPageTokens);  // clamped as in the split kernel, which reports it
  const int d = threadIdx.x;
  if (ctx <= 0) {  // defined output for an empty context
    p.o[(size_t(seq) * p.H + head) * kDecodeD + d] = __float2bfloat16(0.f);
    if (d == 0) p.lse[size_t(seq) * p.H + head] = -INFINITY;
    return;
  }
  const int chunk_tokens = p.chunk_pages * kPageTokens;
  const int n_splits = (ctx + chunk_tokens - 1) / chunk_tokens;
  if (n_splits == 1) return;  // finished by the split kernel
  const int max_splits = decode_max_splits(p.max_pages);
  const float* ws_o = reinterpret_cast<const float*>(p.workspace);
  const size_t o_bytes = (size_t(p.S) * p.H * max_splits * kDecodeD * sizeof(float) + 255) & ~size_t(255);
  const float* ws_ml = reinterpret_cast<const float*>(reinterpret_cast<const uint8_t*>(p.workspace) + o_bytes);
  const size_t slot0 = (size_t(seq) * p.H + head) * max_splits;
  __shared__ float s_w[kMaxCombineSplits];
  __shared__ float s_M, s_L;
  if (threadIdx.x < 32) {
    float M = -INFINITY;
    for (int i = threadIdx.x; i < n_splits; i += 32) M = fmaxf(M, ws_ml[(slot0 + i) * 2]);
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) M = fmaxf(M, __shfl_xor_sync(0xffffffffu, M, off));
    float L = 0.f;
    for (int i = threadIdx.x; i < n_splits; i += 32) {
      const float w = ptx::ex2_approx((ws_ml[(slot0 + i) * 2] - M) * p.scale_log2);
      s_w[i] = w;
      L += w * ws_ml[(slot0 + i) * 2 + 1];
    }
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) L += __shfl_xor_sync(0xffffffffu, L, off);
    if (threadIdx.x == 0) {
      s_M = M;
      s_L = L;
    }
  }
  __syncthreads();
  float acc = 0.f;
#pragma unroll 4
  for (int i = 0; i < n_splits; ++i) acc += s_w[i] * ws_o[(slot0 + i) * kDecodeD + d];
  p.o[(size_t(seq) * p.H + head) * kDecodeD + d] = __float2bfloat16(acc / s_L);
  if (d == 0) p.lse[size_t(seq) * p.H + head] = s_M * p.scale + __logf(s_L);
}

template <int G, bool CLUSTER, int W>
cudaError_t prepare_decode_kernel() {
  auto* fn = paged_decode_split_kernel<G, CLUSTER, W>;
  const cudaError_t e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, decode_smem_bytes(W));
  if (e != cudaSuccess || !CLUSTER) return e;
  return cudaFuncSetAttribute(fn, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
}
template <int G>
cudaError_t prepare_decode_kernels_of() {
  cudaError_t e = prepare_decode_kernel<G, false, 4>();
  if (e == cudaSuccess) e = prepare_decode_kernel<G, true, 4>();
  if (e == cudaSuccess) e = prepare_decode_kernel<G, true, 8>();
  return e;
}
inline int prepare_decode_kernels(char* err, size_t err_len, int sm_count, DecodeLimits* lim) {
  for (auto* prepare : {prepare_decode_kernels_of<1>, prepare_decode_kernels_of<2>, prepare_decode_kernels_of<3>,
                        prepare_decode_kernels_of<4>, prepare_decode_kernels_of<5>, prepare_decode_kernels_of<6>,
                        prepare_decode_kernels_of<7>, prepare_decode_kernels_of<8>}) {
    const cudaError_t e = prepare();
    if (e != cudaSuccess) {
      snprintf(err, err_len, "decode kernel attribute: %s", cudaGetErrorString(e));
      return -3;
    }
  }
  lim->sm_count = sm_count;
  for (int n = 2; n <= kMaxCluster; ++n) lim->clusters4[n] = clusters_held(paged_decode_split_kernel<8, true, 4>, 4 * 32, decode_smem_bytes(4), n);
  lim->clusters8 = clusters_held(paged_decode_split_kernel<8, true, 8>, 8 * 32, decode_smem_bytes(8), kMaxCluster);
  return 0;
}

template <int G>
cudaError_t launch_decode_split(const DecodeParams& p, int splits, int cluster, int warps, cudaStream_t stream) {
  const dim3 grid(cluster ? cluster : splits, p.H_KV, p.S);
  if (cluster == 0)
    return launch_dependent(true, paged_decode_split_kernel<G, false, 4>, grid, 128, decode_smem_bytes(4), stream, p);
  auto* fn = warps == 8 ? paged_decode_split_kernel<G, true, 8> : paged_decode_split_kernel<G, true, 4>;
  return launch_dependent(true, fn, grid, warps * 32, decode_smem_bytes(warps), stream, ClusterX{unsigned(cluster)}, p);
}

inline cudaError_t launch_paged_decode(DecodeParams p, const DecodeLimits& lim, cudaStream_t stream, int* launched) {
  const DecodeShape shape = decode_pick_shape(p.S, p.H_KV, p.max_pages, lim);
  const int cluster = shape.cluster, warps = shape.warps;
  p.chunk_pages = decode_pick_chunk_pages(p.S, p.H_KV, p.max_pages, lim.sm_count);
  const int splits = (p.max_pages + p.chunk_pages - 1) / p.chunk_pages;
  if (splits > kMaxCombineSplits) return cudaErrorInvalidValue;
  cudaError_t e;
  switch (p.H / p.H_KV) {
#define HK_CASE(g) \
  case g: e = launch_decode_split<g>(p, splits, cluster, warps, stream); break;
    HK_CASE(1) HK_CASE(2) HK_CASE(3) HK_CASE(4) HK_CASE(5) HK_CASE(6) HK_CASE(7) HK_CASE(8)
#undef HK_CASE
    default: return cudaErrorInvalidValue;
  }
  *launched += 1;
  if (e != cudaSuccess || cluster) return e;
  e = launch_dependent(true, paged_decode_combine_kernel, dim3(p.H, p.S), kDecodeD, 0, stream, p);
  *launched += 1;
  return e;
}

}  // namespace hk
