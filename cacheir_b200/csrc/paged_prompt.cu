// Causal attention of prompt rows over the paged pool: fp16, head_dim 64 or 128, 16-token pages.
//
// The rows of a step belong to sequences; a tile is up to 64 (token, head) rows of neighbouring tokens of one sequence and
// one KV head (16 tokens at four heads per KV head), so that the keys and values it shares are fetched once for all of them
// instead of once per token. One CTA per (tile, KV head): a producer warp walks the sequence's page table and brings four pages
// of K and V (64 keys, 32 KB at head_dim 128) per stage with TMA tensor copies, four warps take 16 rows each: S = Q K^T and
// O += P V on the tensor cores (mma.sync, fp32 accumulation), running maximum and sum per row in registers as in the decode
// kernel. A warp reads 32 KB of shared memory per 64 keys for 128 MMAs: both take about 256 cycles, which is the bound. Two CTAs share an
// SM. 2048 tokens, 32 heads of 128 on 8 KV heads: 160 us, 211 TFLOP/s; the MMAs alone are 119 us at the
// 512 multiplications per clock and SM that mma.sync reaches here. Pages past a warp's last token are skipped, only the page that holds it is masked. The host lists tiles with
// the most keys first.
#include <cuda.h>

#include "common.cuh"
#include "paged_attention_common.cuh"
#include "tc_ptx.cuh"

namespace cb200 {
namespace {

using namespace ptx;

constexpr int kPage = 16;
constexpr int kStagePages = 4;
constexpr int kStages = 3;
constexpr int kWarps = 4;
constexpr int kThreads = (kWarps + 1) * 32;
constexpr int kTileRows = 16 * kWarps;

__device__ int g_prompt_status = 0;

struct PromptParams {
  const __half* q;
  __half* out;
  const int32_t* page_table;   // [sequences][max_pages]
  const int4* tiles;           // (sequence, first row, first position, tokens)
  const int* n_tiles;
  long long q_stride, out_stride;
  int kv_heads, group, max_pages, num_sequences;
  float scale_log2;
};

__device__ __forceinline__ void tma_load_3d(uint32_t dst, const CUtensorMap* map, uint32_t bar, int x, int y, int z) {
  asm volatile(
      "cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5}], [%2];"
      ::"r"(dst), "l"(reinterpret_cast<uint64_t>(map)), "r"(bar), "r"(x), "r"(y), "r"(z) : "memory");
}
__device__ __forceinline__ void ldmatrix_x4(uint32_t addr, uint32_t (&r)[4]) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr));
}
__device__ __forceinline__ void ldmatrix_x4_trans(uint32_t addr, uint32_t (&r)[4]) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr));
}
__device__ __forceinline__ void mma_16816(float (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
               : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
               : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
__device__ __forceinline__ uint32_t pack_halves(float lo, float hi) {
  const __half2 v = __floats2half2_rn(lo, hi);
  return *reinterpret_cast<const uint32_t*>(&v);
}

template <int D>
__global__ void __launch_bounds__(kThreads, 2)
paged_prompt_kernel(const __grid_constant__ CUtensorMap tmap_k, const __grid_constant__ CUtensorMap tmap_v, const PromptParams p) {
  chain_enter();
  constexpr int kTileBytes = kPage * D * 2;        // one K or V page of one head
  constexpr int kPageBytes = 2 * kTileBytes;
  constexpr int kStageBytes = kStagePages * kPageBytes;
  constexpr int kKSteps = D / 16;
  constexpr int kDimTiles = D / 8;

  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~static_cast<uintptr_t>(1023));
  uint64_t* full = reinterpret_cast<uint64_t*>(smem + kStages * kStageBytes);
  uint64_t* empty = full + kStages;

  const int tile_index = blockIdx.x / p.kv_heads, kvh = blockIdx.x % p.kv_heads;
  if (tile_index >= *p.n_tiles) return;
  const int4 tile = p.tiles[tile_index];
  const int tokens = tile.w;
  if (tile.x < 0 || tile.x >= p.num_sequences || tokens <= 0) return;
  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  const int pages = min((tile.z + tokens + kPage - 1) / kPage, p.max_pages);
  const int iters = (pages + kStagePages - 1) / kStagePages;

  if (threadIdx.x == 0) {
    for (int s = 0; s < kStages; ++s) {
      mbar_init(smem_u32(&full[s]), 1);
      mbar_init(smem_u32(&empty[s]), kWarps);
    }
    mbar_fence_init();
  }
  __syncthreads();

  if (warp == kWarps) {
    // ---------------- copies: lane j brings page j of each stage ----------------
    const int32_t* table = p.page_table + static_cast<size_t>(tile.x) * p.max_pages;
    int next = lane < min(kStagePages, pages) ? table[lane] : 0;          // page ids one stage ahead
    bool ok = true;
    int issued = 0;
    for (int it = 0; it < iters && ok; ++it) {
      const int s = it % kStages, first = it * kStagePages, count = min(kStagePages, pages - first);
      const int page = next;
      if (lane < kStagePages && first + kStagePages + lane < pages) next = table[first + kStagePages + lane];
      if (lane == 0) {
        ok = it < kStages || mbar_wait(smem_u32(&empty[s]), ((it / kStages) & 1) ^ 1, &g_prompt_status, (13 << 8) | 1);
        if (ok) mbar_expect_tx(smem_u32(&full[s]), count * kPageBytes);
      }
      ok = __shfl_sync(0xffffffffu, ok ? 1 : 0, 0) != 0;
      if (ok && lane < count) {
        const uint32_t dst = smem_u32(smem + s * kStageBytes + lane * kPageBytes);
        const int row = (page * p.kv_heads + kvh) * kPage;
        tma_load_3d(dst, &tmap_k, smem_u32(&full[s]), 0, row, 0);
        tma_load_3d(dst + kTileBytes, &tmap_v, smem_u32(&full[s]), 0, row, 0);
        issued = it + 1;
      }
    }
    // nothing may still be on its way when the block ends (a consumer's wait may have given up); lane 0 copies in every stage
    if (lane == 0)
      for (int it = issued > kStages ? issued - kStages : 0; it < issued; ++it)
        if (!mbar_wait(smem_u32(&full[it % kStages]), (it / kStages) & 1, &g_prompt_status, (13 << 8) | 4)) break;
    return;
  }

  // ---------------- 16 rows per warp: row = token * group + head ----------------
  const int g = lane >> 2, t4 = lane & 3;
  const int first_row = warp * 16;
  if (first_row >= tokens * p.group) {             // nothing for this warp: it only keeps the ring moving
    for (int it = 0; it < iters; ++it) {
      const int s = it % kStages;
      const bool ok = __all_sync(0xffffffffu, mbar_wait(smem_u32(&full[s]), (it / kStages) & 1, &g_prompt_status, (13 << 8) | 2));
      if (!ok) break;
      if (lane == 0) mbar_arrive(smem_u32(&empty[s]));
    }
    return;
  }
  const int last_token = min((first_row + 15) / p.group, tokens - 1);
  const int warp_pages = min((tile.z + last_token) / kPage + 1, pages);
  const int clear_pages = (tile.z + first_row / p.group + 1) / kPage;      // pages that every row of the warp sees whole
  int pos[2];
  uint32_t qa[kKSteps][4];
  const __half* q_row[2];
  __half* out_row[2];
#pragma unroll
  for (int r = 0; r < 2; ++r) {
    const int row = first_row + g + 8 * r, token = row / p.group;
    const int at = min(token, tokens - 1), head = kvh * p.group + row % p.group;
    pos[r] = tile.z + at;
    q_row[r] = p.q + static_cast<size_t>(tile.y + at) * p.q_stride + static_cast<size_t>(head) * D;
    out_row[r] = token < tokens ? p.out + static_cast<size_t>(tile.y + at) * p.out_stride + static_cast<size_t>(head) * D : nullptr;
  }
#pragma unroll
  for (int ks = 0; ks < kKSteps; ++ks)
#pragma unroll
    for (int r = 0; r < 4; ++r) qa[ks][r] = *reinterpret_cast<const uint32_t*>(q_row[r & 1] + ks * 16 + 2 * t4 + (r >> 1) * 8);

  float m_run[2] = {-INFINITY, -INFINITY}, l_run[2] = {0.f, 0.f};
  float o[kDimTiles][4];
#pragma unroll
  for (int i = 0; i < kDimTiles; ++i) o[i][0] = o[i][1] = o[i][2] = o[i][3] = 0.f;
  const uint32_t lrow = lane & 7, lmat = lane >> 3;
  bool ok = true;
  for (int it = 0; it < iters; ++it) {
    const int s = it % kStages;
    ok = __all_sync(0xffffffffu, mbar_wait(smem_u32(&full[s]), (it / kStages) & 1, &g_prompt_status, (13 << 8) | 3));
    if (!ok) break;
    const int count = min(kStagePages, warp_pages - it * kStagePages);     // pages of the stage this warp looks at
    if (count > 0) {
      const uint32_t stage = smem_u32(smem + s * kStageBytes);
      float sc[kStagePages][2][4];
      float top[2] = {-INFINITY, -INFINITY};
#pragma unroll
      for (int pg = 0; pg < kStagePages; ++pg) {
#pragma unroll
        for (int nt = 0; nt < 2; ++nt) {
          sc[pg][nt][0] = sc[pg][nt][1] = sc[pg][nt][2] = sc[pg][nt][3] = 0.f;
          if (pg < count) {
            const uint32_t token = nt * 8 + lrow;
#pragma unroll
            for (int kk = 0; kk < kKSteps / 2; ++kk) {
              const uint32_t c = 4 * kk + lmat;
              uint32_t kb[4];
              ldmatrix_x4(stage + pg * kPageBytes + (c >> 3) * (kPage * 128) + token * 128 + (((c & 7) ^ (token & 7)) << 4), kb);
              mma_16816(sc[pg][nt], qa[2 * kk], kb[0], kb[1]);
              mma_16816(sc[pg][nt], qa[2 * kk + 1], kb[2], kb[3]);
            }
          }
        }
        const int page = it * kStagePages + pg;
        if (pg < count && page < clear_pages) {
#pragma unroll
          for (int nt = 0; nt < 2; ++nt)
#pragma unroll
            for (int e = 0; e < 4; ++e) top[e >> 1] = fmaxf(top[e >> 1], sc[pg][nt][e]);
        } else {
#pragma unroll
          for (int nt = 0; nt < 2; ++nt)
#pragma unroll
            for (int e = 0; e < 4; ++e) {
              const int key = page * kPage + nt * 8 + 2 * t4 + (e & 1);
              if (pg >= count || key > pos[e >> 1]) sc[pg][nt][e] = -INFINITY;
              top[e >> 1] = fmaxf(top[e >> 1], sc[pg][nt][e]);
            }
        }
      }
      float corr[2], base[2];
#pragma unroll
      for (int r = 0; r < 2; ++r) {
        top[r] = fmaxf(top[r], __shfl_xor_sync(0xffffffffu, top[r], 1));
        top[r] = fmaxf(top[r], __shfl_xor_sync(0xffffffffu, top[r], 2));
        const float m_new = fmaxf(m_run[r], top[r] * p.scale_log2);        // finite: the first page holds a key of every row
        corr[r] = exp2f(m_run[r] - m_new);
        m_run[r] = m_new;
        base[r] = -m_new;
      }
#pragma unroll
      for (int pg = 0; pg < kStagePages; ++pg)
#pragma unroll
        for (int nt = 0; nt < 2; ++nt)
#pragma unroll
          for (int e = 0; e < 4; ++e) sc[pg][nt][e] = exp2f(fmaf(sc[pg][nt][e], p.scale_log2, base[e >> 1]));
#pragma unroll
      for (int r = 0; r < 2; ++r) {
        float sum = 0.f;
#pragma unroll
        for (int pg = 0; pg < kStagePages; ++pg)
          sum += (sc[pg][0][2 * r] + sc[pg][0][2 * r + 1]) + (sc[pg][1][2 * r] + sc[pg][1][2 * r + 1]);
        l_run[r] = fmaf(l_run[r], corr[r], sum);
      }
      if (__any_sync(0xffffffffu, corr[0] != 1.f || corr[1] != 1.f)) {     // (a maximum moved)
#pragma unroll
        for (int i = 0; i < kDimTiles; ++i) { o[i][0] *= corr[0]; o[i][1] *= corr[0]; o[i][2] *= corr[1]; o[i][3] *= corr[1]; }
      }
#pragma unroll
      for (int pg = 0; pg < kStagePages; ++pg) {
        if (pg < count) {
          const uint32_t pa[4] = {pack_halves(sc[pg][0][0], sc[pg][0][1]), pack_halves(sc[pg][0][2], sc[pg][0][3]),
                                  pack_halves(sc[pg][1][0], sc[pg][1][1]), pack_halves(sc[pg][1][2], sc[pg][1][3])};
          const uint32_t token = (lmat & 1) * 8 + lrow;
#pragma unroll
          for (int j = 0; j < kDimTiles / 2; ++j) {
            const uint32_t c = 2 * j + (lmat >> 1);
            uint32_t vb[4];
            ldmatrix_x4_trans(stage + pg * kPageBytes + kTileBytes + (c >> 3) * (kPage * 128) + token * 128 + (((c & 7) ^ (token & 7)) << 4), vb);
            mma_16816(o[2 * j], pa, vb[0], vb[1]);
            mma_16816(o[2 * j + 1], pa, vb[2], vb[3]);
          }
        }
      }
    }
    __syncwarp();
    if (lane == 0) mbar_arrive(smem_u32(&empty[s]));
  }
#pragma unroll
  for (int r = 0; r < 2; ++r) {
    l_run[r] += __shfl_xor_sync(0xffffffffu, l_run[r], 1);
    l_run[r] += __shfl_xor_sync(0xffffffffu, l_run[r], 2);
    if (!out_row[r]) continue;
    const float inv = l_run[r] > 0.f ? 1.f / l_run[r] : 0.f;
#pragma unroll
    for (int i = 0; i < kDimTiles; ++i)
      *reinterpret_cast<uint32_t*>(out_row[r] + 8 * i + 2 * t4) = pack_halves(o[i][2 * r] * inv, o[i][2 * r + 1] * inv);
  }
}

// The pool [slots, kv_heads, 16, D] as [D/64 spans][rows][64 elements]: a box {64, 16, D/64} is one page of one head.
bool encode_pool(CUtensorMap* map, const void* base, uint64_t rows, int head_dim) {
  EncodeTiledFn fn = tensor_map_encoder();
  if (!fn) return false;
  const cuuint64_t dims[3] = {64, rows, static_cast<cuuint64_t>(head_dim / 64)};
  const cuuint64_t strides[2] = {static_cast<cuuint64_t>(head_dim) * 2, 128};
  const cuuint32_t box[3] = {64, kPage, static_cast<cuuint32_t>(head_dim / 64)};
  const cuuint32_t elem_strides[3] = {1, 1, 1};
  return fn(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 3, const_cast<void*>(base), dims, strides, box, elem_strides, CU_TENSOR_MAP_INTERLEAVE_NONE,
            CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

template <int D>
int launch(const PromptParams& p, const void* k_cache, const void* v_cache, uint64_t pool_rows, int max_tiles, cudaStream_t stream) {
  CUtensorMap tmap_k, tmap_v;
  if (!encode_pool(&tmap_k, k_cache, pool_rows, D) || !encode_pool(&tmap_v, v_cache, pool_rows, D)) return CACHEIR_B200_EUNSUPPORTED;
  constexpr int kSmem = 1024 + kStages * kStagePages * 2 * kPage * D * 2 + 2 * kStages * 8;
  auto kern = paged_prompt_kernel<D>;
  const cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmem);
  if (e != cudaSuccess) return static_cast<int>(e);
  launch_chained(kern, max_tiles * p.kv_heads, kThreads, kSmem, stream, tmap_k, tmap_v, p);
  return launch_status();
}

}  // namespace

int paged_prompt_device_status(bool reset) {
  int status = 0;
  if (cudaMemcpyFromSymbol(&status, g_prompt_status, sizeof(int)) != cudaSuccess) return -1;
  if (reset && status != 0) {
    const int zero = 0;
    cudaMemcpyToSymbol(g_prompt_status, &zero, sizeof(int));
  }
  return status;
}

}  // namespace cb200

using namespace cb200;

extern "C" int cacheir_b200_paged_attention_prompt(const void* q, const void* k_cache, const void* v_cache, const int32_t* page_table,
                                                   const int32_t* tiles, const int32_t* n_tiles, void* out, int max_tiles, int num_sequences,
                                                   int heads, int kv_heads, int max_pages, int page_size, int head_dim, long long q_stride,
                                                   long long out_stride, float softmax_scale, int num_slots, void* stream) {
  if (max_tiles <= 0) return 0;
  if (!q || !k_cache || !v_cache || !page_table || !tiles || !n_tiles || !out) return CACHEIR_B200_EINVAL;
  if (num_sequences <= 0 || heads <= 0 || kv_heads <= 0 || heads % kv_heads != 0 || max_pages <= 0 || num_slots <= 0) return CACHEIR_B200_EINVAL;
  if (page_size != kPage || (head_dim != 64 && head_dim != 128) || heads / kv_heads > kTileRows) return CACHEIR_B200_EUNSUPPORTED;
  if (!aligned_to(k_cache, 16) || !aligned_to(v_cache, 16) || !aligned_to(q, 4) || !aligned_to(out, 4) || !aligned_to(tiles, 16) ||
      q_stride % 2 != 0 || out_stride % 2 != 0)
    return CACHEIR_B200_EALIGN;
  PromptParams p{};
  p.q = static_cast<const __half*>(q); p.out = static_cast<__half*>(out);
  p.page_table = page_table; p.tiles = reinterpret_cast<const int4*>(tiles); p.n_tiles = n_tiles;
  p.q_stride = q_stride; p.out_stride = out_stride;
  p.kv_heads = kv_heads; p.group = heads / kv_heads; p.max_pages = max_pages; p.num_sequences = num_sequences;
  const float scale = softmax_scale > 0.f ? softmax_scale : 1.f / sqrtf(static_cast<float>(head_dim));
  p.scale_log2 = scale * kLog2e;
  const uint64_t rows = static_cast<uint64_t>(num_slots) * kv_heads * kPage;
  return head_dim == 128 ? launch<128>(p, k_cache, v_cache, rows, max_tiles, as_stream(stream))
                         : launch<64>(p, k_cache, v_cache, rows, max_tiles, as_stream(stream));
}
