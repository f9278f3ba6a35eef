// Integer dequant-GEMM for prompts: more than 64 activation rows against tile-ordered int8 or int4 codes, sm_100a.
//
//   y[M, N] = x[M, K] . ((code[N, K] - zero[N]) * scale[N])^T      M > 64, fp16 x/y
//
// The arithmetic is that of qgemm_i8.cu (16-bit fixed-point activations split into two planes of signed bytes, exact int32
// sums, the same recombination), so the results are the same bits. What differs is the shape of the work: a pass of 64 rows is
// bound by streaming the weights, hundreds of rows are bound by the tensor cores and by what an SM can take in from L2.
//
// A pair of CTAs (cta_group::2) owns 256 weight rows x 128 activation rows: each CTA brings its 128 weight rows (16 KB per
// 128-column k block) and one of the two planes (128 rows, 16 KB), and one MMA of M 256, N 256 (128 high, 128 low columns)
// serves both. That is 32 KB per CTA and 512 tensor-core cycles; a CTA by itself would need 48 KB for the same cycles (both planes), more
// than L2 delivers. The accumulator takes 256 of the 512 tensor-memory columns, so the epilogue of one tile runs under the main
// loop of the next. Persistent: pairs walk the tiles with the row blocks innermost, so that the weights of the few tiles
// in flight are read from HBM once and the activation planes stay in L2. 2048 rows, int8 28672 x 4096 with SwiGLU: 297 us, 3.2 POPS
// (311 us and 80 % of the tensor cycles while a branch that one lane took issued the MMAs; 32 passes of 64 rows take 26 us each for half of these weights).
//
// Few tiles leave most SMs idle, so that a tile's K range is split over the SPLIT pairs of a larger cluster (one tile per
// cluster then): every CTA lays its partial sums for the other pairs' shares of the activation rows out in its drained ring, one bulk copy
// each brings them there, and a pair adds what has come to its own sums in tensor memory (read one by one through distributed shared
// memory they took 4000 cycles per 16 rows). Integer sums: the order cannot matter. 256 rows of 2048 x 5632: 44 k blocks on 32 SMs, or 22 on 64.
//
// Warps: 0 copies, 1 issues MMAs (even CTA only), 2-9 or 2-17 epilogue (four per group of activation rows), with int4 codes 10-21
// widen nibble tiles to byte tiles in three groups that take every third stage.
#include "common.cuh"
#include "qgemv_common.cuh"
#include "tc_ptx.cuh"
#include "i8_recombine.cuh"

namespace cb200 {
namespace {

using namespace ptx;

constexpr int kRows = 128;            // weight rows per CTA, activation rows per tile, bytes of k per stage
constexpr int kTile = kRows * kRows;  // 16 KB: a weight tile, or one plane of an activation tile
constexpr int kAccCols = 256;         // [128 high | 128 low]
constexpr int kPairHalf = 64;         // SwiGLU: 64 gate and 64 up rows per weight tile
constexpr int kChunk = 16;            // activation rows an epilogue thread handles at a time

__device__ int g_i8_rows_status = 0;

__host__ __device__ constexpr int stage_bytes(int bits) { return 2 * kTile + (bits == 4 ? kTile / 2 : 0); }
__host__ __device__ constexpr int num_stages(int bits) { return bits == 4 ? 5 : 6; }
constexpr int kConverterGroups = 3;     // one group needs 1770 cycles from barrier to barrier for a stage of 512 tensor-core cycles
__host__ __device__ constexpr int num_threads(int bits, int groups) { return 64 + groups * 128 + (bits == 4 ? kConverterGroups * 128 : 0); }
constexpr int kExchangeBytes = 4 * kChunk * kPairHalf * 4;
constexpr int kTailBytes = kExchangeBytes + 2 * kRows * 16 + 512;     // SwiGLU exchange, row scales and sums of two tiles, barriers

struct RowsParams {
  const void* scales;
  const float* zero_points;
  const __half* residual;
  __half* y;
  const float* sx;
  const int* qsum;
  const int* n_rows;
  const uint8_t* w_tiled;
  int M, N, K, n_out;
  int scale_f16;
  int bands;          // weight tiles of 128 rows
};

// G: groups of four epilogue warps, a share of the tile's activation rows each
template <int BITS, bool SWIGLU, int SPLIT, int G>
__global__ void __launch_bounds__(num_threads(BITS, G), 1)
qgemm_i8_rows_kernel(const __grid_constant__ CUtensorMap tmap_w, const __grid_constant__ CUtensorMap tmap_x, const RowsParams p) {
  chain_enter();
  constexpr int S = num_stages(BITS), kGroupRows = kRows / SPLIT / G;
  constexpr int kEpilogueThreads = 128 * G, kConverters = 2 + 4 * G;      // (first converter warp)
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~static_cast<uintptr_t>(1023));
  uint8_t* s_w = smem;                       // [S] byte tiles of this CTA's weight rows
  uint8_t* s_x = s_w + S * kTile;            // [S] this CTA's plane
  uint8_t* s_raw = s_x + S * kTile;          // [S] int4: nibble tiles
  float* s_up = reinterpret_cast<float*>(s_raw + (BITS == 4 ? S * kTile / 2 : 0));    // [group][4 / G][kChunk][64]
  int4* s_row = reinterpret_cast<int4*>(s_up + 4 * kChunk * kPairHalf);               // [2][128] (scale, sum >> 8, sum & 255, sum)
  uint64_t* full = reinterpret_cast<uint64_t*>(s_row + 2 * kRows);   // [S] (even CTA) operands of both CTAs have landed
  uint64_t* empty = full + S;                // [S] the MMAs that read the stage have retired
  uint64_t* raw_full = empty + S;            // [S] int4: this CTA's nibble tile has landed
  uint64_t* ready = raw_full + S;            // [S] int4 (even CTA): the byte tiles of both CTAs are written
  uint64_t* acc_full = ready + S;            // [2]
  uint64_t* acc_empty = acc_full + 2;        // [2] (even CTA) both CTAs' epilogues have read the accumulator
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(acc_empty + 2);
  uint64_t* xch = reinterpret_cast<uint64_t*>(tmem_slot + 2);      // SPLIT > 1: the other pairs' sums have landed
  // SPLIT > 1, over the drained ring: sums for the other pairs, then what they send, a slab [activation row][high, low][weight row] each
  constexpr int kShare = kRows / SPLIT, kSlab = kShare * 2 * kRows;
  int* s_out = reinterpret_cast<int*>(smem);
  int* s_in = s_out + (SPLIT - 1) * kSlab;

  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  const uint32_t cluster_rank = cluster_ctarank();
  const uint32_t rank = cluster_rank & 1, first = cluster_rank & ~1u;      // in the pair; the pair's even CTA
  const int share = static_cast<int>(cluster_rank >> 1);                   // of K, and of the tile's activation rows
  const int rows = p.n_rows ? min(p.M, *p.n_rows) : p.M;
  const int row_blocks = (rows + kRows - 1) / kRows;
  const int kblocks_all = p.K / kRows;
  const int kb0 = kblocks_all * share / SPLIT, kblocks = kblocks_all * (share + 1) / SPLIT - kb0;
  const int tiles = (p.bands + 1) / 2 * row_blocks;
  const int pairs = gridDim.x / (2 * SPLIT);
  const int pair = blockIdx.x / (2 * SPLIT);

  if (warp == 0 && lane == 0) {
    for (int s = 0; s < S; ++s) {
      mbar_init(smem_u32(&full[s]), 1);
      mbar_init(smem_u32(&empty[s]), 1);
      mbar_init(smem_u32(&raw_full[s]), 1);
      mbar_init(smem_u32(&ready[s]), 8);          // four converter warps of each CTA
    }
    for (int a = 0; a < 2; ++a) {
      mbar_init(smem_u32(&acc_full[a]), 1);
      mbar_init(smem_u32(&acc_empty[a]), 8 * G);     // the epilogue warps of both CTAs
    }
    if (SPLIT > 1) mbar_init(smem_u32(xch), 1);
    mbar_fence_init();
    if (SPLIT > 1) mbar_expect_tx(smem_u32(xch), (SPLIT - 1) * kSlab * 4);
  }
  if (warp == 1) tc_alloc_pair(smem_u32(tmem_slot), 2 * kAccCols);
  tc_fence_before();
  __syncthreads();
  cluster_sync_release();                         // both CTAs' barriers exist before either is signalled
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;

  if (warp == 0) {
    if (lane == 0) {
      // ---------------- copies ----------------
      int it = 0;
      bool ok = true;
      for (int t = pair; t < tiles && ok; t += pairs) {
        const int band = t / row_blocks * 2 + static_cast<int>(rank), block = t % row_blocks;
        for (int kb = 0; kb < kblocks; ++kb, ++it) {
          const int s = it % S;
          if (it >= S && !mbar_wait(smem_u32(&empty[s]), ((it / S) & 1) ^ 1, &g_i8_rows_status, (12 << 8) | 1)) { ok = false; break; }
          const uint32_t bar = map_to_rank(smem_u32(&full[s]), first);
          if (rank == 0) mbar_expect_tx(smem_u32(&full[s]), BITS == 8 ? 4 * kTile : 2 * kTile);
          // (a band beyond the last one, where their number is odd, reads as zero)
          if constexpr (BITS == 8) {
            tma_load_2d_pair(smem_u32(s_w + s * kTile), &tmap_w, bar, 0, (band * kblocks_all + kb0 + kb) * kRows);
          } else {
            const int b = min(band, p.bands - 1);
            mbar_expect_tx(smem_u32(&raw_full[s]), kTile / 2);
            bulk_load(smem_u32(s_raw + s * (kTile / 2)), p.w_tiled + (static_cast<size_t>(b) * kblocks_all + kb0 + kb) * (kTile / 2), kTile / 2,
                      smem_u32(&raw_full[s]));
          }
          tma_load_2d_pair(smem_u32(s_x + s * kTile), &tmap_x, bar, 0, ((block * kblocks_all + kb0 + kb) * 2 + static_cast<int>(rank)) * kRows);
        }
      }
      // Nothing may still be on its way when the blocks end: a wait elsewhere may have given up. (The even CTA sees the copies of both.)
      for (int i = it > S ? it - S : 0; i < it; ++i) {
        if (rank == 0 && !mbar_wait(smem_u32(&full[i % S]), (i / S) & 1, &g_i8_rows_status, (12 << 8) | 7)) break;
        if (BITS == 4 && !mbar_wait(smem_u32(&raw_full[i % S]), (i / S) & 1, &g_i8_rows_status, (12 << 8) | 8)) break;
      }
    }
  } else if (warp == 1) {
    if (rank == 0) {
      // ---------------- MMAs of the pair: the whole warp waits, one elected lane issues ----------------
      // D = s32, A (codes) unsigned 8 bit, B (activation bytes) signed 8 bit, both K-major, N = 256, M = 256
      constexpr uint32_t idesc = (2u << 4) | (0u << 7) | (1u << 10) | (static_cast<uint32_t>(kAccCols >> 3) << 17) | (static_cast<uint32_t>(256 >> 4) << 24);
      const uint64_t w_desc = smem_desc_sw128(smem_u32(s_w)), x_desc = smem_desc_sw128(smem_u32(s_x));    // (offsets add to the lowest bits, by 16 bytes)
      const bool leader = elect_one();
      int s = 0, n = 0;
      uint32_t phase = 0;
      bool ok = true;
      for (int t = pair; t < tiles && ok; t += pairs, ++n) {
        const int a = n & 1;
        if (n >= 2 && !__all_sync(0xffffffffu, mbar_wait(smem_u32(&acc_empty[a]), ((n >> 1) & 1) ^ 1, &g_i8_rows_status, (12 << 8) | 2))) break;
        tc_fence_after();
        const uint32_t d = tmem_base + a * kAccCols;
        for (int kb = 0; kb < kblocks; ++kb) {
          ok = mbar_wait(smem_u32(&full[s]), phase, &g_i8_rows_status, (12 << 8) | 3);
          if (BITS == 4) ok = ok && mbar_wait(smem_u32(&ready[s]), phase, &g_i8_rows_status, (12 << 8) | 4);
          ok = __all_sync(0xffffffffu, ok);
          if (!ok) break;
          tc_fence_after();
          if (leader) {
            const uint64_t wd = w_desc + s * (kTile / 16), xd = x_desc + s * (kTile / 16);
#pragma unroll
            for (int j = 0; j < 4; ++j) tc_mma_i8_ss_pair(d, wd + j * 2, xd + j * 2, idesc, (kb > 0 || j > 0) ? 1u : 0u);
            tc_commit_pair(smem_u32(&empty[s]), first);
          }
          __syncwarp();
          if (++s == S) { s = 0; phase ^= 1; }
        }
        if (leader) tc_commit_pair(smem_u32(&acc_full[a]), first);
        __syncwarp();
      }
    }
  } else if (warp < kConverters) {
    // ---------------- epilogue: lane quarter = warp % 4, a thread owns one weight row and kGroupRows of the activation rows ----------------
    // About ten instructions per output; a scheduler has G (two or four) of these warps, so the loops keep 16 independent outputs going.
    const int q = warp & 3;
    const int r = q * 32 + lane;
    const int group = (warp - 2) >> 2;
    const int tid = threadIdx.x - 64;
    const bool is_up = SWIGLU && r >= kPairHalf;
    int n = 0;
    bool ok = true;       // (a wait that gave up leaves the loops and their barriers as they are, without stores)
    for (int t = pair; t < tiles; t += pairs, ++n) {
      const int a = n & 1;
      const int band = t / row_blocks * 2 + static_cast<int>(rank), m0 = t % row_blocks * kRows;
      const int col = SWIGLU ? band * kPairHalf + (r & (kPairHalf - 1)) : band * kRows + r;      // output column
      bool col_ok = col < p.n_out;
      const int w_row = is_up ? p.N / 2 + col : col;
      if (tid < kRows) {                                   // (the arrays cover whole blocks of 128 rows)
        const int sum = p.qsum[m0 + tid];
        s_row[a * kRows + tid] = make_int4(__float_as_int(p.sx[m0 + tid]), sum >> 8, sum & 255, sum);
      }
      float scale = 0.f, zero = 128.f;
      if (col_ok) {
        scale = p.scale_f16 ? __half2float(static_cast<const __half*>(p.scales)[w_row]) : static_cast<const float*>(p.scales)[w_row];
        if (p.zero_points) zero = p.zero_points[w_row];
      }
      const bool zero_is_int = zero == rintf(zero) && fabsf(zero) <= 255.f;
      const int zero_int = zero_is_int ? __float2int_rn(zero) : 0;
      const bool all_int = __all_sync(0xffffffffu, zero_is_int);
      asm volatile("bar.sync 1, %0;" ::"n"(kEpilogueThreads) : "memory");
      ok = ok && mbar_wait(smem_u32(&acc_full[a]), (n >> 1) & 1, &g_i8_rows_status, (12 << 8) | 5);
      col_ok = col_ok && ok;
      __syncwarp();
      tc_fence_after();
      const uint32_t lanes = tmem_base + a * kAccCols + (static_cast<uint32_t>(q * 32) << 16);
      const int real = min(kRows, rows - m0);
      __half* y = p.y + static_cast<size_t>(m0) * p.n_out + col;
      const __half* res = p.residual ? p.residual + static_cast<size_t>(m0) * p.n_out + col : nullptr;
      if constexpr (SPLIT > 1) {       // sums of the other pairs' activation rows to them, one bulk copy each
#pragma unroll 1
        for (int e = 0; e < SPLIT - 1; ++e) {
          const int to = e < share ? e : e + 1;
#pragma unroll 1
          for (int c0 = group * kGroupRows; c0 < (group + 1) * kGroupRows; c0 += kChunk) {
            uint32_t hi[kChunk], lo[kChunk];
            tc_ld_x16(lanes + to * kShare + c0, hi);
            tc_ld_x16(lanes + kRows + to * kShare + c0, lo);
            tc_wait_ld();
#pragma unroll
            for (int j = 0; j < kChunk; ++j) {
              s_out[e * kSlab + (2 * (c0 + j)) * kRows + r] = kblocks > 0 ? static_cast<int>(hi[j]) : 0;
              s_out[e * kSlab + (2 * (c0 + j) + 1) * kRows + r] = kblocks > 0 ? static_cast<int>(lo[j]) : 0;
            }
          }
        }
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        __syncwarp();
        cluster_sync_release();        // every CTA's sums are in place and its ring is no longer read
        if (tid == 0)
          for (int e = 0; e < SPLIT - 1; ++e) {
            const int to = e < share ? e : e + 1, slot = share < to ? share : share - 1;
            bulk_copy_to_rank(smem_u32(s_in + slot * kSlab), smem_u32(s_out + e * kSlab), kSlab * 4, smem_u32(xch), 2 * to + rank);
          }
        // (also where an earlier wait gave up: the other pairs send all the same, and this block must not end before their sums have landed)
        ok = mbar_wait(smem_u32(xch), 0, &g_i8_rows_status, (12 << 8) | 10) && ok;
        col_ok = col_ok && ok;
        __syncwarp();
      }
#pragma unroll 1
      for (int c0 = 0; c0 < kGroupRows; c0 += kChunk) {
        const int first_row = (share * G + group) * kGroupRows + c0;          // activation row of the tile
        uint32_t hi[kChunk], lo[kChunk];
        tc_ld_x16(lanes + first_row, hi);
        tc_ld_x16(lanes + kRows + first_row, lo);
        float add[kChunk];
        if constexpr (!SWIGLU) {
#pragma unroll
          for (int j = 0; j < kChunk; ++j)
            add[j] = res && col_ok && first_row + j < real ? __half2float(res[static_cast<size_t>(first_row + j) * p.n_out]) : 0.f;
        }
        tc_wait_ld();
        if constexpr (SPLIT > 1) {
#pragma unroll
          for (int j = 0; j < kChunk; ++j) {
            if (kblocks == 0) { hi[j] = 0u; lo[j] = 0u; }
            const int* in = s_in + (2 * (group * kGroupRows + c0 + j)) * kRows + r;
#pragma unroll
            for (int k = 0; k < SPLIT - 1; ++k) {
              hi[j] += static_cast<uint32_t>(in[k * kSlab]);
              lo[j] += static_cast<uint32_t>(in[k * kSlab + kRows]);
            }
          }
        }
        if (SPLIT == 1 && c0 + kChunk >= kGroupRows) {       // the accumulator is in registers: the next tile may have it
          tc_fence_before();
          __syncwarp();
          if (lane == 0) mbar_arrive_cluster(map_to_rank(smem_u32(&acc_empty[a]), first));
        }
        const int4* row = s_row + a * kRows + first_row;
        float v[kChunk];
        if (all_int) {
#pragma unroll
          for (int j = 0; j < kChunk; ++j) {
            const int4 at = row[j];
            v[j] = fmaf(static_cast<float>(static_cast<int>(hi[j]) - zero_int * at.y), 256.f, static_cast<float>(static_cast<int>(lo[j]) - zero_int * at.z)) *
                   (scale * __int_as_float(at.x));
          }
        } else {
#pragma unroll 1
          for (int j = 0; j < kChunk; ++j) {                // (rolled, on registers picked by comparison: rare)
            int h = 0, l = 0;
#pragma unroll
            for (int i = 0; i < kChunk; ++i)
              if (i == j) { h = static_cast<int>(hi[i]); l = static_cast<int>(lo[i]); }
            const float f = recombine(h, l, zero, zero_int, zero_is_int, row[j].w) * (scale * __int_as_float(row[j].x));
#pragma unroll
            for (int i = 0; i < kChunk; ++i)
              if (i == j) v[i] = f;
          }
        }
        if constexpr (SWIGLU) {
          // gate and up of a column sit 64 lanes apart: the up side hands over the first half of the chunk and finishes
          // the second, the gate side the other way round
          constexpr int H = kChunk / 2;
          float* buf = s_up + (G == 4 ? group : group * 2 + ((c0 / kChunk) & 1)) * kChunk * kPairHalf + (r & (kPairHalf - 1));
#pragma unroll
          for (int j = 0; j < H; ++j) {
            if (is_up) buf[j * kPairHalf] = v[j];
            else buf[(H + j) * kPairHalf] = v[H + j];
          }
          asm volatile("bar.sync %0, 128;" ::"r"(2 + group) : "memory");
#pragma unroll
          for (int j = 0; j < H; ++j) {
            const float other = buf[(is_up ? H + j : j) * kPairHalf];
            const float g = is_up ? other : v[j], u = is_up ? v[H + j] : other;
            const int m = first_row + (is_up ? H + j : j);
            if (col_ok && m < real) y[static_cast<size_t>(m) * p.n_out] = __float2half_rn(silu_fast(g) * u);
          }
          if (G == 4) asm volatile("bar.sync %0, 128;" ::"r"(2 + group) : "memory");      // (one buffer: it has been read)
        } else {
#pragma unroll
          for (int j = 0; j < kChunk; ++j)
            if (col_ok && first_row + j < real) y[static_cast<size_t>(first_row + j) * p.n_out] = __float2half_rn(__fadd_rn(v[j], add[j]));
        }
      }
    }
  } else if constexpr (BITS == 4) {
    // ---------------- int4: nibble tile -> byte tile ----------------
    // Thread r owns tile row r: 64 bytes of nibbles (16-byte chunk c at c ^ ((r >> 1) & 3)) become 128 bytes of codes in the
    // 128-byte swizzle order (chunk c at c ^ (r & 7)); even columns sit in the low nibbles.
    const int r = threadIdx.x & 127;
    static_assert((kConverters * 32) % 128 == 64, "converter warps start at a multiple of two warps");
    const int steps = tiles > pair ? ((tiles - pair - 1) / pairs + 1) * kblocks : 0;
    bool ok = true;
    const int group = (warp - kConverters) >> 2;
    // A barrier's parity only tells neighbouring phases apart. A group therefore waits for its own stages alone, first until the MMAs
    // have retired that read the place before (the copy behind which this group's last stage came had waited for the use before that one), then
    // for the bytes. Neither barrier can move on without this group's conversion, so that no phase is missed, however late the group looks.
    static_assert(kConverterGroups < S, "a group's last stage was copied after the place's last one");
    for (int it = group; it < steps; it += kConverterGroups) {
      const int s = it % S;
      ok = __all_sync(0xffffffffu, (it < S || mbar_wait(smem_u32(&empty[s]), ((it / S) & 1) ^ 1, &g_i8_rows_status, (12 << 8) | 9)) &&
                                       mbar_wait(smem_u32(&raw_full[s]), (it / S) & 1, &g_i8_rows_status, (12 << 8) | 6));
      if (!ok) break;
      const uint8_t* raw_row = s_raw + s * (kTile / 2) + r * (kRows / 2);
      uint8_t* out_row = s_w + s * kTile + r * kRows;
      uint4 raw[4];
#pragma unroll
      for (int c = 0; c < 4; ++c) raw[c] = *reinterpret_cast<const uint4*>(raw_row + ((c ^ ((r >> 1) & 3)) * 16));
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        const uint32_t w[4] = {raw[c].x, raw[c].y, raw[c].z, raw[c].w};
        uint32_t o[8];
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const uint32_t even = w[j] & 0x0F0F0F0Fu;
          const uint32_t odd = (w[j] >> 4) & 0x0F0F0F0Fu;
          o[2 * j] = __byte_perm(even, odd, 0x5140);
          o[2 * j + 1] = __byte_perm(even, odd, 0x7362);
        }
        *reinterpret_cast<uint4*>(out_row + (((2 * c) ^ (r & 7)) * 16)) = make_uint4(o[0], o[1], o[2], o[3]);
        *reinterpret_cast<uint4*>(out_row + (((2 * c + 1) ^ (r & 7)) * 16)) = make_uint4(o[4], o[5], o[6], o[7]);
      }
      asm volatile("fence.proxy.async.shared::cta;" ::: "memory");   // the tensor core reads these bytes through the async proxy
      __syncwarp();
      if (lane == 0) mbar_arrive_cluster(map_to_rank(smem_u32(&ready[s]), first));
    }
  }
  if constexpr (SPLIT > 1) {                      // (the cluster barrier between the partial sums and their readers is everyone's)
    if ((warp < 2 || warp >= kConverters) && pair < tiles) {
      __syncwarp();
      cluster_sync_release();
    }
  }
  // Nobody leaves while the other CTA may still signal its barriers, read its operands or use the pair's tensor memory.
  __syncwarp();
  tc_fence_before();
  cluster_sync_release();
  if (warp == 1) {
    tc_fence_after();
    tc_dealloc_pair(tmem_base, 2 * kAccCols);
  }
}

template <int BITS, bool SWIGLU, int SPLIT, int G>
int launch_split(const CUtensorMap& tmap_w, const CUtensorMap& tmap_x, const RowsParams& p, int tiles, cudaStream_t stream) {
  constexpr int kSmem = 1024 + num_stages(BITS) * stage_bytes(BITS) + kTailBytes;
  static_assert((4 * num_stages(BITS) + 5) * 8 + 8 <= 512, "barriers and the tensor-memory base fit in the tail");
  static_assert(num_stages(BITS) * stage_bytes(BITS) >= 2 * (SPLIT - 1) * (kRows / SPLIT) * 2 * kRows * 4, "sums that leave and come fit in the drained ring");
  auto kern = qgemm_i8_rows_kernel<BITS, SWIGLU, SPLIT, G>;
  cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmem);
  if (e != cudaSuccess) return static_cast<int>(e);
  const int clusters = SPLIT > 1 || tiles < kNumSMs / 2 ? tiles : kNumSMs / 2;
  e = launch_clusters(kern, dim3(2 * SPLIT * clusters, 1, 1), num_threads(BITS, G), kSmem, stream, dim3(2 * SPLIT, 1, 1), tmap_w, tmap_x, p);
  if (e != cudaSuccess) return static_cast<int>(e);
  return launch_status();
}

// (Times from before partial sums travelled in bulk, which takes 10 to 15 % off the split forms.)
// Pairs along K, with at least four k blocks each: four for up to twelve tiles (sixteen clusters of eight CTAs do not run at
// once: 100 rows of int8 4096 x 4096 30.0 us with four, 19.5 with two, 23.5 with one; 1280 x 8192 19.6, 32.7 with one), two
// for up to 33 (4096 x 14336 43.6 us with four, 32.6 with two, 47.5 with one; so many clusters of four CTAs run at once: 37 tiles
// in two pairs each take two turns, 65 rows of int4 9344 x 4096 53.5 us, 9728 x 4096 in one pair each 36.5).
int pairs_along_k(int tiles, int kblocks) {
  if (tiles <= 12 && kblocks >= 16) return 4;
  return tiles <= 33 && kblocks >= 8 ? 2 : 1;
}

template <int BITS, bool SWIGLU>
int launch_rows(const CUtensorMap& tmap_w, const CUtensorMap& tmap_x, const RowsParams& p, cudaStream_t stream) {
  const int tiles = (p.bands + 1) / 2 * ((p.M + kRows - 1) / kRows);
  const int split = pairs_along_k(tiles, p.K / kRows);
  // With a split K an epilogue covers nothing, and it is latency: twice the warps and one bulk copy per pair instead of reads from its shared
  // memory take 10 to 15 % off (256 rows of int8 2048x2048 13.0 / 11.3 us, 4096x2048 13.7 / 11.9, 4096x4096 16.4 / 14.6). Where pairs have
  // whole tiles more warps get in the way (384 rows of 4096x14336 47.2 / 49.3), except with SwiGLU and at most two tiles (11264x2048
  // 2 us less). With int4 codes the converters have the registers; four pairs along K leave each 32 activation rows.
  if (split == 4) return launch_split<BITS, SWIGLU, 4, 2>(tmap_w, tmap_x, p, tiles, stream);
  if (split == 2) return launch_split<BITS, SWIGLU, 2, BITS == 8 ? 4 : 2>(tmap_w, tmap_x, p, tiles, stream);
  if constexpr (BITS == 8 && SWIGLU)
    if (tiles <= kNumSMs) return launch_split<BITS, SWIGLU, 1, 4>(tmap_w, tmap_x, p, tiles, stream);
  return launch_split<BITS, SWIGLU, 1, 2>(tmap_w, tmap_x, p, tiles, stream);
}

}  // namespace

// Tile-ordered per-row codes, fp16 activations, more than 64 rows; the 64-row kernel takes what is left.
bool qgemm_i8_rows_supported(const QGemvParams& q, const void* workspace, size_t workspace_bytes) {
  if (q.x_dtype != CACHEIR_B200_F16 || (q.bits != 8 && q.bits != 4) || q.group_size != 0 || !q.tiled || q.norm_weight) return false;
  if (q.M <= 64 || q.K % kRows != 0 || q.K < kRows || q.K > 32768) return false;
  const bool swiglu = q.epilogue == CACHEIR_B200_EPI_SWIGLU;
  if (q.epilogue != CACHEIR_B200_EPI_NONE && q.epilogue != CACHEIR_B200_EPI_RESIDUAL && !swiglu) return false;
  if (swiglu != q.paired || (swiglu && (q.N / 2) % kPairHalf != 0)) return false;
  if (!workspace || workspace_bytes < qgemm_i8_workspace_bytes(q.M, q.K) || !aligned_to(workspace, 128)) return false;
  if (!aligned_to(q.packed, 16) || !aligned_to(q.x, 16) || (q.x_stride * 2) % 16 != 0) return false;
  return tensor_map_encoder() != nullptr;
}

// Against passes of 64 rows. A pair needs about 1 us for a k block of int4 codes, so that up to 128 rows with a long K and less
// than half of the pairs at work are faster as two passes over all SMs: 100 rows of 4096 x 14336 56.5 us here, 54.6 in passes
// (49 for up to 96 rows); 4096 x 4096 29.6 and 36.7, 1280 x 8192 27.4 and 29.8, 14336 x 4096 38 and 61. Bytes: 20 to 45 % faster here.
// Up to 80 rows the second pass is a short one, and passes win from half as many k blocks on (65 rows of 1280 x 8192 27.7 and 25.1,
// 4096 x 4096 28.9 and 27.5), unless their own clusters along K need two turns (2048 x 8192 27.9 and 35.6).
bool qgemm_i8_rows_preferred(const QGemvParams& q) {
  if (q.bits == 8 || q.M > kRows) return true;
  const int tiles = (q.N + 2 * kRows - 1) / (2 * kRows), kblocks = q.K / kRows, split = pairs_along_k(tiles, kblocks);
  if (tiles * split * 4 > kNumSMs) return true;
  QGemvParams pass = q;
  pass.M = 64;
  const int bands = (q.N + kRows - 1) / kRows, along = qgemm_i8_plan(pass);
  if (along * bands > (along == 8 ? 8 * 14 : along == 4 ? 4 * 32 : kNumSMs)) return true;
  return q.M <= 80 ? kblocks < 8 * split || kblocks < 32 : kblocks <= 16 * split;
}

int launch_qgemm_i8_rows(const QGemvParams& q, const int* n_rows, void* workspace, cudaStream_t stream) {
  const TallPlanes planes = tall_planes(workspace, q.M, q.K);
  if (!q.x_prequantized) {
    const int rc = qgemm_i8_quantize_tall(q.x, q.x_stride, q.M, n_rows, q.K, workspace, stream);
    if (rc != 0) return rc;
  }
  const bool swiglu = q.epilogue == CACHEIR_B200_EPI_SWIGLU;
  RowsParams p{};
  p.scales = q.scales; p.zero_points = q.zero_points;
  p.residual = q.epilogue == CACHEIR_B200_EPI_RESIDUAL ? static_cast<const __half*>(q.residual) : nullptr;
  p.y = static_cast<__half*>(q.y);
  p.sx = planes.sx; p.qsum = planes.qsum; p.n_rows = n_rows;
  p.w_tiled = static_cast<const uint8_t*>(q.packed);
  p.M = q.M; p.N = q.N; p.K = q.K;
  p.n_out = swiglu ? q.N / 2 : q.N;
  p.scale_f16 = q.scale_dtype == CACHEIR_B200_F16 ? 1 : 0;
  p.bands = swiglu ? (p.n_out + kPairHalf - 1) / kPairHalf : (p.n_out + kRows - 1) / kRows;
  const uint64_t kblocks = static_cast<uint64_t>(q.K / kRows), blocks = static_cast<uint64_t>((q.M + kRows - 1) / kRows);
  CUtensorMap tmap_w, tmap_x;
  // (nibble tiles travel by plain bulk copies: their map is only a valid placeholder)
  if (!encode_u8_tiles_plain(&tmap_w, q.packed, static_cast<uint64_t>(p.bands) * kblocks * (q.bits == 4 ? kRows / 2 : kRows)) ||
      !encode_u8_tiles_plain(&tmap_x, planes.planes, blocks * kblocks * 2 * kRows))
    return CACHEIR_B200_EUNSUPPORTED;
  if (q.bits == 4) return swiglu ? launch_rows<4, true>(tmap_w, tmap_x, p, stream) : launch_rows<4, false>(tmap_w, tmap_x, p, stream);
  return swiglu ? launch_rows<8, true>(tmap_w, tmap_x, p, stream) : launch_rows<8, false>(tmap_w, tmap_x, p, stream);
}

int qgemm_i8_rows_device_status(bool reset) {
  int status = 0;
  if (cudaMemcpyFromSymbol(&status, g_i8_rows_status, sizeof(int)) != cudaSuccess) return -1;
  if (reset && status != 0) {
    const int zero = 0;
    cudaMemcpyToSymbol(g_i8_rows_status, &zero, sizeof(int));
  }
  return status;
}

}  // namespace cb200
