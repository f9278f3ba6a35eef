// Streaming dequant-GEMM for up to 32 activation rows, sm_100a: weights from HBM to registers once, warp MMAs.
//
//   y[M, N] = x[M, K] . deq(W)[N, K]^T        fp16 x/y, int4 codes (per row affine or group-wise symmetric)
//
// Why not tcgen05 here: its weight operand comes through shared memory at about 37 bytes per clock and SM whatever the number
// of activation rows, after int4 codes have been inflated to 16 (bytes) or 32 KB (fp16) per 128 x 128 tile that takes 440 or 880
// cycles, where HBM delivers the tile's 8 KB in 350 (bytes would need their sums scaled per k block to serve group scales). mma.sync takes the weights from registers, where a few byte permutes
// turn codes into exact fp16 integers (code - zero), so nothing is written back to shared memory; its price, 64 MMAs per eight activation rows
// and tile of 4 cycles each, is 256 to 1024 cycles. No activation pre-pass.
//
// A CTA has 32 * RG weight rows; its warps are RG row groups x KG k groups. A warp owns two 16-row MMA tiles and every KG-th k
// block of 128 columns (one 16-byte piece per row and lane). Each lane copies the pieces it will use itself
// into a private ring (cp.async, S stages deep, no barrier), the row groups of a k group share the activations of the block
// through a second ring (one named barrier per block). The MMA's k order is the memory order of a lane's piece: its operand registers hold
// the columns 32t .. 32t+31 of lane group t, and the activations are read with the same columns. Group scales multiply
// a block's sums in fp32. The k groups' sums meet in shared memory and are added in order: deterministic.
#include "common.cuh"
#include "qgemv_common.cuh"
#include "tc_ptx.cuh"

namespace cb200 {
namespace {

constexpr int kU = 2;                   // MMA tiles (16 rows) per warp
constexpr int kCols = 128;              // columns of a k block
constexpr int kXRow = 2 * kCols;        // bytes of an activation row in it
constexpr int kSmemLimit = 192 * 1024;  // rings; group scales come on top
constexpr int kScaleLimit = 34 * 1024;
constexpr int kAhead = 32;              // k blocks a CTA asks for before its turn

struct StreamParams {
  const __half* x;
  const uint8_t* packed;
  const void* scales;
  const float* zero_points;
  const __half* residual;
  __half* y;
  int M, N, K, n_out;
  long long x_stride;
  int scale_f16, groups, kb_per_group;   // groups per row; k blocks of 128 per group
  int tiled, paired, residual_on;
  int per_band;                          // CTAs per 128-row band (64 or 128 output columns of it with SwiGLU)
  int split;                             // CTAs of a cluster along K
};

__host__ __device__ constexpr int k_groups(int rg) { return rg == 4 ? 4 : 8; }
// bytes of a k block in the rings of one k group: the warps' pieces, and `m` activation rows
__host__ __device__ constexpr int stage_bytes(int m, int rg) { return rg * kU * 2 * 512 + m * kXRow; }
__host__ __device__ constexpr int stages(int nt, int rg) {
  const int s = kSmemLimit / (k_groups(rg) * stage_bytes(8 * nt, rg));
  return s > 4 ? 4 : s;
}
__host__ __device__ constexpr int sum_bytes(int m, int rg) { return k_groups(rg) * m * (32 * rg + 4) * 4; }
__host__ __device__ constexpr int total_bytes(int m, int rg) { return m * (32 * rg + 4) * 4; }
__host__ __device__ constexpr int area_bytes(int nt, int m, int rg) {
  const int ring = k_groups(rg) * stages(nt, rg) * stage_bytes(m, rg), sums = sum_bytes(m, rg) + total_bytes(m, rg);
  return ((ring > sums ? ring : sums) + 127) / 128 * 128;
}
__device__ __forceinline__ float load_from_rank(const float* local, uint32_t rank) {
  float v;
  asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v) : "r"(ptx::map_to_rank(ptx::smem_u32(local), rank)) : "memory");
  return v;
}

__device__ __forceinline__ void copy16(uint32_t dst, const void* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory");
}
__device__ __forceinline__ void mma(float (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
               : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3]) : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
__device__ __forceinline__ __half2 as_half2(uint32_t v) { return *reinterpret_cast<__half2*>(&v); }
__device__ __forceinline__ uint32_t as_bits(__half2 v) { return *reinterpret_cast<uint32_t*>(&v); }
// byte j of w: its two nibbles as (low - zero, high - zero). (0x6400 | n, 0x6400 | n << 4) = (1024 + n, 1024 + 16 n); one exact fma
__device__ __forceinline__ uint32_t nibble_pair(uint32_t w, int j, __half2 sub) {
  const uint32_t t = __byte_perm(w, 0x64646464u, 0x4040 + 0x101 * j) & 0x64F0640Fu;
  return as_bits(__hfma2(as_half2(t), __floats2half2_rn(1.f, 0.0625f), sub));
}

template <int NT, int RG, bool GROUPED, bool SWIGLU>
__global__ void __launch_bounds__(32 * RG * k_groups(RG), RG == 1 ? 2 : 1)
qgemv_stream_kernel(const StreamParams p) {
  constexpr int KG = k_groups(RG), S = stages(NT, RG);
  constexpr int kThreads = 32 * RG * KG;
  constexpr int kRows = 32 * RG;                     // weight rows of the CTA
  const int kStage = stage_bytes(p.M, RG);
  static_assert(S >= 2, "the ring needs two stages");
  extern __shared__ __align__(128) uint8_t smem[];
  __half* s_scale = reinterpret_cast<__half*>(smem + area_bytes(NT, p.M, RG));     // [k block of 128][kRows], group-wise fp16 or fp32
  float* s_scale32 = reinterpret_cast<float*>(s_scale);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
  const int rg = warp % RG, kg = warp / RG;
  const int band = blockIdx.x / p.per_band, part = blockIdx.x % p.per_band;

  // MMA tile j of the CTA (0 .. 2 RG - 1) -> its first weight row. SwiGLU: the first RG tiles are gate rows, the others the up
  // rows of the same columns (64 rows further in a paired band, N / 2 rows further otherwise).
  auto tile_row = [&](int j) {
    if (!SWIGLU) return band * 128 + part * kRows + 16 * j;
    const int first = band * 128 + part * 16 * RG + 16 * (j % RG);
    return j < RG ? first : first + (p.paired ? 64 : p.N / 2);
  };
  // scale and zero point index of a weight row as it lies in memory (paired bands interleave the halves by 64 rows)
  auto param_row = [&](int row) {
    if (!SWIGLU || !p.paired) return row;
    return (row >> 7) * 64 + (row & 63) + ((row & 64) ? p.N / 2 : 0);
  };

  const uint8_t* rows[kU][2];
  const long long block_step = p.tiled ? 128 * 64 : 64;              // bytes to the next k block
  const int rank = p.split > 1 ? static_cast<int>(ptx::cluster_ctarank()) : 0;
  const int kblocks_all = p.K / kCols;
  const int kb0 = kblocks_all * rank / p.split, kblocks = kblocks_all * (rank + 1) / p.split;      // this CTA's: kb0 .. kblocks - 1
#pragma unroll
  for (int u = 0; u < kU; ++u)
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const int row = tile_row(rg * kU + u) + g + 8 * h;
      if (p.tiled) rows[u][h] = p.packed + (static_cast<size_t>(row >> 7) * (p.K / 128) * 128 + (row & 127)) * 64 + 16 * (t ^ ((g >> 1) & 3));   // (chunks in swizzled order)
      else rows[u][h] = p.packed + static_cast<size_t>(min(row, p.N - 1)) * (p.K / 2) + 16 * t;
    }

  const uint32_t ring = static_cast<uint32_t>(__cvta_generic_to_shared(smem)) + kg * S * kStage;
  const int group_thread = rg * 32 + lane;
  auto load = [&](int j) {                              // k block kg + j * KG of the warp's group
    const int kb = kb0 + kg + j * KG;
    if (kb < kblocks) {
      const uint32_t stage = ring + (j % S) * kStage;
      const long long off = kb * block_step;
#pragma unroll
      for (int u = 0; u < kU; ++u)
#pragma unroll
        for (int h = 0; h < 2; ++h) copy16(stage + ((rg * kU + u) * 2 + h) * 512 + lane * 16, rows[u][h] + off);
      // activations: piece c of 16 bytes of row m goes where its reader finds it without bank conflicts
#pragma unroll
      for (int i = 0; i < (NT * 8 * (kXRow / 16) + 32 * RG - 1) / (32 * RG); ++i) {
        const int piece = group_thread + i * 32 * RG;
        if (piece >= p.M * (kXRow / 16)) break;
        const int m = piece / (kXRow / 16), c = piece % (kXRow / 16);
        const int q = c / (kXRow / 64), sub = c % (kXRow / 64);         // reader t = q, its piece number
        const int slot = (sub * 4 + q) ^ ((m & 1) << 2);
        copy16(stage + RG * kU * 2 * 512 + m * kXRow + slot * 16, p.x + static_cast<size_t>(m) * p.x_stride + kb * kCols + c * 8);
      }
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  // The weights set out for L2 while the kernel before this one is at work: in tile order 1 KB per MMA tile and k block, in
  // row order a run of each row.
  if (p.tiled) {
    const int items = 2 * RG * min(kblocks - kb0, kAhead);
    for (int i = threadIdx.x; i < items; i += kThreads) {
      const int row = tile_row(i % (2 * RG));
      if (row < p.N) ptx::bulk_prefetch(p.packed + ((static_cast<size_t>(row >> 7) * kblocks_all + kb0 + i / (2 * RG)) * 128 + (row & 127)) * 64, 16 * 64);
    }
  } else {
    for (int i = threadIdx.x; i < kRows; i += kThreads) {
      const int row = tile_row(i >> 4) + (i & 15);
      if (row < p.N) ptx::bulk_prefetch(p.packed + static_cast<size_t>(row) * (p.K / 2) + kb0 * 64, 64 * min(kblocks - kb0, kAhead));
    }
  }
  chain_enter();
  for (int j = 0; j < S - 1; ++j) load(j);

  // per-row constants: scale (per row formats) and the zero point as an exact fp16 offset
  __half2 sub[kU][2];
  bool odd_zero = false;                               // a zero point that is no small integer: corrected at the end
#pragma unroll
  for (int u = 0; u < kU; ++u)
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const int row = tile_row(rg * kU + u) + g + 8 * h;
      float zero = 8.f;
      if (!GROUPED && p.zero_points && row < p.N) zero = p.zero_points[param_row(row)];
      const bool exact = zero == rintf(zero) && fabsf(zero) <= 960.f;
      odd_zero = odd_zero || !exact;
      const float z = exact ? zero : 0.f;
      sub[u][h] = __floats2half2_rn(-(1024.f + z), -(64.f + z));
    }
  if constexpr (GROUPED) {
    const int blocks128 = kblocks - kb0;
    for (int i = threadIdx.x; i < kRows * blocks128; i += kThreads) {
      const int local = i / blocks128, kb = i % blocks128;
      const int row = min(tile_row(local >> 4) + (local & 15), p.N - 1);
      const size_t at = static_cast<size_t>(row) * p.groups + (kb0 + kb) / p.kb_per_group;
      if (p.scale_f16) s_scale[kb * kRows + local] = static_cast<const __half*>(p.scales)[at];
      else s_scale32[kb * kRows + local] = static_cast<const float*>(p.scales)[at];
    }
    __syncthreads();
  }

  float acc[kU][NT][4];
#pragma unroll
  for (int u = 0; u < kU; ++u)
#pragma unroll
    for (int n = 0; n < NT; ++n) acc[u][n][0] = acc[u][n][1] = acc[u][n][2] = acc[u][n][3] = 0.f;

  const int turns = (kblocks - kb0 - kg + KG - 1) / KG;      // (a k group without blocks has none)
  for (int j = 0; j < turns; ++j) {
    asm volatile("cp.async.wait_group %0;" ::"n"(S - 2) : "memory");
    if constexpr (RG > 1) asm volatile("bar.sync %0, %1;" ::"r"(1 + kg), "n"(32 * RG) : "memory");
    else __syncwarp();
    load(j + S - 1);                                   // into the stage that everyone has left behind
    const uint8_t* stage = smem + kg * S * kStage + (j % S) * kStage;
    const uint8_t* s_x = stage + RG * kU * 2 * 512;
    uint4 raw[kU][2];
#pragma unroll
    for (int u = 0; u < kU; ++u)
#pragma unroll
      for (int h = 0; h < 2; ++h) raw[u][h] = *reinterpret_cast<const uint4*>(stage + ((rg * kU + u) * 2 + h) * 512 + lane * 16);
    float part_sum[kU][NT][4];
    if constexpr (GROUPED) {
#pragma unroll
      for (int u = 0; u < kU; ++u)
#pragma unroll
        for (int n = 0; n < NT; ++n) part_sum[u][n][0] = part_sum[u][n][1] = part_sum[u][n][2] = part_sum[u][n][3] = 0.f;
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) {                      // 32-bit word of the pieces: 8 columns
      uint4 xv[NT];
#pragma unroll
      for (int n = 0; n < NT; ++n)
        xv[n] = n * 8 + g < p.M ? *reinterpret_cast<const uint4*>(s_x + (n * 8 + g) * kXRow + (((i * 4 + t) ^ ((g & 1) << 2)) * 16)) : make_uint4(0u, 0u, 0u, 0u);
#pragma unroll
      for (int step = 0; step < 2; ++step) {
#pragma unroll
        for (int u = 0; u < kU; ++u) {
          const uint32_t w0 = i == 0 ? raw[u][0].x : i == 1 ? raw[u][0].y : i == 2 ? raw[u][0].z : raw[u][0].w;
          const uint32_t w1 = i == 0 ? raw[u][1].x : i == 1 ? raw[u][1].y : i == 2 ? raw[u][1].z : raw[u][1].w;
          const uint32_t a[4] = {nibble_pair(w0, 2 * step, sub[u][0]), nibble_pair(w1, 2 * step, sub[u][1]),
                                 nibble_pair(w0, 2 * step + 1, sub[u][0]), nibble_pair(w1, 2 * step + 1, sub[u][1])};
#pragma unroll
          for (int n = 0; n < NT; ++n) mma(GROUPED ? part_sum[u][n] : acc[u][n], a, step ? xv[n].z : xv[n].x, step ? xv[n].w : xv[n].y);
        }
      }
    }
    if constexpr (GROUPED) {
      const int kb = kg + j * KG;
#pragma unroll
      for (int u = 0; u < kU; ++u) {
        const int at = kb * kRows + (rg * kU + u) * 16 + g;
        const float s0 = p.scale_f16 ? __half2float(s_scale[at]) : s_scale32[at];
        const float s1 = p.scale_f16 ? __half2float(s_scale[at + 8]) : s_scale32[at + 8];
#pragma unroll
        for (int n = 0; n < NT; ++n) {
          acc[u][n][0] = fmaf(part_sum[u][n][0], s0, acc[u][n][0]); acc[u][n][1] = fmaf(part_sum[u][n][1], s0, acc[u][n][1]);
          acc[u][n][2] = fmaf(part_sum[u][n][2], s1, acc[u][n][2]); acc[u][n][3] = fmaf(part_sum[u][n][3], s1, acc[u][n][3]);
        }
      }
    }
  }
  asm volatile("cp.async.wait_all;" ::: "memory");

  // ---- the k groups' sums meet: [k group][activation row][weight row], padded so that the stores hit all banks ----
  const bool correct = __syncthreads_or(odd_zero) != 0;
  float* sums = reinterpret_cast<float*>(smem);
  constexpr int kPitch = kRows + 4;
#pragma unroll
  for (int u = 0; u < kU; ++u)
#pragma unroll
    for (int n = 0; n < NT; ++n)
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const int m = n * 8 + 2 * t + (e & 1);
        if (m < p.M) sums[(kg * p.M + m) * kPitch + (rg * kU + u) * 16 + g + 8 * (e >> 1)] = acc[u][n][e];
      }
  __shared__ float s_xsum[NT * 8];
  if (correct) {                                       // sums of x, for the rows whose zero point has not been subtracted (rare)
    for (int m = warp; m < p.M; m += kThreads / 32) {
      float v = 0.f;
      for (int k = lane; k < p.K; k += 32) v += __half2float(p.x[static_cast<size_t>(m) * p.x_stride + k]);
      v = warp_sum(v);
      if (lane == 0) s_xsum[m] = v;
    }
  }
  __syncthreads();
  // with a split the CTAs of the cluster add their sums up first and share the outputs between them, in rank order
  float* mine = reinterpret_cast<float*>(smem + sum_bytes(p.M, RG));
  if (p.split > 1) {
    for (int i = threadIdx.x; i < kRows * p.M; i += kThreads) {
      const int local = i % kRows, m = i / kRows;
      float v = 0.f;
#pragma unroll
      for (int k = 0; k < KG; ++k) v += sums[(k * p.M + m) * kPitch + local];
      mine[m * kPitch + local] = v;
    }
    ptx::cluster_sync_release();
  }
  auto total = [&](int local, int m) {                 // finished product of a weight row of this CTA with activation row m
    float v = 0.f;
    if (p.split > 1) {
      for (int k = 0; k < p.split; ++k) v += load_from_rank(mine + m * kPitch + local, k);
    } else {
#pragma unroll
      for (int k = 0; k < KG; ++k) v += sums[(k * p.M + m) * kPitch + local];
    }
    if constexpr (!GROUPED) {
      const int row = param_row(tile_row(local >> 4) + (local & 15));
      if (row >= p.N) return 0.f;
      if (correct) {
        const float zero = p.zero_points ? p.zero_points[row] : 8.f;
        if (!(zero == rintf(zero) && fabsf(zero) <= 960.f)) v -= zero * s_xsum[m];
      }
      v *= p.scale_f16 ? __half2float(static_cast<const __half*>(p.scales)[row]) : static_cast<const float*>(p.scales)[row];
    }
    return v;
  };
  constexpr int kOut = SWIGLU ? kRows / 2 : kRows;
  const int col0 = SWIGLU ? band * (p.paired ? 64 : 128) + part * kOut : band * 128 + part * kOut;
  for (int i = rank * kThreads + threadIdx.x; i < kOut * p.M; i += p.split * kThreads) {
    const int local = i % kOut, m = i / kOut, col = col0 + local;
    if (col >= p.n_out) continue;
    float v = total(local, m);
    if constexpr (SWIGLU) v = silu_fast(v) * total(kOut + local, m);
    const size_t o = static_cast<size_t>(m) * p.n_out + col;
    if (p.residual_on) v = __fadd_rn(v, __half2float(p.residual[o]));
    p.y[o] = __float2half_rn(v);
  }
  if (p.split > 1) ptx::cluster_sync_release();        // nobody's sums are read any more
}

template <int NT, int RG, bool GROUPED, bool SWIGLU>
int launch(const StreamParams& p, int ctas, cudaStream_t stream) {
  const int smem = area_bytes(NT, p.M, RG) + (GROUPED ? (p.K / 128 + p.split - 1) / p.split * 32 * RG * (p.scale_f16 ? 2 : 4) : 0);
  auto kern = qgemv_stream_kernel<NT, RG, GROUPED, SWIGLU>;
  cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
  if (e != cudaSuccess) return static_cast<int>(e);
  e = launch_clusters(kern, dim3(ctas, p.split, 1), 32 * RG * k_groups(RG), smem, stream, dim3(1, p.split, 1), p);
  if (e != cudaSuccess) return static_cast<int>(e);
  return launch_status();
}

template <int NT, int RG, bool GROUPED>
int launch_epilogue(StreamParams p, bool swiglu, cudaStream_t stream) {
  if (swiglu) {
    const int span = p.paired ? 64 : 128;              // output columns of a band
    p.per_band = span / (16 * RG);
    return launch<NT, RG, GROUPED, true>(p, (p.n_out + span - 1) / span * p.per_band, stream);
  }
  p.per_band = 4 / RG;
  return launch<NT, RG, GROUPED, false>(p, (p.n_out + 127) / 128 * p.per_band, stream);
}

struct Split { int rg, split; };
// Row groups per CTA and CTAs along K: what the busiest SM has to take in, its weights and the activations that come with every
// CTA, plus the exchange of a split and the start of every further wave. A cluster lives in one GPC, so that fewer of them run at
// once than the SMs would hold: 33 of four CTAs and 15 of eight (sixteen take two turns: 2048 x 8192, 1 row, 13.2 us with eight
// CTAs along K, 8.0 with four of half the rows). Four k blocks per CTA are enough to split (4096 x 2048, 32 rows: 12.5 us in one CTA
// along K, 9.6 in four). Over 740 products of 512 to 28672 rows and 512 to 14336 columns the choice is 1.1 % behind the best
// one, 17 % at most.
Split choose_split(int weight_rows, int K, int m) {
  constexpr struct { int split, at_once; } kForms[] = {{1, kNumSMs}, {2, kNumSMs / 2}, {3, 44}, {4, 32}, {6, 20}, {8, 14}};
  Split best{4, 1};
  long long best_cost = -1;
  for (int rg = 4; rg >= 1; rg /= 2)
    for (const auto form : kForms) {
      if (form.split > 1 && K / kCols / form.split < 4) break;
      const int per_sm = rg == 1 ? 2 : 1;
      const long long clusters = (weight_rows + 32 * rg - 1) / (32 * rg);
      const long long waves = (clusters + form.at_once * per_sm - 1) / (form.at_once * per_sm);
      const long long sharing = per_sm == 2 && clusters * form.split > kNumSMs ? 2 : 1;       // CTAs of an SM share its bandwidth
      const long long bytes = sharing * (K / form.split) * (32 * rg + 5 * m) / 2;
      const long long cost = waves * bytes + (waves - 1) * 96 * 1024 + (form.split > 1 ? 24 * 1024 : 0);
      if (best_cost < 0 || cost < best_cost) { best = {rg, form.split}; best_cost = cost; }
    }
  return best;
}

template <int NT, bool GROUPED>
int launch_rg(StreamParams p, bool swiglu, cudaStream_t stream) {
  const Split s = choose_split(p.N, p.K, p.M);
  p.split = s.split;
  switch (s.rg) {
    case 4: return launch_epilogue<NT, 4, GROUPED>(p, swiglu, stream);
    case 2: return launch_epilogue<NT, 2, GROUPED>(p, swiglu, stream);
    default: return launch_epilogue<NT, 1, GROUPED>(p, swiglu, stream);
  }
}

template <bool GROUPED>
int launch_nt(const StreamParams& p, bool swiglu, cudaStream_t stream) {
  if constexpr (GROUPED) {
    if (p.M > 16) return launch_rg<4, GROUPED>(p, swiglu, stream);
    if (p.M > 8) return launch_rg<2, GROUPED>(p, swiglu, stream);
  }
  return launch_rg<1, GROUPED>(p, swiglu, stream);
}

}  // namespace

// Where it takes over (us, with the pre-pass where there is one; weights N x K):
//   group-wise int4, up to 32 rows, against the fp16 tcgen05 kernel: 14336x4096 1 row 16 / 32, 16 rows 22 / 33, 32 rows 30 / 33;
//     1280x8192 6.7 / 19, 8.7 / 19, 11.6 / 21; 2048x2048 4.5 / 8.7, 7.6 / 8.7, 10.5 / 10.1
//   per-row int4, up to 8 rows, against the integer kernel: 1 row 14336x4096 13.6 / 17.0, 4096x4096 7.7 / 10.2, 2048x2048 4.3 / 8.1;
//     at 16 rows 19.9 / 17.7, so no further
// Codes in row order: the streaming int4 GEMV keeps the weights that fill all SMs with 64-row shares (14336x4096, 1 row: 17 / 15). On
// smaller ones it is up to a tenth faster for group-wise codes of K <= 4096 in 5632 to 8192 rows (5632x2048, 1 row: 7.1 / 6.4), slower on the
// others (4096x14336, 8 rows: 18.6 / 27.8), and its sums, which the constant 1024 of its operands leaves at the end, are a little less exact.
// Per-row codes in tile order: more bands than SMs leave the second turn half empty, the integer kernel keeps them (28672x4096, 8 rows:
// 27.4 / 24.1, the pre-pass included).
bool qgemv_stream_supported(const QGemvParams& q) {
  if (q.x_dtype != CACHEIR_B200_F16 || q.x_prequantized || q.norm_weight) return false;
  if (q.M < 1 || q.M > (q.group_size > 0 ? 32 : 8) || q.K % 128 != 0 || q.K < 128) return false;
  if (q.bits != 4 || q.group_size % 128 != 0) return false;
  if (q.group_size > 0 && q.K / 128 * 128 * (q.scale_dtype == CACHEIR_B200_F16 ? 2 : 4) > kScaleLimit) return false;   // of 128 rows
  if (!q.tiled && q.N >= 64 * kNumSMs && qgemv_mma_supported(q)) return false;
  if (q.tiled && q.group_size == 0 && q.N > 128 * kNumSMs) return false;
  const bool swiglu = q.epilogue == CACHEIR_B200_EPI_SWIGLU;
  if (q.epilogue == kEpiQkvRopeAppend) return false;
  if (q.paired && (q.group_size > 0 || !(swiglu && q.tiled && (q.N / 2) % 64 == 0))) return false;   // (group scales lie in logical row order)
  if (swiglu && !q.paired && (q.N / 2) % 128 != 0) return false;
  return aligned_to(q.packed, 16) && aligned_to(q.x, 16) && (q.x_stride * 2) % 16 == 0;
}

int qgemv_stream_plan(const QGemvParams& q) {
  const Split s = choose_split(q.N, q.K, q.M);
  return (s.rg << 4) | s.split;
}

int launch_qgemv_stream(const QGemvParams& q, cudaStream_t stream) {
  const bool swiglu = q.epilogue == CACHEIR_B200_EPI_SWIGLU;
  StreamParams p{};
  p.x = static_cast<const __half*>(q.x); p.packed = static_cast<const uint8_t*>(q.packed); p.scales = q.scales; p.zero_points = q.zero_points;
  p.residual_on = q.epilogue == CACHEIR_B200_EPI_RESIDUAL ? 1 : 0;
  p.residual = static_cast<const __half*>(q.residual); p.y = static_cast<__half*>(q.y);
  p.M = q.M; p.N = q.N; p.K = q.K; p.n_out = swiglu ? q.N / 2 : q.N; p.x_stride = q.x_stride;
  p.scale_f16 = q.scale_dtype == CACHEIR_B200_F16 ? 1 : 0;
  p.groups = q.group_size > 0 ? q.K / q.group_size : 1;
  p.kb_per_group = q.group_size > 0 ? q.group_size / 128 : 1;
  p.tiled = q.tiled ? 1 : 0; p.paired = q.paired ? 1 : 0;
  return q.group_size > 0 ? launch_nt<true>(p, swiglu, stream) : launch_nt<false>(p, swiglu, stream);
}

}  // namespace cb200
