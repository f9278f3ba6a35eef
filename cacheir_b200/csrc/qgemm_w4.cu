// int4 dequant-GEMM for up to 128 activation rows with the weights as a tensor-memory operand, sm_100a.
//
//   y[M, N] = x[M, K] . deq(W)[N, K]^T        fp16 x/y, int4 codes (per row affine or group-wise symmetric), tile or row order
//
// The weights are the 128-row operand A of tcgen05.mma and come from tensor memory: a converter thread owns a weight row, reads its
// 64 bytes of a k block of 128 columns from the ring that the copies fill, turns them into exact fp16 integers (code - zero) and
// stores them with tcgen05.st into columns of its own lane. Through shared memory the same tile costs 32 KB of stores and 32 KB of
// reads by the tensor core (880 cycles of a k block of 128 x 128 in qgemm_tc.cu); warp MMAs take 64 x 4 cycles for
// every eight activation rows. Here a k block costs the integer pipe 256 cycles (two of its operations for each pair of weights),
// whatever the number of activation rows up to 64, and HBM delivers a k block per SM in 350. x is the other operand, straight from
// memory by TMA.
//
// Group scales: the sums of a k block start from zero in one of several accumulators, and drain warps add them up in fp32 registers with
// the row's scale while the next k block is multiplied. Per-row formats leave their sums in one accumulator.
// A K split runs over the CTAs of a cluster; their fp32 sums meet in rank order: deterministic.
//
// Warps: 0 and 2 copy codes, 1 issues MMAs, 3 copies x, 4.. converters in groups of four (a k block each), then the drain warps.
#include "common.cuh"
#include "qgemv_common.cuh"
#include "tc_ptx.cuh"

namespace cb200 {
namespace {

using namespace ptx;

constexpr int kRows = 128;                 // weight rows of a CTA
constexpr int kCols = 128;                 // columns of a k block
constexpr int kRaw = kRows * kCols / 2;    // bytes of its codes
constexpr int kPitch = kRows + 4;          // of the sums in shared memory, in floats
constexpr int kACols = kCols / 2;          // tensor-memory columns of a weight tile

__device__ int g_w4_status = 0;            // 0 ok; otherwise (14 << 8 | id) of the first wait that gave up

// Up to 16 activation rows two CTAs fit on an SM, so that the next kernel's are there when this one's last k blocks are multiplied.
__host__ __device__ constexpr int converters(int nt) { return nt == 16 || nt == 128 ? 2 : 3; }          // groups of four warps
__host__ __device__ constexpr int drains(int nt) { return nt <= 32 ? 1 : 2; }
__host__ __device__ constexpr int threads(int nt) { return 128 * (1 + converters(nt) + drains(nt)); }
__host__ __device__ constexpr int ctas_per_sm(int nt) { return nt == 16 ? 2 : 1; }
__host__ __device__ constexpr int op_stages(int nt) { return nt == 16 ? 3 : nt == 32 ? 6 : 4; }          // a weight tile and its activations
__host__ __device__ constexpr int accumulators(int nt) { return nt == 16 ? 3 : nt == 128 ? 2 : 4; }      // (no more than stages: a phase of `done` must not pass its reader twice)
__host__ __device__ constexpr int tmem_cols(int nt) { return nt == 16 ? 256 : 512; }
__host__ __device__ constexpr int raw_stages(int nt) { return nt == 16 ? 9 : nt == 128 ? 11 : 16; }
__host__ __device__ constexpr int x_bytes(int nt) { return nt * kCols * 2; }
__host__ __device__ constexpr int ring_bytes(int nt) { return raw_stages(nt) * kRaw + op_stages(nt) * x_bytes(nt); }
constexpr int kTail = 1024;                // barriers, tensor-memory base, sums of x
constexpr int kAhead = 16;                 // k blocks a CTA asks for before its turn

struct W4Params {
  const __half* x;
  const void* scales;
  const float* zero_points;
  const __half* residual;
  __half* y;
  int M, N, K, n_out;
  long long x_stride;
  int scale_f16, groups, kb_per_group;
  int tiled, paired, residual_on, split;
};

__device__ __forceinline__ void mma_f16_ts(uint32_t tmem_d, uint32_t tmem_a, uint64_t b_desc, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}"
      ::"r"(tmem_d), "r"(tmem_a), "l"(b_desc), "r"(idesc), "r"(accumulate) : "memory");
}
__device__ __forceinline__ void tmem_st_x32(uint32_t addr, const uint32_t (&v)[32]) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,"
      "%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31,%32};"
      ::"r"(addr), "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7]), "r"(v[8]), "r"(v[9]), "r"(v[10]),
      "r"(v[11]), "r"(v[12]), "r"(v[13]), "r"(v[14]), "r"(v[15]), "r"(v[16]), "r"(v[17]), "r"(v[18]), "r"(v[19]), "r"(v[20]), "r"(v[21]),
      "r"(v[22]), "r"(v[23]), "r"(v[24]), "r"(v[25]), "r"(v[26]), "r"(v[27]), "r"(v[28]), "r"(v[29]), "r"(v[30]), "r"(v[31]) : "memory");
}
__device__ __forceinline__ void tmem_wait_st() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }
__device__ __forceinline__ void tma_load_3d(uint32_t dst, const CUtensorMap* map, uint32_t bar, int x, int y, int z) {
  asm volatile(
      "cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5}], [%2];"
      ::"r"(dst), "l"(reinterpret_cast<uint64_t>(map)), "r"(bar), "r"(x), "r"(y), "r"(z) : "memory");
}
__device__ __forceinline__ float load_peer(const float* local, uint32_t rank) {
  float v;
  asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v) : "r"(map_to_rank(smem_u32(local), rank)) : "memory");
  return v;
}
__device__ __forceinline__ __half2 as_half2(uint32_t v) { return *reinterpret_cast<__half2*>(&v); }
__device__ __forceinline__ uint32_t as_bits(__half2 v) { return *reinterpret_cast<uint32_t*>(&v); }
// byte j of w: its two nibbles as (low - zero, high - zero). (0x6400 | n, 0x6400 | n << 4) = (1024 + n, 1024 + 16 n); one exact fma
__device__ __forceinline__ uint32_t nibble_pair(uint32_t w, int j, __half2 sub) {
  const uint32_t t = __byte_perm(w, 0x64646464u, 0x4040 + 0x101 * j) & 0x64F0640Fu;
  return as_bits(__hfma2(as_half2(t), __floats2half2_rn(1.f, 0.0625f), sub));
}
__device__ __forceinline__ bool exact_zero(float zero) { return zero == rintf(zero) && fabsf(zero) <= 960.f; }

// stage and phase of a ring of S stages
template <int S>
struct Ring {
  uint32_t s = 0, phase = 0;
  __device__ __forceinline__ void next(uint32_t step = 1) {
    s += step;
    if (s >= S) { s -= S; phase ^= 1; }
  }
};

template <int NT, bool GROUPED, bool SWIGLU>
__global__ void __launch_bounds__(threads(NT), ctas_per_sm(NT))
qgemm_w4_kernel(const __grid_constant__ CUtensorMap tmap_w, const __grid_constant__ CUtensorMap tmap_x, const W4Params p) {
  constexpr int SR = raw_stages(NT), SO = op_stages(NT), DB = GROUPED ? accumulators(NT) : 1;
  constexpr int CG = converters(NT), DG = drains(NT), kThreads = threads(NT);
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~static_cast<uintptr_t>(1023));
  uint8_t* s_x = smem;                               // [SO][2][NT][128 bytes]
  uint8_t* s_w = smem + SO * x_bytes(NT);            // [SR][128][64 bytes]
  uint64_t* raw_full = reinterpret_cast<uint64_t*>(smem + ring_bytes(NT));
  uint64_t* raw_empty = raw_full + SR;
  uint64_t* full = raw_empty + SR;                   // [SO] the weight tile is in tensor memory, the activations in shared memory
  uint64_t* done = full + SO;                        // [SO] its MMAs have retired: the stage is free, the sums are there
  uint64_t* drained = done + SO;                     // [DB] the accumulator has been read; per-row formats: [0] all MMAs have retired
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(drained + accumulators(NT));
  float* s_xsum = reinterpret_cast<float*>(smem + ring_bytes(NT) + 512);
  float* part = reinterpret_cast<float*>(smem);      // [M][kPitch], over the drained rings

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int rank = p.split > 1 ? static_cast<int>(cluster_ctarank()) : 0;
  const int kblocks = p.K / kCols;
  const int kb0 = kblocks * rank / p.split, total = kblocks * (rank + 1) / p.split - kb0;
  // first weight row of each half of 64 rows; with SwiGLU the gate rows and the up rows of the same outputs
  const int row0 = blockIdx.x * (SWIGLU ? 64 : 128), row1 = SWIGLU ? p.N / 2 + row0 : row0 + 64;
  auto weight_row = [&](int r) { return (r < 64 ? row0 : row1 - 64) + r; };
  // Tile order is read as rows of 128 bytes (32 for 64 weight rows of a k block; paired bands hold the gate and up rows of an output):
  // a thread issues a tensor copy of a tile in about 200 cycles, a plain bulk copy of the same 8 KB in 500.
  const bool whole = p.tiled && (!SWIGLU || p.paired);       // (the two halves lie behind one another)
  const int line0 = (SWIGLU && p.paired ? static_cast<int>(blockIdx.x) * kblocks * 64 : (row0 >> 7) * kblocks * 64 + ((row0 >> 6) & 1) * 32) + kb0 * 64;
  const int line1 = SWIGLU && !p.paired ? (row1 >> 7) * kblocks * 64 + ((row1 >> 6) & 1) * 32 + kb0 * 64 : line0 + 32;

  if (warp == 2) {                                   // the weights set out for L2 while the kernel before this one is at work
    for (int i = lane; i < min(total, kAhead); i += 32) {
      if (p.tiled) {
        tma_prefetch_2d(&tmap_w, 0, line0 + i * 64);
        if (!whole) tma_prefetch_2d(&tmap_w, 0, line1 + i * 64);
      } else {
        tma_prefetch_2d(&tmap_w, (kb0 + i) * (kCols / 2), row0);
        tma_prefetch_2d(&tmap_w, (kb0 + i) * (kCols / 2), row1);
      }
    }
  } else if (threadIdx.x == 0) {
    for (int s = 0; s < SR; ++s) { mbar_init(smem_u32(&raw_full[s]), 1); mbar_init(smem_u32(&raw_empty[s]), 4); }
    for (int s = 0; s < SO; ++s) { mbar_init(smem_u32(&full[s]), 5); mbar_init(smem_u32(&done[s]), 1); }      // (four converter warps, the copies)
    for (int s = 0; s < DB; ++s) mbar_init(smem_u32(&drained[s]), GROUPED ? 4 * DG : 1);
    mbar_fence_init();
  }
  __syncthreads();
  chain_enter();
  if (warp == 1 || warp >= 4) {                      // (the copies do not wait for tensor memory)
    if (warp == 1) tc_alloc(smem_u32(tmem_slot), tmem_cols(NT));
    tc_fence_before();
    asm volatile("bar.sync 1, %0;" ::"n"(kThreads - 96) : "memory");
    tc_fence_after();
  }
  const uint32_t tmem = warp == 1 || warp >= 4 ? *tmem_slot : 0u;  // weight tiles, then accumulators
  const uint32_t tmem_d = tmem + SO * kACols;
  const uint32_t b_full = smem_u32(full), b_done = smem_u32(done), b_drained = smem_u32(drained);

  // (One thread's waits, copies and MMAs are a chain of dependent instructions, several hundred cycles for a k block if every
  // stage and phase is worked out from the k block's number: they are carried along.)
  bool odd_zero = false;                             // a zero point that is no small integer: corrected at the end
  if (warp == 0 || warp == 2) {
    if (lane == 0) {
      // ---------------- copies of the codes: two warps take turns (a thread needs 300 to 500 cycles for a k block) ----------------
      Ring<SR> rw{static_cast<uint32_t>(warp >> 1), 0};
      const uint32_t w_full = smem_u32(raw_full), w_empty = smem_u32(raw_empty), w_at = smem_u32(s_w);
      int issued = warp >> 1;
      for (; issued < total; issued += 2) {
        if (issued >= SR && !mbar_wait(w_empty + 8 * rw.s, rw.phase ^ 1, &g_w4_status, (14 << 8) | 1)) break;
        const uint32_t bar = w_full + 8 * rw.s, dst = w_at + kRaw * rw.s;
        mbar_expect_tx(bar, kRaw);
        if (p.tiled) {
          tma_load_2d(dst, &tmap_w, bar, 0, line0 + issued * 64);
          if (!whole) tma_load_2d(dst + kRaw / 2, &tmap_w, bar, 0, line1 + issued * 64);
        } else {
          const int k = (kb0 + issued) * (kCols / 2);
          tma_load_2d(dst, &tmap_w, bar, k, row0);
          tma_load_2d(dst + kRaw / 2, &tmap_w, bar, k, row1);
        }
        rw.next(2);
      }
      if (issued < total)                            // a wait gave up: nothing may still be on its way when the block ends
        for (int i = issued - 2 * (SR / 2); i < issued; i += 2)
          if (i >= 0 && !mbar_wait(w_full + 8 * (i % SR), (i / SR) & 1, &g_w4_status, (14 << 8) | 3)) break;
    }
    __syncwarp();
  } else if (warp == 3) {
    if (lane == 0) {
      // ---------------- copies of the activations ----------------
      // (they also wait for the accumulator that the k block's sums go to, so that the MMAs have one barrier to wait for)
      Ring<SO> ro;
      Ring<DB> rd;
      // (rows past M are left as they are: they only reach sums that nobody stores)
      const uint32_t x_at = smem_u32(s_x), x_row_bytes = static_cast<uint32_t>(p.M) * kCols * 2, half = NT * 128;
      int issued = 0;
      for (; issued < total; ++issued) {
        if (issued >= SO && !mbar_wait(b_done + 8 * ro.s, ro.phase ^ 1, &g_w4_status, (14 << 8) | 2)) break;
        if (GROUPED && issued >= DB && !mbar_wait(b_drained + 8 * rd.s, rd.phase ^ 1, &g_w4_status, (14 << 8) | 5)) break;
        mbar_expect_tx(b_full + 8 * ro.s, x_row_bytes);
        if (p.M == NT) {
          tma_load_3d(x_at + x_bytes(NT) * ro.s, &tmap_x, b_full + 8 * ro.s, 0, 0, (kb0 + issued) * 2);
        } else {
          tma_load_2d(x_at + x_bytes(NT) * ro.s, &tmap_x, b_full + 8 * ro.s, (kb0 + issued) * kCols, 0);
          tma_load_2d(x_at + x_bytes(NT) * ro.s + half, &tmap_x, b_full + 8 * ro.s, (kb0 + issued) * kCols + 64, 0);
        }
        ro.next();
        if (GROUPED) rd.next();
      }
      if (issued < total)
        for (int i = issued > SO ? issued - SO : 0; i < issued; ++i)
          if (!mbar_wait(b_full + 8 * (i % SO), (i / SO) & 1, &g_w4_status, (14 << 8) | 3)) break;
    }
    __syncwarp();
  } else if (warp == 1) {
    // ---------------- MMAs: fp32 sums, fp16 x fp16, x K-major, M 128, N = NT (one elected thread issues them) ----------------
    constexpr uint32_t idesc = (1u << 4) | (static_cast<uint32_t>(NT >> 3) << 17) | (static_cast<uint32_t>(kRows >> 4) << 24);
    const uint64_t x_desc = smem_desc_sw128(smem_u32(s_x));          // (an offset in shared memory adds to the lowest bits, by 16 bytes)
    const bool leader = elect_one();
    Ring<SO> ro;
    Ring<DB> rd;
    for (int i = 0; i < total; ++i) {
      if (!__all_sync(0xffffffffu, mbar_wait(b_full + 8 * ro.s, ro.phase, &g_w4_status, (14 << 8) | 4))) break;
      tc_fence_after();
      if (leader) {
        const uint64_t desc = x_desc + ro.s * (x_bytes(NT) >> 4);
        const uint32_t a_at = tmem + ro.s * kACols, d_at = tmem_d + rd.s * NT;
#pragma unroll
        for (int j = 0; j < kCols / 16; ++j)
          mma_f16_ts(d_at, a_at + j * 8, desc + ((j >> 2) * (NT * 128) + (j & 3) * 32) / 16, idesc, (GROUPED ? j > 0 : i > 0 || j > 0) ? 1u : 0u);
        tc_commit(b_done + 8 * ro.s);
      }
      __syncwarp();
      ro.next();
      if (GROUPED) rd.next();
    }
    if (!GROUPED && leader) tc_commit(b_drained);
    __syncwarp();
  } else if (warp >= 4 && warp < 4 + 4 * CG) {
    // ---------------- converters: thread = weight row, group = every CG-th k block ----------------
    const int group = (warp - 4) >> 2, r = (warp & 3) * 32 + lane;
    float zero = 8.f;
    const int wrow = weight_row(r);
    if (!GROUPED && p.zero_points && wrow < p.N) zero = p.zero_points[wrow];
    odd_zero = !exact_zero(zero);
    const float z = odd_zero ? 0.f : zero;
    const __half2 sub = __floats2half2_rn(-(1024.f + z), -(64.f + z));
    const uint32_t a_base = tmem + (static_cast<uint32_t>((warp & 3) * 32) << 16);
    const int turn = (r >> 1) & 3;                   // 16-byte pieces lie in swizzled order
    const uint8_t* const row = s_w + r * 64;
    const uint32_t w_full = smem_u32(raw_full), w_empty = smem_u32(raw_empty);
    Ring<SR> rw{static_cast<uint32_t>(group), 0};
    Ring<SO> ro{static_cast<uint32_t>(group), 0};
    for (int i = group; i < total; i += CG) {
      bool ok = mbar_wait(w_full + 8 * rw.s, rw.phase, &g_w4_status, (14 << 8) | 7);
      if (i >= SO) ok = ok && mbar_wait(b_done + 8 * ro.s, ro.phase ^ 1, &g_w4_status, (14 << 8) | 8);
      if (!__all_sync(0xffffffffu, ok)) break;
      tc_fence_after();
      const uint8_t* const at = row + rw.s * kRaw;
#pragma unroll
      for (int h = 0; h < 2; ++h) {                  // 64 columns
        const uint4 c0 = *reinterpret_cast<const uint4*>(at + 16 * ((2 * h) ^ turn));
        const uint4 c1 = *reinterpret_cast<const uint4*>(at + 16 * ((2 * h + 1) ^ turn));
        const uint32_t w[8] = {c0.x, c0.y, c0.z, c0.w, c1.x, c1.y, c1.z, c1.w};
        uint32_t v[32];
#pragma unroll
        for (int k = 0; k < 8; ++k)
#pragma unroll
          for (int j = 0; j < 4; ++j) v[4 * k + j] = nibble_pair(w[k], j, sub);
        tmem_st_x32(a_base + ro.s * kACols + h * 32, v);
      }
      tmem_wait_st();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) {
        mbar_arrive(b_full + 8 * ro.s);
        mbar_arrive(w_empty + 8 * rw.s);
      }
      rw.next(CG);
      ro.next(CG);
    }
  } else if (warp >= 4 + 4 * CG) {
    // ---------------- drain: thread = weight row, group = a share of the activation rows ----------------
    constexpr int kShare = NT / DG;
    const int group = (warp - 4 - 4 * CG) >> 2, r = (warp & 3) * 32 + lane;
    const uint32_t lane_addr = static_cast<uint32_t>((warp & 3) * 32) << 16;
    float acc[kShare];
    if constexpr (GROUPED) {
#pragma unroll
      for (int j = 0; j < kShare; ++j) acc[j] = 0.f;
      // scales of kNext k blocks are asked for at a time, a turn ahead of their use
      constexpr int kNext = 4;
      const size_t first = static_cast<size_t>(min(weight_row(r), p.N - 1)) * p.groups;
      int block = kb0, group_at = kb0 / p.kb_per_group, group_end = (group_at + 1) * p.kb_per_group;
      auto ask = [&](float (&sc)[kNext]) {
#pragma unroll
        for (int k = 0; k < kNext; ++k) {
          const size_t at = first + min(group_at, p.groups - 1);
          sc[k] = p.scale_f16 ? __half2float(static_cast<const __half*>(p.scales)[at]) : static_cast<const float*>(p.scales)[at];
          if (++block == group_end) { ++group_at; group_end += p.kb_per_group; }
        }
      };
      float now[kNext], next[kNext];
      ask(now);
      Ring<SO> ro;
      Ring<DB> rd;
      bool ok = true;
      for (int i0 = 0; i0 < total && ok; i0 += kNext) {
        ask(next);
#pragma unroll
        for (int k = 0; k < kNext; ++k) {
          if (i0 + k >= total || !ok) break;
          ok = __all_sync(0xffffffffu, mbar_wait(b_done + 8 * ro.s, ro.phase, &g_w4_status, (14 << 8) | 9));
          if (!ok) break;
          tc_fence_after();
#pragma unroll
          for (int c = 0; c < kShare; c += 16) {
            uint32_t v[16];
            tc_ld_x16(tmem_d + lane_addr + rd.s * NT + group * kShare + c, v);
            tc_wait_ld();
            if (c + 16 == kShare) {                  // the accumulator is free before its last sums are added up
              tc_fence_before();
              __syncwarp();
              if (lane == 0) mbar_arrive(b_drained + 8 * rd.s);
            }
#pragma unroll
            for (int j = 0; j < 16; ++j) acc[c + j] = fmaf(__uint_as_float(v[j]), now[k], acc[c + j]);
          }
          ro.next();
          rd.next();
        }
#pragma unroll
        for (int k = 0; k < kNext; ++k) now[k] = next[k];
      }
    } else {
      mbar_wait(b_drained, 0, &g_w4_status, (14 << 8) | 9);
      __syncwarp();
      tc_fence_after();
#pragma unroll
      for (int c = 0; c < kShare; c += 16) {
        uint32_t v[16];
        tc_ld_x16(tmem_d + lane_addr + group * kShare + c, v);
        tc_wait_ld();
#pragma unroll
        for (int j = 0; j < 16; ++j) acc[c + j] = __uint_as_float(v[j]);
      }
    }
    // (all k blocks have been multiplied: nothing reads the rings any more)
#pragma unroll
    for (int j = 0; j < kShare; ++j)
      if (group * kShare + j < p.M) part[(group * kShare + j) * kPitch + r] = acc[j];
  }

  // ---- the sums of the cluster's CTAs meet; each finishes a share of the outputs ----
  tc_fence_before();
  const bool correct = __syncthreads_or(odd_zero) != 0;
  if (warp == 1) {
    tc_fence_after();
    tc_dealloc(tmem, tmem_cols(NT));
  }
  if (!GROUPED && correct) {                         // sums of x, for the rows whose zero point has not been subtracted (rare)
    for (int m = warp; m < p.M; m += kThreads / 32) {
      float v = 0.f;
      for (int k = lane; k < p.K; k += 32) v += __half2float(p.x[static_cast<size_t>(m) * p.x_stride + k]);
      v = warp_sum(v);
      if (lane == 0) s_xsum[m] = v;
    }
    __syncthreads();
  }
  if (p.split > 1) cluster_sync_release();
  // A thread keeps its output column (the threads are a multiple of them) and goes down the activation rows.
  constexpr int kOut = SWIGLU ? 64 : 128, kStep = kThreads / kOut;
  const int r = threadIdx.x % kOut, col = row0 + r;
  if (col < p.n_out) {
    float scale[2] = {1.f, 1.f}, zero[2] = {0.f, 0.f};
    if constexpr (!GROUPED) {
#pragma unroll
      for (int h = 0; h < (SWIGLU ? 2 : 1); ++h) {
        const int row = h ? p.N / 2 + col : col;
        scale[h] = p.scale_f16 ? __half2float(static_cast<const __half*>(p.scales)[row]) : static_cast<const float*>(p.scales)[row];
        if (correct) {
          zero[h] = p.zero_points ? p.zero_points[row] : 8.f;
          if (exact_zero(zero[h])) zero[h] = 0.f;
        }
      }
    }
    auto product = [&](int h, int m) {
      const float* at = part + m * kPitch + h * 64 + r;
      float v;
      if (p.split > 1) {                             // all of them are asked for before the first is added
        float sums[8];
#pragma unroll
        for (int k = 0; k < 8; ++k) sums[k] = k < p.split ? load_peer(at, k) : 0.f;
        v = sums[0];
#pragma unroll
        for (int k = 1; k < 8; ++k) v += sums[k];
      } else {
        v = *at;
      }
      if constexpr (!GROUPED) {
        if (correct && zero[h] != 0.f) v -= zero[h] * s_xsum[m];
        v *= scale[h];
      }
      return v;
    };
    const int m0 = rank * kStep + static_cast<int>(threadIdx.x) / kOut;
#pragma unroll 4
    for (int m = m0; m < p.M; m += p.split * kStep) {
      const size_t o = static_cast<size_t>(m) * p.n_out + col;
      const float res = p.residual_on ? __half2float(p.residual[o]) : 0.f;
      float v = product(0, m);
      if constexpr (SWIGLU) v = silu_fast(v) * product(1, m);
      if (p.residual_on) v = __fadd_rn(v, res);
      p.y[o] = __float2half_rn(v);
    }
  }
  if (p.split > 1) cluster_sync_release();           // nobody's sums are read any more
}

// x[M, K]: a box is 64 columns of all rows, in swizzled order; with NT rows as [K/64][M][64], both halves of a k block in one box
bool encode_x(CUtensorMap* map, const void* base, uint64_t K, uint64_t M, uint64_t stride_bytes, uint32_t nt) {
  EncodeTiledFn fn = tensor_map_encoder();
  if (!fn) return false;
  const bool full = M == nt;
  const cuuint64_t dims[3] = {full ? 64 : K, M, K / 64};
  const cuuint64_t strides[2] = {stride_bytes, 128};
  const cuuint32_t box[3] = {64, static_cast<cuuint32_t>(M), 2};
  const cuuint32_t elem_strides[3] = {1, 1, 1};
  return fn(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, full ? 3 : 2, const_cast<void*>(base), dims, strides, box, elem_strides, CU_TENSOR_MAP_INTERLEAVE_NONE,
            CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

// CTAs along K. A cluster lives in one GPC, so that fewer of them run at once than the SMs would hold. In cycles: a k block is 500, the
// first and the last steps of a CTA 3000, the exchange 1200.
int choose_split(int tiles, int kblocks) {
  constexpr struct { int split, at_once; } kForms[] = {{1, kNumSMs}, {2, kNumSMs / 2}, {3, 44}, {4, 32}, {6, 20}, {8, 14}};
  int best = 1;
  long long best_cost = -1;
  for (const auto form : kForms) {
    if (form.split > 1 && kblocks / form.split < 4) break;
    const long long waves = (tiles + form.at_once - 1) / form.at_once;
    const long long cost = waves * (500LL * ((kblocks + form.split - 1) / form.split) + 3000) + (form.split > 1 ? 1200 : 0);
    if (best_cost < 0 || cost < best_cost) { best = form.split; best_cost = cost; }
  }
  return best;
}

template <int NT, bool GROUPED, bool SWIGLU>
int launch(const QGemvParams& q, cudaStream_t stream) {
  constexpr int kSmem = 1024 + ring_bytes(NT) + kTail;
  static_assert(kSmem * ctas_per_sm(NT) <= 227 * 1024, "the rings must fit");
  static_assert(NT * kPitch * 4 <= ring_bytes(NT), "the sums must fit in the drained rings");
  static_assert((2 * (raw_stages(NT) + op_stages(NT)) + accumulators(NT) + 1) * 8 <= 512, "barriers fit in front of the sums of x");
  static_assert(op_stages(NT) * kACols + accumulators(NT) * NT <= tmem_cols(NT), "tiles and accumulators fit in tensor memory");
  CUtensorMap tw, tx;
  if (!encode_x(&tx, q.x, q.K, q.M, static_cast<uint64_t>(q.x_stride) * 2, NT)) return CACHEIR_B200_EUNSUPPORTED;
  // codes in tile order: 32 lines are 64 weight rows of a k block, copied as they lie (in swizzled order)
  const uint64_t lines = static_cast<uint64_t>((q.N + 127) / 128) * (q.K / kCols) * 64;
  if (!(q.tiled ? encode_u8_lines(&tw, q.packed, lines, !SWIGLU || q.paired ? 64 : 32) : encode_u8_rows_sw64(&tw, q.packed, q.K / 2, q.N, q.K / 2, 64))) return CACHEIR_B200_EUNSUPPORTED;
  W4Params p{};
  p.x = static_cast<const __half*>(q.x);
  p.scales = q.scales; p.zero_points = q.zero_points;
  p.residual = static_cast<const __half*>(q.residual); p.y = static_cast<__half*>(q.y);
  p.residual_on = q.epilogue == CACHEIR_B200_EPI_RESIDUAL ? 1 : 0;
  p.M = q.M; p.N = q.N; p.K = q.K; p.n_out = SWIGLU ? q.N / 2 : q.N; p.x_stride = q.x_stride;
  p.scale_f16 = q.scale_dtype == CACHEIR_B200_F16 ? 1 : 0;
  p.groups = GROUPED ? q.K / q.group_size : 1;
  p.kb_per_group = GROUPED ? q.group_size / kCols : 1;
  p.tiled = q.tiled ? 1 : 0; p.paired = q.paired ? 1 : 0;
  const int tiles = SWIGLU ? (p.n_out + 63) / 64 : (p.N + 127) / 128;
  p.split = choose_split(tiles, q.K / kCols);
  auto kern = qgemm_w4_kernel<NT, GROUPED, SWIGLU>;
  cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmem);
  if (e != cudaSuccess) return static_cast<int>(e);
  e = launch_clusters(kern, dim3(tiles, p.split, 1), threads(NT), kSmem, stream, dim3(1, p.split, 1), tw, tx, p);
  if (e != cudaSuccess) return static_cast<int>(e);
  return launch_status();
}

template <int NT>
int launch_nt(const QGemvParams& q, cudaStream_t stream) {
  const bool swiglu = q.epilogue == CACHEIR_B200_EPI_SWIGLU;
  if (q.group_size > 0) return swiglu ? launch<NT, true, true>(q, stream) : launch<NT, true, false>(q, stream);
  return swiglu ? launch<NT, false, true>(q, stream) : launch<NT, false, false>(q, stream);
}

}  // namespace

// Where it takes over (us with the pre-pass where there is one; weights N x K in tile order):
//   group-wise int4, 8 rows: 14336x4096 17.5 / 15.3, 4096x4096 8.0 / 6.9, 4096x2048 6.1 / 5.2 against the streaming kernel (one row
//     15.7 / 15.0, 6.5 / 6.7, 5.1 / 4.9: no further down); 32 rows 30.6 / 15.3, 12.2 / 8.1, 8.5 / 6.4; 64 and 128 rows against qgemm_tc.cu
//     37.5 / 17.4 and 35.3 / 27.9, 19.1 / 9.4 and 15.3 / 13.4
//   per-row int4, 16 rows against the integer kernel 15.1 / 13.5, 9.1 / 7.2, 6.9 / 5.8; 64 rows 30.0 / 14.9, 16.4 / 9.0, 14.6 / 7.7; 128
//     rows 34.3 / 17.6, 26.5 / 11.5, 21.5 / 10.0; 2048x2048 6.8 / 5.2 (16 rows), 13.5 / 7.0, 18.2 / 9.2
// Group-wise codes of fewer than 6 M numbers stay with the streaming kernel up to 32 rows (1024x2048 9 rows 3.9 / 4.3, 32 rows 5.3 / 5.3) and
// leave qgemm_tc.cu beyond (64 rows 14.3 / 6.4; of less than 1 M numbers not measured). Per-row codes of fewer than 3 M numbers or 1024 rows keep the
// integer kernels, which give a row the same bits in passes of 64 rows and of thousands. Codes in row order of N >= 9472 up
// to 8 rows stay, too (a few percent either way).
bool qgemm_w4_preferred(const QGemvParams& q) {
  if (!qgemm_w4_supported(q)) return false;
  const long long numbers = static_cast<long long>(q.N) * q.K;
  if (q.group_size == 0) return q.M > 8 && numbers >= 3LL << 20 && q.N >= 1024;
  return (q.M > 32 && numbers >= 1LL << 20) || (numbers >= 6LL << 20 && (q.M > 8 || (q.M >= 4 && (q.tiled || q.N < 64 * kNumSMs))));
}

int qgemm_w4_plan(const QGemvParams& q) {
  const bool swiglu = q.epilogue == CACHEIR_B200_EPI_SWIGLU;
  return 128 | (4 << 4) | choose_split(swiglu ? (q.N / 2 + 63) / 64 : (q.N + 127) / 128, q.K / kCols);
}

bool qgemm_w4_supported(const QGemvParams& q) {
  if (q.x_dtype != CACHEIR_B200_F16 || q.x_prequantized || q.norm_weight || q.bits != 4) return false;
  if (q.M < 1 || q.M > 128 || q.K % kCols != 0 || q.K < kCols) return false;
  if (q.group_size % kCols != 0) return false;
  if (q.epilogue == kEpiQkvRopeAppend) return false;
  if (q.paired && q.group_size > 0) return false;                                   // (group scales lie in logical row order)
  if (q.epilogue == CACHEIR_B200_EPI_SWIGLU && (q.N / 2) % 64 != 0) return false;
  if (q.scale_dtype != CACHEIR_B200_F16 && q.scale_dtype != CACHEIR_B200_F32) return false;
  if (tensor_map_encoder() == nullptr) return false;
  return aligned_to(q.packed, 16) && aligned_to(q.x, 16) && (q.x_stride * 2) % 16 == 0;
}

int launch_qgemm_w4(const QGemvParams& q, cudaStream_t stream) {
  if (q.M <= 16) return launch_nt<16>(q, stream);
  if (q.M <= 32) return launch_nt<32>(q, stream);
  if (q.M <= 64) return launch_nt<64>(q, stream);
  return launch_nt<128>(q, stream);
}

int qgemm_w4_device_status(bool reset) {
  int status = 0;
  if (cudaMemcpyFromSymbol(&status, g_w4_status, sizeof(int)) != cudaSuccess) return -1;
  if (reset && status != 0) {
    const int zero = 0;
    cudaMemcpyToSymbol(g_w4_status, &zero, sizeof(int));
  }
  return status;
}

}  // namespace cb200
