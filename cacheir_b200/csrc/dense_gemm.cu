// Plain entry points of the dense tensor-core GEMM (dense_gemm.cuh).
#include "dense_gemm.cuh"

namespace cb200 {
namespace {

// Tokens from which pairs are considered: below, a tile of 256 weight rows often leaves the last turn emptier than K split over single
// CTAs. Measured over whole prompts of width 4096, single CTAs and pairs: 230 tokens 1603 and 1574 us, 330 tokens 2877 and 3064, another
// family 1944 and 1982; 2048 tokens 6155 and 5432. Nothing between 331 and 767 tokens was measured.
constexpr int kPairTokens = 768;

struct Shape { int mt, split; };
Shape choose_shape(int T, int N, int K, int batch) {
  const int n_tiles = (N + kTileN - 1) / kTileN * batch;
  int mt = T <= 16 ? 16 : T <= 32 ? 32 : T <= 64 ? 64 : 128;
  // (products per head with a short K are all epilogue: two CTAs per SM take turns. 32 heads of 128 x 512, 2048 tokens: 87 to 54 us;
  // fewer tokens than the line keep tiles of 256: not measured)
  if (T >= 256 && !(batch > 1 && K <= 1024 && T >= kPairTokens) && n_tiles * ((T + 255) / 256) >= kNumSMs) mt = 256;
  const int tiles = n_tiles * ((T + mt - 1) / mt);
  const int kblocks = (K + kBlockK - 1) / kBlockK;
  const int slots = kNumSMs * ctas_per_sm(mt);
  int split = 1;
  while (split < 8 && tiles * split * 2 <= slots && kblocks / (split * 2) >= 4) split *= 2;
  return {mt, split};
}

// Time of the product in nanoseconds on pairs (tiles of 256 weight rows x `tt` tokens) and on single CTAs: a turn is the k blocks of a
// tile plus its epilogue, of which pairs show only what the next tile's main loop does not cover. Fitted to 325 plain products of
// 768 to 2048 tokens, 512 to 22016 rows and K of 512 to 8192, timed on both forms; 3 to 7 % off (standard deviation). Since pairs issue and copy
// faster their tiles of 128 tokens take up to a third less than this says (1001x6144x2048 37.7 / 25.2 us): the choice leaves some of that unused.
long long pair_cost(int T, int N, int K, int batch, int tt) {
  const long long tiles = static_cast<long long>((T + tt - 1) / tt) * ((N + 2 * kTileN - 1) / (2 * kTileN)) * batch;
  const long long turns = (tiles + kNumSMs / 2 - 1) / (kNumSMs / 2), kblocks = (K + kBlockK - 1) / kBlockK;
  return tt == 256 ? 7300 + turns * (300 * kblocks + 4600) : 6000 + turns * (300 * kblocks + 1700);
}

long long single_cost(int T, int N, int K, int batch) {
  const Shape s = choose_shape(T, N, K, batch);
  const long long ctas = static_cast<long long>((T + s.mt - 1) / s.mt) * ((N + kTileN - 1) / kTileN) * batch * s.split;
  const long long turns = (ctas + kNumSMs - 1) / kNumSMs, kblocks = ((K + kBlockK - 1) / kBlockK + s.split - 1) / s.split;
  if (s.mt == 256) return 900 + turns * (350 * kblocks + 8900);
  return s.split > 1 ? 2400 + turns * (195 * kblocks + 4800) : 1600 + turns * (195 * kblocks + 3100);
}

// Tokens per tile of a CTA pair, 0: single CTAs. Pairs only where they come out ahead: taken for all of those 325 products they were
// up to 1.35 times slower (1153 x 1024 x 8192 46.2 us, on single CTAs that split K 34.3; 1001 x 4096 x 512 14.0 and 10.9, where the
// epilogue is most of it), up to 1.6 times faster (2048 x 14336 x 2048 94.9 and 144.1). By cost the 325 take 4.9 % less time than on
// pairs alone and 12.1 % less than on single CTAs alone (geometric means), 0.1 % more than the better form of each (9 % at most).
int choose_pair(int T, int N, int K, int batch) {
  if (T < kPairTokens || (batch > 1 && (K <= 1024 || N % (2 * kTileN) != 0))) return 0;
  auto cost = [&](int tt) {          // turns of the busiest pair, in tiles of 128 tokens (a narrow tile asks more of L2)
    const long long tiles = static_cast<long long>((T + tt - 1) / tt) * ((N + 2 * kTileN - 1) / (2 * kTileN)) * batch;
    return (tiles + kNumSMs / 2 - 1) / (kNumSMs / 2) * (tt == 256 ? 16 : 10);
  };
  const long long tiles = static_cast<long long>((T + 127) / 128) * ((N + 2 * kTileN - 1) / (2 * kTileN)) * batch;
  if (tiles < kNumSMs / 4) return 0;          // few tiles: single CTAs that split K
  const int tt = cost(256) <= cost(128) ? 256 : 128;
  return pair_cost(T, N, K, batch, tt) <= single_cost(T, N, K, batch) ? tt : 0;
}

template <int EPI>
int launch_mt(const cacheir_b200_dense_args& p, cudaStream_t stream) {
  switch (choose_pair(p.T, p.N, p.K, p.batch)) {
    case 256: return launch_pair<EPI, 256>(p, stream);
    case 128: return launch_pair<EPI, 128>(p, stream);
    default: break;
  }
  const Shape s = choose_shape(p.T, p.N, p.K, p.batch);
  switch (s.mt) {
    case 16: return launch<EPI, 16, false>(p, s.split, stream, {});
    case 32: return launch<EPI, 32, false>(p, s.split, stream, {});
    case 64: return launch<EPI, 64, false>(p, s.split, stream, {});
    case 128: return launch<EPI, 128, false>(p, s.split, stream, {});
    default: return launch<EPI, 256, false>(p, s.split, stream, {});
  }
}

}  // namespace

}  // namespace cb200

using namespace cb200;

extern "C" int cacheir_b200_dense_supported(int K, long long w_stride, long long x_stride, int batch, int x_batch_cols) {
  return K > 0 && w_stride % 8 == 0 && x_stride % 8 == 0 && (batch <= 1 || x_batch_cols % 8 == 0) ? 1 : 0;
}

extern "C" int cacheir_b200_dense_pair_tokens(int T, int N, int K, int batch) {
  return T > 0 && N > 0 && K > 0 && batch > 0 ? choose_pair(T, N, K, batch) : 0;
}

extern "C" int cacheir_b200_dense_gemm(const cacheir_b200_dense_args* args, void* stream) {
  if (!args) return CACHEIR_B200_EINVAL;
  cacheir_b200_dense_args p = *args;
  if (p.T <= 0 || p.N <= 0) return 0;
  if (p.batch < 1) p.batch = 1;
  if (p.K <= 0 || !p.x || !p.w) return CACHEIR_B200_EINVAL;
  if (!cacheir_b200_dense_supported(p.K, p.w_stride, p.x_stride, p.batch, p.x_batch_cols) || !aligned_to(p.x, 16) || !aligned_to(p.w, 16))
    return CACHEIR_B200_EALIGN;
  if (p.w_stride < p.K || p.x_stride < static_cast<long long>(p.x_batch_cols) * (p.batch - 1) + p.K) return CACHEIR_B200_EINVAL;
  if (p.batch > 1 && (p.w_batch_rows < p.N || p.bias)) return CACHEIR_B200_EINVAL;
  if ((static_cast<long long>(p.N) + kTileN - 1) / kTileN * p.batch > 65535) return CACHEIR_B200_ELIMIT;
  const bool tail_ok = p.tail_cols >= 0 && p.tail_cols <= p.N && (p.tail_cols == 0 || (p.tail && p.batch == 1));
  cudaStream_t st = as_stream(stream);
  switch (p.epilogue) {
    case CACHEIR_B200_DENSE_BF16: return p.y && tail_ok ? launch_mt<CACHEIR_B200_DENSE_BF16>(p, st) : CACHEIR_B200_EINVAL;
    case CACHEIR_B200_DENSE_F32: return p.y ? launch_mt<CACHEIR_B200_DENSE_F32>(p, st) : CACHEIR_B200_EINVAL;
    case CACHEIR_B200_DENSE_SILU: return p.y && tail_ok ? launch_mt<CACHEIR_B200_DENSE_SILU>(p, st) : CACHEIR_B200_EINVAL;
    case CACHEIR_B200_DENSE_RELU2: return p.y ? launch_mt<CACHEIR_B200_DENSE_RELU2>(p, st) : CACHEIR_B200_EINVAL;
    case CACHEIR_B200_DENSE_GEGLU:
    case CACHEIR_B200_DENSE_SWIGLU:
    case CACHEIR_B200_DENSE_CLAMPED_GLU:
      if (!p.y || !tail_ok || (p.N - p.tail_cols) % 2 != 0 || p.batch != 1)
        return CACHEIR_B200_EINVAL;
      if (p.epilogue == CACHEIR_B200_DENSE_GEGLU) return launch_mt<CACHEIR_B200_DENSE_GEGLU>(p, st);
      if (p.epilogue == CACHEIR_B200_DENSE_SWIGLU) return launch_mt<CACHEIR_B200_DENSE_SWIGLU>(p, st);
      return launch_mt<CACHEIR_B200_DENSE_CLAMPED_GLU>(p, st);
    case CACHEIR_B200_DENSE_GATED:
      return p.y && p.gate ? launch_mt<CACHEIR_B200_DENSE_GATED>(p, st) : CACHEIR_B200_EINVAL;
    case CACHEIR_B200_DENSE_GELU_EMBED:
      if (!p.y || !p.ids || !p.table || p.vocab <= 0 || p.batch != 1) return CACHEIR_B200_EINVAL;
      return launch_mt<CACHEIR_B200_DENSE_GELU_EMBED>(p, st);
    case CACHEIR_B200_DENSE_RESIDUAL:
      if (!p.residual || !p.norm_w || !p.norm_b || p.batch != 1) return CACHEIR_B200_EINVAL;
      if (p.next_mode != CACHEIR_B200_NEXT_NONE && !p.next_out) return CACHEIR_B200_EINVAL;
      if (p.next_mode == CACHEIR_B200_NEXT_DYT && (!p.next_w || !p.next_b)) return CACHEIR_B200_EINVAL;
      return launch_mt<CACHEIR_B200_DENSE_RESIDUAL>(p, st);
    default: return CACHEIR_B200_EINVAL;
  }
}

extern "C" int cacheir_b200_ragged_device_status(int reset) { return device_status_word(g_dense_status, reset != 0); }
