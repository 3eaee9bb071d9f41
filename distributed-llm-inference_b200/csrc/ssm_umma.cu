// The selective scan (ssm.cu says what is computed) for prompt portions in bfloat16: tiles of 128 tokens in closed form on tcgen05.  Inside a
// tile that starts from S0 (kept transposed: P x N), with l_t the sum of the log decays -exp(A_log) dt up to t,
//   y_t = exp(l_t) S0 C_t + sum_{j <= t} exp(l_t - l_j) dt_j (C_t . B_j) x_j + D x_t,
//   S   = exp(l_last) S0 + sum_j exp(l_last - l_j) dt_j x_j B_j^T.
//
// x, B and C are bfloat16 as the convolution left them; step sizes, decays, weights, the state and every sum are float32, and nothing
// float32 is rounded on its way into a product (mma_split.cuh: three bfloat16 terms, the small ones' products first).  The sums of log
// decays are taken in double and kept as two floats, so that a difference of two of them is as exact as a token-by-token product of the
// decays.
//
// A CTA owns 64 columns p of one head of one sequence and walks its tiles.  Four products a tile, all with 128 rows:
//   G  = C B^T              rows t, columns j, over n: the scores, C and B as TMA brought them
//   dS = B^T (wl o x)       rows n, columns p, over j: B the M-major operand; the weighted values in three terms, written by the warps
//   Yb = C S0^T             rows t, columns p, over n: S0 in three terms, written by the warps
//   Ya = W x                rows t, columns p, over j: the weighted scores in three terms, from tensor memory, where a thread puts them in the
//                           place of the scores that it has read
// Sixteen warps: a thread has row 32 (warp % 4) + lane and sixteen (of G 32) of the columns; the state, in its thread's registers, has rows n.
// Sums over 128 that count (G, Ya, Yb) are kept as two halves and added by the CUDA cores: an addition on the tensor cores cuts off where a
// plain one rounds.  Three more warps issue the products, copy (TMA), and make the tables of step sizes and decays a tile ahead.
//
// Tensor memory, columns: [0, 128) the first half of G, [128, 256) the second, and in their place the terms of W: of sixteen tokens j = 16 k .. the
// high one at 16 k, the low one at 16 k + 8, the middle one at 128 + 16 k; [256, 384) Yb; [384, 512) Ya, in its second half before it dS.
//
// A few long sequences leave most of the GPU idle, because a sequence's tiles follow one another.  They are cut into segments, in two
// launches, as in ssm_tc.cu: the first walks segment 0 and computes what every later segment but the last adds to a state from zero; the
// second starts every later segment from the states in front of it.
//
// A masked weight is 0, and 0 times an infinity or a NaN is a NaN; an infinity in three terms is one too; and the rows of a last tile behind
// the sequence's end are another sequence's.  So a CTA looks at what it computed: where a read-out or the state is not finite, it walks its
// columns again token after token (walk_again), and infinities and NaNs appear where ssm.cu has them.
//
// What bounds it: a tile's chain of steps in the sixteen warps (8,500 clocks; scores and weights 2,000, the terms of the weighted values and the state 1,800, the
// read-outs 1,500, and between them waits for the products, 3,800 clocks of which a tile has), in which a scheduler issues an instruction every other
// clock.  On the way there: the code has to fit the instruction cache (products and scores as loops and a wait of six instructions: 105 -> 80 us with 128 heads
// of 2,048 tokens), read-outs leave by TMA (a row a thread: 3,300 clocks).  Measured, us, against tiles of 64 tokens by mma.sync (ssm_tc.cu; 64 heads, P 64, N 128):
// prompts of 666, 1,000 and 1,335 tokens 160 -> 73, one of 4,096 207 -> 108, of 600 48 -> 28, of 300 38 -> 19, of 33 10 -> 10; 128 heads, one of 2,048
// 195 -> 80; 32 heads, N 64, prompts of 654, 981 and 1,310 67 -> 53.  The errors of y and S against 64 bits are smaller (1,500 tokens: 1.1e-7 and 7.8e-8, before 2.2e-7 and 1.9e-7).
//
// Every wait is bounded: after `wait_limit` polls a code goes to *error_flag, and the CTA goes on to its end without another wait; from then on it stores no read-outs, and
// states not at all.
#include "umma_tiles.cuh"

using namespace dli;
using namespace dli::umma;
typedef __nv_bfloat16 bf16;

namespace {

constexpr int TOKENS = 128;  // of a tile
constexpr int COLS = 64;     // columns p of a CTA
constexpr int WARPS = 16;
constexpr int THREADS = (WARPS + 3) * 32;
constexpr float LOG_FLOOR = -1e4f;  // a log decay below this is 0 as a decay, and its sums stay finite
constexpr double LOG2E = 1.4426950408889634074;
constexpr int SHORT = 4;  // sequences of up to so many tokens are walked

struct Params {
  float* y;
  const bf16* xbc;        // [n][heads P + 2 groups N]: x | B | C
  const bf16* u;          // dt_raw: column dt_col + head
  long long u_stride;
  int dt_col;
  const float *dt_bias, *A_log, *D;
  float* state;           // [slots][heads][P][N]
  const int *q_start, *state_slot;
  int num_seqs, heads, P, N, groups;
  int segments;           // of a sequence; with more than one:
  float* part;            // [seqs][segments - 1][heads][P][N]: the state behind segment 0, then what each segment adds
  float* part_log;        // [seqs][segments - 1][heads]: the sum of its log decays
  // Heads of a short sequence that a CTA walks (the CTAs of the others leave), 2^0 to 2^3: a CTA has an SM to itself, and with a head each 24 single tokens
  // of 64 heads beside a portion of 100 took 44 us of 54; but eight heads take four times as long as one, and few short sequences had better spread.
  int short_shift;
  int y_vec;              // sixteen read-outs side by side lie on a 16-byte boundary
  int* error_flag;
  unsigned wait_limit;
  int skip_tile;          // -1 in every launch of the engine: the tile of every CTA whose copies of B and C a test leaves out
};

// Per tile, floats: l in log2 units (two terms) | dt | exp(l) | exp(l_last - l) dt | exp(l_e - l) dt with e the last token of the block of 32, and exp(l_last)
struct Table {
  static constexpr int HI = 0, LO = TOKENS, DT = 2 * TOKENS, OUT = 3 * TOKENS, IN = 4 * TOKENS, BLOCK = 5 * TOKENS, END = 6 * TOKENS, FLOATS = 6 * TOKENS + 4;
};

template <int NB> struct Shape {  // NB: the state size in slabs of 64
  static constexpr int C = 0, B = NB * SLAB, X = 2 * NB * SLAB, WX = X + 2 * SLAB, S0 = WX + 3 * SLAB, S_TERM = NB * 64 * 128;
  static constexpr int Y = S0 + 3 * S_TERM;  // columns 0..31 of the read-outs on their way out; the others lie where the tile's x lay
  static constexpr int TABLES = Y + SLAB,
                       BARS = TABLES + 2 * Table::FLOATS * 4, SMEM = BARS + 160 + 1024;
  static_assert(SMEM <= 227 * 1024, "shared memory");
};
// Columns of tensor memory
constexpr int T_G = 0, T_YB = 256, T_YA = 384, T_DS = 448, T_ALL = 512;

__device__ __forceinline__ float softplus(float x) { return x > 20.f ? x : log1pf(expf(x)); }

// Token range of segment `seg` of a sequence of `tiles` tiles: segment 0 has what the others' even shares leave (a segment without read-outs costs
// 0.45 of one with).
__device__ __forceinline__ void segment_tiles(int tiles, int segments, int seg, int& from, int& to) {
  if (segments == 1) { from = 0; to = tiles; return; }
  const int rest = segments - 1, share = (20 * tiles + 20 * rest + 8) / (20 * rest + 9);
  const int head = max(1, tiles - share * rest);
  from = seg == 0 ? 0 : min(tiles, head + (seg - 1) * share);
  to = min(tiles, head + seg * share);
}

// The scan of a CTA's columns token after token: from the state `from` in front of token t_from, with read-outs of tokens t_emit .. t_end - 1, the
// state behind them to `to` (or null).  A warp takes four columns; a lane holds every 32nd number of them.
__device__ __noinline__ void walk_again(const Params& p, int head, int col0, const float* from, int t_from, int t_emit, int t_end, float* to) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, N = p.N, P = p.P, inner = p.heads * P, width = inner + 2 * p.groups * N;
  const float A = expf(p.A_log[head]), bias = p.dt_bias[head], Dh = p.D[head];
  const int g = head / (p.heads / p.groups), c0 = col0 + warp * 4;
  if (warp >= WARPS || c0 >= P) return;  // (P is a multiple of 8)
  float S[4][4];
#pragma unroll
  for (int c = 0; c < 4; ++c)
#pragma unroll
    for (int m = 0; m < 4; ++m) S[c][m] = lane + 32 * m < N ? from[(size_t)(c0 + c) * N + lane + 32 * m] : 0.f;
  for (int t = t_from; t < t_end; ++t) {
    const bf16* row = p.xbc + (size_t)t * width;
    const float dt = softplus(to_float(p.u[(size_t)t * p.u_stride + p.dt_col + head]) + bias), decay = expf(-A * dt);
    float B[4], C[4];
#pragma unroll
    for (int m = 0; m < 4; ++m) {
      const bool in = lane + 32 * m < N;
      B[m] = in ? to_float(row[inner + g * N + lane + 32 * m]) : 0.f;
      C[m] = in ? to_float(row[inner + (p.groups + g) * N + lane + 32 * m]) : 0.f;
    }
#pragma unroll
    for (int c = 0; c < 4; ++c) {
      const float x = to_float(row[head * P + c0 + c]), dtx = dt * x;
      float sum = 0.f;
#pragma unroll
      for (int m = 0; m < 4; ++m)
        if (lane + 32 * m < N) {  // (0 times an infinity of a number that is not there must not get through)
          S[c][m] = fmaf(decay, S[c][m], B[m] * dtx);
          sum = fmaf(S[c][m], C[m], sum);
        }
      sum = warp_sum(sum);
      if (t >= t_emit && lane == 0) p.y[(size_t)t * inner + head * P + c0 + c] = fmaf(Dh, x, sum);
    }
  }
  if (to) {
#pragma unroll
    for (int c = 0; c < 4; ++c)
#pragma unroll
      for (int m = 0; m < 4; ++m)
        if (lane + 32 * m < N) to[(size_t)(c0 + c) * N + lane + 32 * m] = S[c][m];
  }
}

// Few tokens of columns from_col .. to_col - 1 of a head, by a warp, COUNT columns at a time.
template <int COUNT> __device__ __noinline__ void walk_short(const Params& p, int head, int from_col, int to_col, float* state, int t_from, int t_end) {
  const int lane = threadIdx.x & 31, N = p.N, P = p.P, inner = p.heads * P, width = inner + 2 * p.groups * N;
  const float A = expf(p.A_log[head]), bias = p.dt_bias[head], Dh = p.D[head];
  const int g = head / (p.heads / p.groups);
  for (int c0 = from_col; c0 < to_col; c0 += COUNT) {
    float S[COUNT][4];
#pragma unroll
    for (int c = 0; c < COUNT; ++c)
#pragma unroll
      for (int m = 0; m < 4; ++m) S[c][m] = lane + 32 * m < N ? state[(size_t)(c0 + c) * N + lane + 32 * m] : 0.f;
    for (int t = t_from; t < t_end; ++t) {
      const bf16* row = p.xbc + (size_t)t * width;
      const float dt = softplus(to_float(p.u[(size_t)t * p.u_stride + p.dt_col + head]) + bias), decay = expf(-A * dt);
      float B[4], C[4], sum[COUNT];
#pragma unroll
      for (int m = 0; m < 4; ++m) {
        const bool in = lane + 32 * m < N;
        B[m] = in ? to_float(row[inner + g * N + lane + 32 * m]) : 0.f;
        C[m] = in ? to_float(row[inner + (p.groups + g) * N + lane + 32 * m]) : 0.f;
      }
#pragma unroll
      for (int c = 0; c < COUNT; ++c) {
        const float dtx = dt * to_float(row[head * P + c0 + c]);
        sum[c] = 0.f;
#pragma unroll
        for (int m = 0; m < 4; ++m)
          if (lane + 32 * m < N) {  // (0 times an infinity of a number that is not there must not get through)
            S[c][m] = fmaf(decay, S[c][m], B[m] * dtx);
            sum[c] = fmaf(S[c][m], C[m], sum[c]);
          }
      }
      sum_over_lanes<COUNT>(sum, lane);
      const int c = head * P + c0 + lane / (32 / COUNT);
      if (lane % (32 / COUNT) == 0) p.y[(size_t)t * inner + c] = fmaf(Dh, to_float(row[c]), sum[0]);
    }
#pragma unroll
    for (int c = 0; c < COUNT; ++c)
#pragma unroll
      for (int m = 0; m < 4; ++m)
        if (lane + 32 * m < N) state[(size_t)(c0 + c) * N + lane + 32 * m] = S[c][m];
  }
}

// SECOND: the second of the two launches over segments.
template <int NB, bool SECOND>
__global__ void __launch_bounds__(THREADS, 1) ssm_umma_kernel(const __grid_constant__ CUtensorMap map, const __grid_constant__ CUtensorMap map_y, const __grid_constant__ Params p) {
  pdl_launch_dependents();
  using Z = Shape<NB>;
  extern __shared__ unsigned char smem_raw[];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  pdl_wait();
  const int launched = p.segments > 1 ? p.segments - 1 : 1;
  const int z = blockIdx.z / launched, seq = p.num_seqs - 1 - z;  // single tokens come first in a step: the long portions start first
  const int seg = blockIdx.z - z * launched + (SECOND ? 1 : 0), head = blockIdx.y;
  const int first = p.q_start[seq], last = p.q_start[seq + 1];
  int from, to;
  segment_tiles((last - first + TOKENS - 1) / TOKENS, p.segments, seg, from, to);
  const int t0 = first + from * TOKENS, t1 = min(last, first + to * TOKENS);
  if (t1 <= t0) return;
  const bool emit = SECOND || seg == 0;   // with read-outs
  if (!emit && t1 == last) return;        // nothing starts behind the last segment
  const int N = p.N, P = p.P, inner = p.heads * P;
  const int g = head / (p.heads / p.groups), col0 = blockIdx.x * COLS;
  const size_t block = (size_t)P * N;
  float* slot_state = p.state + ((size_t)p.state_slot[seq] * p.heads + head) * block;
  if (last - first <= SHORT) {  // (one tile, so it is segment 0)
    if (head & ((1 << p.short_shift) - 1)) return;
    const int columns = 4 << p.short_shift, more = warp >> (4 - p.short_shift), from_col = col0 + (warp & ((WARPS >> p.short_shift) - 1)) * columns;
    if (warp < WARPS && head + more < p.heads) {  // (P is a multiple of 8)
      if (columns == 4) walk_short<4>(p, head + more, from_col, min(P, from_col + 4), slot_state + more * block, t0, t1);
      else walk_short<8>(p, head + more, from_col, min(P, from_col + columns), slot_state + more * block, t0, t1);
    }
    return;
  }

  unsigned char* smem = (unsigned char*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  const uint32_t sm = smem_u32(smem);
  float* tables = reinterpret_cast<float*>(smem + Z::TABLES);
  const uint32_t bars = sm + Z::BARS;
  // cb_full, x_full[2], wx_ready, w_ready, y_read, g_done, d_done, y_done, tab_full[2], tile_done[2], tab_done[2], s_ready, yb_done
  const uint32_t cb_full = bars, x_full = bars + 8, wx_ready = bars + 24, w_ready = bars + 32, y_read = bars + 40, g_done = bars + 48, d_done = bars + 56,
                 y_done = bars + 64, tab_full = bars + 72, tile_done = bars + 88, tab_done = bars + 104, s_ready = bars + 120, yb_done = bars + 128;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(smem + Z::BARS + 136);
  volatile int* failed = reinterpret_cast<volatile int*>(smem + Z::BARS + 140);
  if (tid == 0) {
    bar_init(cb_full, 1);
    bar_init(x_full, 1); bar_init(x_full + 8, 1);
    bar_init(wx_ready, WARPS); bar_init(w_ready, WARPS); bar_init(y_read, WARPS);
    bar_init(s_ready, WARPS); bar_init(yb_done, 1);
    bar_init(g_done, 1); bar_init(d_done, 1); bar_init(y_done, 1);
    bar_init(tab_full, 1); bar_init(tab_full + 8, 1);
    bar_init(tile_done, WARPS); bar_init(tile_done + 8, WARPS);
    bar_init(tab_done, WARPS); bar_init(tab_done + 8, WARPS);
    *failed = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == WARPS) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)), "r"(T_ALL) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  tmem_before();
  __syncthreads();
  tmem_after();
  const uint32_t tmem = *tmem_slot;
  const int tiles = (t1 - t0 + TOKENS - 1) / TOKENS;
  auto pbase = [&](int slot) { return (((size_t)seq * launched + slot) * p.heads + head); };
  float fin = 0.f;  // 0 while every result was finite, NaN from the first one on that was not
  float S[16];
  const int quad = warp & 3, cg = (warp >> 2) & 3, row = quad * 32 + lane;  // this thread's row, and which sixteen columns
  auto each_state = [&](auto&& fn) {  // fn(number e of S, its offset in a [P][N] block) for those that exist
    if (row < N) {
#pragma unroll
      for (int e = 0; e < 16; ++e) {
        const int c = col0 + cg * 16 + e;
        if (c < P) fn(e, (size_t)c * N + row);
      }
    }
  };

  if (warp == WARPS) {
    // ---- products
    const uint32_t one = elect_one();
    const int k16 = N / 16;
    unsigned left = p.wait_limit;
    auto wait = [&](uint32_t bar, uint32_t parity, int code) { bar_wait(bar, parity, left, failed, p.error_flag, code); };
    const uint64_t c_desc = operand(sm + Z::C), b_desc = operand(sm + Z::B), bt_desc = operand(sm + Z::B, SLAB), wx_desc = operand(sm + Z::WX), s0_desc = operand(sm + Z::S0),
                   x_desc = operand(sm + Z::X);  // (a descriptor counts 16 bytes)
    const uint32_t tm = __shfl_sync(0xffffffffu, tmem, 0);
    for (int i = 0; i < tiles && left > 1; ++i) {
      const uint32_t parity = i & 1;
      wait(cb_full, parity, 1);
      if (emit) {
        if (i > 0) wait(y_read, parity ^ 1, 2);
        tmem_after();
        const uint32_t idesc = instruction(TOKENS, false, false);
#pragma unroll 1
        for (int k = 0; k < k16; ++k) {  // the second half of n goes to an accumulator of its own
          const bool half = 2 * k >= k16;
          const uint32_t at = ((k >> 2) * SLAB + (k & 3) * 32) >> 4;
          product(one, tm + T_G + (half ? TOKENS : 0), c_desc + at, b_desc + at, idesc, !(k == 0 || (half && 2 * (k - 1) < k16)));
        }
        commit(one, g_done);
      }
      wait(wx_ready, parity, 3);
      tmem_after();
      {
        const uint32_t idesc = instruction(COLS, true, true);
#pragma unroll 1
        for (int s = 2; s >= 0; --s) {
          const uint64_t terms = wx_desc + (uint32_t)((s * SLAB) >> 4);
#pragma unroll
          for (int k = 0; k < TOKENS / 16; ++k) product(one, tm + T_DS, bt_desc + ((k * 2048) >> 4), terms + ((k * 2048) >> 4), idesc, s < 2 || k > 0);
        }
      }
      commit(one, d_done);
      if (!emit) continue;
      const uint32_t idesc = instruction(COLS, false, true);
      wait(s_ready, parity, 4);
#pragma unroll 1
      for (int s = 2; s >= 0; --s) {
        const uint64_t terms = s0_desc + (uint32_t)((s * Z::S_TERM) >> 4);
#pragma unroll
        for (int k = 0; k < NB * 4; ++k)
          if (k < k16) {
            const bool half = s == 0 && 2 * k >= k16;
            product(one, tm + T_YB + (half ? COLS : 0), c_desc + (((k >> 2) * SLAB + (k & 3) * 32) >> 4), terms + ((k * 2048) >> 4), idesc,
                    !((s == 2 && k == 0) || (half && 2 * (k - 1) < k16)));
          }
      }
      commit(one, yb_done);
      wait(x_full + 8 * parity, (i >> 1) & 1, 5);
      wait(w_ready, parity, 6);
      tmem_after();
      const uint64_t x_at = x_desc + ((parity * SLAB) >> 4);
#pragma unroll 1
      for (int s = 2; s >= 0; --s) {
        const uint32_t terms = tm + T_G + (s == 1 ? TOKENS : 0) + (s == 2 ? 8 : 0);
#pragma unroll
        for (int k = 0; k < TOKENS / 16; ++k) {
          const bool half = s == 0 && k >= TOKENS / 32;
          product_tmem(one, tm + T_YA + (half ? COLS : 0), terms + k * 16, x_at + ((k * 2048) >> 4), idesc, !((s == 2 && k == 0) || (half && k == TOKENS / 32)));
        }
      }
      commit(one, y_done);
    }
    __syncwarp();
  } else if (warp == WARPS + 2) {
    // ---- copies
    const uint32_t one = elect_one();
    unsigned left = p.wait_limit;
    auto wait = [&](uint32_t bar, uint32_t parity, int code) { bar_wait(bar, parity, left, failed, p.error_flag, code); };
    int xs = 0, cbs = 0;  // copies asked for
    for (int i = 0; i < tiles; ++i) {
      if (i >= 2) wait(tile_done + 8 * (i & 1), ((i - 2) >> 1) & 1, 7);  // the tile before the last one has left its buffer of x
      if (left == 1) break;
      if (one) {
        bar_expect(x_full + 8 * (i & 1), SLAB);
        tma_load(sm + Z::X + (i & 1) * SLAB, &map, head * P + col0, t0 + i * TOKENS, x_full + 8 * (i & 1));
      }
      ++xs;
      if (i >= 1) wait(emit ? yb_done : d_done, (i - 1) & 1, 8);  // C and B have been read
      if (left == 1 || *failed) break;
      if (one) {
        bar_expect(cb_full, (emit ? 2 : 1) * NB * SLAB);
#pragma unroll
        for (int b = 0; b < NB && i != p.skip_tile; ++b) {
          tma_load(sm + Z::B + b * SLAB, &map, inner + g * N + b * 64, t0 + i * TOKENS, cb_full);
          if (emit) tma_load(sm + Z::C + b * SLAB, &map, inner + (p.groups + g) * N + b * 64, t0 + i * TOKENS, cb_full);
        }
      }
      ++cbs;
    }
    if (*failed) {  // what is still on its way lands here, not in the next CTA's shared memory
      for (unsigned i = 0; cbs > 0 && i < p.wait_limit && !bar_done(cb_full, (cbs - 1) & 1); ++i) {}
      for (int b = 0; b < 2 && b < xs; ++b)
        for (unsigned i = 0; i < p.wait_limit && !bar_done(x_full + 8 * ((xs - 1 - b) & 1), ((xs - 1 - b) >> 1) & 1); ++i) {}
    }
  } else if (warp == WARPS + 1) {
    // ---- tables: four tokens a lane
    const float A = expf(p.A_log[head]), bias = p.dt_bias[head];
    unsigned left = p.wait_limit;
    double total = 0.0;
    float raw[4];
    auto load_raw = [&](int base) {
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        const int t = base + 4 * lane + k;
        raw[k] = t < t1 ? to_float(p.u[(size_t)t * p.u_stride + p.dt_col + head]) : 0.f;
      }
    };
    load_raw(t0);
    for (int i = 0; i < tiles; ++i) {
      const int base = t0 + i * TOKENS;
      float dt[4];
      double l[4];
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        const bool ok = base + 4 * lane + k < t1;
        dt[k] = ok ? softplus(raw[k] + bias) : 0.f;
        l[k] = ok ? (double)log_decay(-A * dt[k], LOG_FLOOR) : 0.0;
        if (k) l[k] += l[k - 1];
      }
      if (i + 1 < tiles) load_raw(base + TOKENS);
      double incl = l[3];
#pragma unroll
      for (int off = 1; off < 32; off <<= 1) {
        const double other = __shfl_up_sync(0xffffffffu, incl, off);
        if (lane >= off) incl += other;
      }
      const double before = incl - l[3], end = __shfl_sync(0xffffffffu, incl, 31), block_end = __shfl_sync(0xffffffffu, incl, lane | 7);
      if (i >= 2) bar_wait(tab_done + 8 * (i & 1), ((i - 2) >> 1) & 1, left, failed, p.error_flag, 9);
      float* tab = tables + (i & 1) * Table::FLOATS;
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        const double lt = before + l[k], l2 = lt * LOG2E;
        const float hi = (float)l2;
        const int t = 4 * lane + k;
        tab[Table::HI + t] = hi;
        tab[Table::LO + t] = (float)(l2 - (double)hi);
        tab[Table::DT + t] = dt[k];
        tab[Table::OUT + t] = expf((float)lt);
        tab[Table::IN + t] = expf((float)(end - lt)) * dt[k];
        tab[Table::BLOCK + t] = expf((float)(block_end - lt)) * dt[k];
      }
      if (lane == 0) tab[Table::END] = expf((float)end);
      total += end;
      __syncwarp();
      if (lane == 0) bar_arrive(tab_full + 8 * (i & 1));
    }
    if (!SECOND && t1 != last && lane == 0 && blockIdx.x == 0) p.part_log[pbase(seg)] = (float)total;
  } else {
    // ---- the sixteen warps
#pragma unroll
    for (int e = 0; e < 16; ++e) S[e] = 0.f;
    if (emit) {
      const float* src = SECOND ? p.part + pbase(0) * block : slot_state;
      each_state([&](int e, size_t at) { S[e] = src[at]; });
      if (SECOND) {
        for (int s = 1; s < seg; ++s) {
          const float keep = expf(p.part_log[pbase(s)]);
          const float* add = p.part + pbase(s) * block;
          each_state([&](int e, size_t at) { S[e] = fmaf(keep, S[e], add[at]); });
        }
      }
    }
    const float Dh = p.D[head];
    const uint32_t lanes = (uint32_t)(quad * 32) << 16;
    unsigned left = p.wait_limit;
    auto wait = [&](uint32_t bar, uint32_t parity, int code) { bar_wait(bar, parity, left, failed, p.error_flag, code); };
    const bool storer = cg == 0;  // the warp of a quarter of the rows that asks for their way out
    // The weighted values of tile i and the state at its start, in three terms (their readers of the tile before have ended: d_done).
    auto prepare = [&](int i) {
      const uint32_t tab = sm + Z::TABLES + (i & 1) * Table::FLOATS * 4;
      wait(tab_full + 8 * (i & 1), (i >> 1) & 1, 10);
      wait(x_full + 8 * (i & 1), (i >> 1) & 1, 11);
      const int r = tid >> 2, part = tid & 3;
      const float w = lds(tab + (Table::IN + r) * 4);
      float v[16];
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        uint32_t raw[4];
        ld_shared16(sm + Z::X + (i & 1) * SLAB + r * 128 + (((2 * part + h) ^ (r & 7)) << 4), raw);
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          const float2 x = unpack2(raw[e]);
          v[8 * h + 2 * e] = x.x * w;
          v[8 * h + 2 * e + 1] = x.y * w;
        }
      }
      store_terms(sm + Z::WX, SLAB, r, part, v);
      asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
      tmem_before();
      __syncwarp();
      if (lane == 0) bar_arrive(wx_ready);
      if (emit) {
        if (i > 0) wait(yb_done, (i - 1) & 1, 16);  // the state of the tile before has been read
        if (row < NB * 64) store_terms(sm + Z::S0, Z::S_TERM, row, cg, S);
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        __syncwarp();
        if (lane == 0) bar_arrive(s_ready);
      }
    };
    prepare(0);
    for (int i = 0; i < tiles; ++i) {
      const uint32_t parity = i & 1;
      const int base = t0 + i * TOKENS, len = min(TOKENS, t1 - base);
      const uint32_t tab = sm + Z::TABLES + parity * Table::FLOATS * 4;
      const uint32_t sx = sm + Z::X + parity * SLAB;
      uint32_t raw[2][4];  // this thread's x
      if (emit) {
        // ---- the weighted scores of this row and 32 tokens j
        if (storer && i > 0) {  // the read-outs of the tile before have left shared memory
          asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");
          __syncwarp();
          if (lane == 0) bar_arrive(tile_done + 8 * (parity ^ 1));
        }
        const float th = lds(tab + (Table::HI + row) * 4), tl = lds(tab + (Table::LO + row) * 4);
        wait(g_done, parity, 12);
        tmem_after();
        auto scores = [&](auto&& weight) {  // weight(j): those of tokens j .. j + 3
#pragma unroll 1
          for (int m = 0; m < 2; ++m) {  // sixteen tokens; their terms go where their scores lay
            const uint32_t at = tmem + T_G + lanes + cg * 32 + m * 16;
            uint32_t a[2][8], b[2][8], low[4];
#pragma unroll
            for (int h = 0; h < 2; ++h) {
              tmem_ld8(at + h * 8, a[h]);
              tmem_ld8(at + TOKENS + h * 8, b[h]);
            }
#pragma unroll
            for (int h = 0; h < 2; ++h) {
              const float4 f0 = weight(cg * 32 + m * 16 + h * 8), f1 = weight(cg * 32 + m * 16 + h * 8 + 4);
              if (h == 0) tmem_wait_ld();
              uint32_t w[3][4];
              const uint32_t (&g0)[8] = a[h], (&g1)[8] = b[h];
              dli::split3((__uint_as_float(g0[0]) + __uint_as_float(g1[0])) * f0.x, (__uint_as_float(g0[1]) + __uint_as_float(g1[1])) * f0.y, w[0][0], w[1][0], w[2][0]);
              dli::split3((__uint_as_float(g0[2]) + __uint_as_float(g1[2])) * f0.z, (__uint_as_float(g0[3]) + __uint_as_float(g1[3])) * f0.w, w[0][1], w[1][1], w[2][1]);
              dli::split3((__uint_as_float(g0[4]) + __uint_as_float(g1[4])) * f1.x, (__uint_as_float(g0[5]) + __uint_as_float(g1[5])) * f1.y, w[0][2], w[1][2], w[2][2]);
              dli::split3((__uint_as_float(g0[6]) + __uint_as_float(g1[6])) * f1.z, (__uint_as_float(g0[7]) + __uint_as_float(g1[7])) * f1.w, w[0][3], w[1][3], w[2][3]);
              tmem_st4(at + h * 4, w[0]);
              tmem_st4(at + TOKENS + h * 4, w[1]);
              if (h) {
                tmem_st4(at + 8, low);
                tmem_st4(at + 12, w[2]);
              } else {
#pragma unroll
                for (int e = 0; e < 4; ++e) low[e] = w[2][e];
              }
            }
          }
        };
        if (cg < quad) {  // a block below the diagonal: its decays are those of the row behind the block times those of the column up to its end
          const float behind = ex2((th - lds(tab + (Table::HI + cg * 32 + 31) * 4)) + (tl - lds(tab + (Table::LO + cg * 32 + 31) * 4)));
          scores([&](int j) {
            const float4 f = lds4(tab + (Table::BLOCK + j) * 4);
            return make_float4(f.x * behind, f.y * behind, f.z * behind, f.w * behind);
          });
        } else if (cg == quad) {
          scores([&](int j) {
            const float4 jh = lds4(tab + (Table::HI + j) * 4), jl = lds4(tab + (Table::LO + j) * 4), jd = lds4(tab + (Table::DT + j) * 4);
            return make_float4(j <= row ? ex2((th - jh.x) + (tl - jl.x)) * jd.x : 0.f, j + 1 <= row ? ex2((th - jh.y) + (tl - jl.y)) * jd.y : 0.f,
                               j + 2 <= row ? ex2((th - jh.z) + (tl - jl.z)) * jd.z : 0.f, j + 3 <= row ? ex2((th - jh.w) + (tl - jl.w)) * jd.w : 0.f);
          });
        } else {
          uint32_t none[16];
#pragma unroll
          for (int e = 0; e < 16; ++e) none[e] = 0;
#pragma unroll
          for (int e = 0; e < 2; ++e) {
            tmem_st16(tmem + T_G + lanes + cg * 32 + e * 16, none);
            tmem_st16(tmem + T_G + TOKENS + lanes + cg * 32 + e * 16, none);
          }
        }
        asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
      }
      // ---- the state at the tile's end (what is added to it lies where half of Ya goes)
      const float out = lds(tab + (Table::OUT + row) * 4);
      wait(d_done, parity, 13);
      tmem_after();
      {
        uint32_t a[16];
        tmem_ld16(tmem + T_DS + lanes + cg * 16, a);
        const float end = lds(tab + Table::END * 4);
        tmem_wait_ld();
        tmem_before();
        __syncwarp();
        if (emit && lane == 0) bar_arrive(w_ready);
#pragma unroll
        for (int e = 0; e < 16; ++e) S[e] = fmaf(end, S[e], __uint_as_float(a[e]));
      }
      if (emit) {
#pragma unroll
        for (int h = 0; h < 2; ++h) ld_shared16(sx + row * 128 + (((2 * cg + h) ^ (row & 7)) << 4), raw[h]);
      }
      __syncwarp();
      if (lane == 0) bar_arrive(tab_done + 8 * parity);
      if (i + 1 < tiles) prepare(i + 1);  // while Ya is made
      if (emit) {
        // ---- the read-outs
        wait(y_done, parity, 14);
        tmem_after();
        float v[16];
        {
          uint32_t a[16], b[16];
          tmem_ld16(tmem + T_YB + lanes + cg * 16, a);
          tmem_ld16(tmem + T_YB + COLS + lanes + cg * 16, b);
          tmem_wait_ld();
#pragma unroll
          for (int e = 0; e < 16; ++e) v[e] = (__uint_as_float(a[e]) + __uint_as_float(b[e])) * out;
          tmem_ld16(tmem + T_YA + lanes + cg * 16, a);
          tmem_ld16(tmem + T_YA + COLS + lanes + cg * 16, b);
          tmem_wait_ld();
#pragma unroll
          for (int e = 0; e < 16; ++e) v[e] += __uint_as_float(a[e]) + __uint_as_float(b[e]);
        }
        tmem_before();
        __syncwarp();
        if (lane == 0) bar_arrive(y_read);
        const int there = P - col0 - cg * 16;  // (a multiple of 8)
#pragma unroll
        for (int h = 0; h < 2; ++h) {
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            const float2 x = unpack2(raw[h][e]);
            v[8 * h + 2 * e] = fmaf(Dh, x.x, v[8 * h + 2 * e]);
            v[8 * h + 2 * e + 1] = fmaf(Dh, x.y, v[8 * h + 2 * e + 1]);
          }
          if (row < len && 8 * h < there) {
#pragma unroll
            for (int e = 0; e < 8; ++e) fin = fmaf(v[8 * h + e], 0.f, fin);
          }
        }
        // through shared memory (columns 32 .. in the place of the tile's x, which nobody needs any more), and from there in copies of 32 rows: stores of a
        // row a thread took 3,300 clocks a tile, and the next fence waited for them
        asm volatile("bar.sync %0, 128;" ::"r"(1 + quad) : "memory");
        const uint32_t half = cg < 2 ? sm + Z::Y : sx;
#pragma unroll
        for (int e = 0; e < 4; ++e)
          st_shared16(half + row * 128 + (((4 * (cg & 1) + e) ^ (row & 7)) << 4), __float_as_uint(v[4 * e]), __float_as_uint(v[4 * e + 1]), __float_as_uint(v[4 * e + 2]),
                      __float_as_uint(v[4 * e + 3]));
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        asm volatile("bar.sync %0, 128;" ::"r"(1 + quad) : "memory");
        const bool whole = p.y_vec && quad * 32 + 32 <= len, ok = left > 1 && !*failed;  // 32 rows of this sequence
        if (ok && whole && storer) {
          if (lane < 2 && P - col0 >= 32 * (lane + 1))
            asm volatile("cp.async.bulk.tensor.2d.global.shared::cta.bulk_group [%0, {%2, %3}], [%1];"
                         ::"l"(&map_y), "r"((lane ? sx : sm + Z::Y) + quad * 32 * 128), "r"(head * P + col0 + 32 * lane), "r"(base + quad * 32) : "memory");
          asm volatile("cp.async.bulk.commit_group;" ::: "memory");
        }
        // the ragged rest: rows of a last tile, columns of a last block
        const int c = (lane & 15) * 4;
        if (ok && c < P - col0 && (!whole || P - col0 < (c & 32) + 32)) {
          float* dst = p.y + (size_t)base * inner + head * P + col0 + c;
#pragma unroll
          for (int k = 0; k < 4; ++k) {
            const int r = quad * 32 + cg * 8 + k * 2 + (lane >> 4);
            if (r < len) {
              uint32_t o[4];
              ld_shared16((c < 32 ? sm + Z::Y : sx) + r * 128 + (((lane & 7) ^ (r & 7)) << 4), o);
              float* at = dst + (size_t)r * inner;
              if (p.y_vec) {
                *reinterpret_cast<float4*>(at) = make_float4(__uint_as_float(o[0]), __uint_as_float(o[1]), __uint_as_float(o[2]), __uint_as_float(o[3]));
              } else {
                *reinterpret_cast<float2*>(at) = make_float2(__uint_as_float(o[0]), __uint_as_float(o[1]));
                *reinterpret_cast<float2*>(at + 2) = make_float2(__uint_as_float(o[2]), __uint_as_float(o[3]));
              }
            }
          }
        }
      }
      __syncwarp();
      if (lane == 0 && !(emit && storer)) bar_arrive(tile_done + 8 * parity);
    }
    asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");  // (walk_again writes behind these)
  }
  float* dst = t1 == last ? slot_state : (SECOND ? nullptr : p.part + pbase(seg) * block);
  if (warp < WARPS && emit && dst) each_state([&](int e, size_t) { fin = fmaf(S[e], 0.f, fin); });
  const bool again = __syncthreads_or(emit && fin != 0.f);  // (also: nobody writes a read-out behind this)
  if (warp == WARPS) {
    tmem_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(T_ALL) : "memory");
  }
  if (*failed) return;
  if (again) {
    int second = 0, end = 0;  // segments behind the first start again from the state behind it, the last one that was walked from the slot's
    if (SECOND) segment_tiles((last - first + TOKENS - 1) / TOKENS, p.segments, 1, second, end);
    walk_again(p, head, col0, SECOND ? p.part + pbase(0) * block : slot_state, first + second * TOKENS, t0, t1, dst);
  } else if (dst && warp < WARPS) {
    each_state([&](int e, size_t at) { dst[at] = S[e]; });
  }
}

inline int column_blocks(int P) { return (P + COLS - 1) / COLS; }

int* error_flag_device = nullptr;
int* error_flag_host = nullptr;

// as many as leave every SM about one CTA of short sequences
inline int short_shift(long long units) {
  int s = 0;
  while (s < 3 && units > ((long long)sm_count() << s) * 3 / 2) ++s;
  return s;
}

template <int NB>
int launch(const CUtensorMap& map, const CUtensorMap& map_y, const Params& p, cudaStream_t stream) {
  static OncePerDevice configured;
  if (!configured.here()) {
    cudaError_t e = cudaFuncSetAttribute(ssm_umma_kernel<NB, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, Shape<NB>::SMEM);
    if (e == cudaSuccess) e = cudaFuncSetAttribute(ssm_umma_kernel<NB, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, Shape<NB>::SMEM);
    if (e != cudaSuccess) return (int)e;
    configured.here() = true;
  }
  const dim3 grid(column_blocks(p.P), p.heads, p.num_seqs * (p.segments > 1 ? p.segments - 1 : 1)), block(THREADS);
  cudaError_t e = launch_pdl((ssm_umma_kernel<NB, false>), grid, block, (size_t)Shape<NB>::SMEM, stream, 1, map, map_y, p);
  if (e == cudaSuccess && p.segments > 1) e = launch_pdl((ssm_umma_kernel<NB, true>), grid, block, (size_t)Shape<NB>::SMEM, stream, 1, map, map_y, p);
  return (int)e;
}

}  // namespace

// Into how many segments the sequences of a step are cut: a launch (of one segment fewer) gives every SM a CTA, and behind the first there is at most one for every
// four tiles of the longest sequence: those have about four tiles or more, the last of them what is left, and the first what they leave, often one (segment_tiles).  Two segments would follow one another: three is the fewest that gain.  Measured (us at segments 1 / 3 / 4 / 5, 64 heads, P 64, N 128): one
// prompt of 4,096 tokens 143 / 108 / 144 / 130 (four and five: more CTAs than SMs), of 600 28 / 32 / 27 / 27; three prompts (192 CTAs of one segment) 73 / 104.
DLI_EXPORT int dli_ssm_umma_segments(int num_seqs, int heads, int P, int max_len) {
  const long long units = (long long)column_blocks(P) * heads * (num_seqs > 0 ? num_seqs : 1);
  long long fill = sm_count() / (units > 0 ? units : 1);
  const int most = (max_len + TOKENS - 1) / TOKENS / 4;
  if (fill > most) fill = most;
  return fill < 2 ? 1 : (fill > 32 ? 33 : (int)fill + 1);
}

static int run(float* y, const void* xbc, const void* u, long long u_stride, int dt_col, const float* dt_bias, const float* A_log, const float* D, float* state,
               const int* q_start, const int* state_slot, int n, int num_seqs, int heads, int P, int N, int groups, int segments, float* part, float* part_log,
               unsigned wait_limit, int skip_tile, cudaStream_t stream) {
  if (num_seqs == 0 || n == 0) return 0;
  if (n < 0 || heads < 1 || heads > 65535 || groups < 1 || heads % groups || P < 8 || P % 8 || N < 32 || N % 16 || N > 128 || segments < 1 ||
      (long long)num_seqs * segments > 65535 || ((uintptr_t)xbc & 15) || ((uintptr_t)y & 7) || ((uintptr_t)state & 7) || (segments > 1 && (!part || !part_log)))
    return DLI_ERR_UNSUPPORTED;
  if (!error_flag_host) {
    if (cudaHostAlloc((void**)&error_flag_host, sizeof(int), cudaHostAllocMapped) != cudaSuccess) return (int)cudaGetLastError();
    *error_flag_host = 0;
    if (cudaHostGetDevicePointer((void**)&error_flag_device, error_flag_host, 0) != cudaSuccess) return (int)cudaGetLastError();
  }
  const int width = heads * P + 2 * groups * N, y_vec = ((uintptr_t)y & 15) == 0;
  CUtensorMap map, map_y;
  if (!make_map(&map, xbc, false, n, width, width, TOKENS)) return DLI_ERR_UNSUPPORTED;
  map_y = map;  // (not used where y is not aligned)
  if (y_vec && !make_map(&map_y, y, true, n, (long long)heads * P, (long long)heads * P, 32)) return DLI_ERR_UNSUPPORTED;
  Params p;
  p.y = y; p.xbc = (const bf16*)xbc; p.u = (const bf16*)u; p.u_stride = u_stride; p.dt_col = dt_col; p.dt_bias = dt_bias; p.A_log = A_log; p.D = D;
  p.state = state; p.q_start = q_start; p.state_slot = state_slot; p.num_seqs = num_seqs; p.heads = heads; p.P = P; p.N = N; p.groups = groups;
  p.segments = segments; p.part = part; p.part_log = part_log; p.y_vec = y_vec; p.short_shift = short_shift((long long)column_blocks(P) * heads * num_seqs); p.error_flag = error_flag_device;
  p.wait_limit = wait_limit; p.skip_tile = skip_tile;
  return N <= 64 ? launch<1>(map, map_y, p, stream) : launch<2>(map, map_y, p, stream);
}

// n: rows of xbc.  segments > 1: part [num_seqs (segments - 1) heads P N] and part_log [num_seqs (segments - 1) heads] are scratch.
DLI_EXPORT int dli_ssm_umma(float* y, const void* xbc, const void* u, long long u_stride, int dt_col, const float* dt_bias, const float* A_log, const float* D,
                            float* state, const int* q_start, const int* state_slot, int n, int num_seqs, int heads, int P, int N, int groups, int segments,
                            float* part, float* part_log, cudaStream_t stream) {
  return run(y, xbc, u, u_stride, dt_col, dt_bias, A_log, D, state, q_start, state_slot, n, num_seqs, heads, P, N, groups, segments, part, part_log, WAIT_LIMIT, -1, stream);
}

// For tests: in one segment, with every CTA's copies of B and C of tile `skip_tile` left out and every wait given up after `wait_limit` polls.
DLI_EXPORT int dli_ssm_umma_wait_test(float* y, const void* xbc, const void* u, long long u_stride, int dt_col, const float* dt_bias, const float* A_log, const float* D,
                                      float* state, const int* q_start, const int* state_slot, int n, int num_seqs, int heads, int P, int N, int groups,
                                      unsigned wait_limit, int skip_tile, cudaStream_t stream) {
  if (wait_limit < 2 || wait_limit > WAIT_LIMIT || skip_tile < 0) return DLI_ERR_UNSUPPORTED;
  return run(y, xbc, u, u_stride, dt_col, dt_bias, A_log, D, state, q_start, state_slot, n, num_seqs, heads, P, N, groups, 1, nullptr, nullptr, wait_limit, skip_tile, stream);
}

// 0, or the code of the first wait that ran out since the library was loaded or the code was last cleared
DLI_EXPORT int dli_ssm_umma_error() { return error_flag_host ? *error_flag_host : 0; }
DLI_EXPORT int dli_ssm_umma_clear_error() { if (error_flag_host) *error_flag_host = 0; return 0; }
