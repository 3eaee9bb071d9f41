// The matrix memory with exponential gates (matrix_memory.cu says what is computed) for prompt portions in bfloat16: tiles of 128 tokens in closed form on
// tcgen05.  Inside a tile that starts from (S0, n0, m0), with b_t the sum of the log forget gates up to t, a_j = i_j - b_j and g_t = max(m0, max_{j <= t} a_j),
// the running maximum is m_t = b_t + g_t, and the tile's read-outs and end are
//   exp(m0 - g_t) q_t S0 + sum_{j <= t} exp(a_j - g_t) (q_t . k_j) v_j,      exp(m0 - g_C) S0 + sum_j exp(a_j - g_C) k_j v_j^T.
//
// q, k and v are bfloat16 as the projection left them; gates, weights, state and every sum are float32 (the gates' sums and maxima double, kept as two
// floats), and nothing float32 is rounded on its way into a product: three bfloat16 terms.
//
// The kernel is that of the selective scan (ssm_umma.cu says how a tile goes): C, B and x are q, k and v here, a CTA owns 64 value columns of one head of one
// sequence.  Besides, the CTAs of the first 64 columns keep n (a value column of ones): its share of a read-out is a plain dot product of q's row with n0, a
// tile's own the sum of a row's weighted scores, and what a tile adds to it is summed on the CUDA cores too.
//
// Segments, and numbers that are not finite: as there.  A state is added to another by  m' = max(m + B, m_L),  S <- exp(m + B - m') S + exp(m_L - m') L, with L
// what a segment adds to a state from nothing, m_L its maximum, B the sum of its log forget gates.
//
// Measured, us, against tiles of 64 tokens by mma.sync (matrix_memory_tc.cu, every warp with scores of its own; heads of 128): 16 heads, a prompt of 600 tokens
// 77 -> 38, beside seven single tokens 93 -> 38, of 800 and 1,003 114 -> 57, of 4,096 216 -> 107, of 100 18 -> 13; 32 heads, one of 1,500 150 -> 72, 24 single tokens
// beside 300 109 -> 57.  A tile takes 6.1 us where n goes along, 4.4 elsewhere.  Errors against 64 bits (mean of six seeds, 200 tokens): o 2.9e-7, S 3.1e-7, o over its
// divisor 3.9e-7 (before 5.4e-7, 5.7e-7 and 8.3e-7).
//
// Every wait is bounded: after `wait_limit` polls a code goes to *error_flag, and the CTA goes on to its end without another wait; from then on it stores no read-outs, and
// states and maxima not at all.
#include "matrix_memory.cuh"
#include <math_constants.h>
#include "umma_tiles.cuh"

using namespace dli;
using namespace dli::umma;
typedef __nv_bfloat16 bf16;

namespace {

constexpr int TOKENS = 128;  // of a tile
constexpr int COLS = 64;     // columns p of a CTA
constexpr int WARPS = 16;
constexpr int THREADS = (WARPS + 3) * 32;
constexpr double LOG2E = 1.4426950408889634074;
constexpr int SHORT = 4;  // sequences of up to so many tokens are walked

struct Params {
  float* o;               // [n][heads dv]
  float* divisor;         // [n][heads]
  const bf16* u;          // rows: q | k | v
  long long u_stride;
  const float* gates;     // [n][2 heads]
  const float* bias;      // [2 heads]
  float cap;
  float* state;           // [slots][heads][dv + 1][d]
  float* top;             // [slots][heads][dv + 1]
  const int *q_start, *state_slot;
  int num_seqs, heads, d, dv;
  int segments;           // of a sequence; with more than one:
  float* part;            // [seqs][segments - 1][heads][dv + 1][d]: the state behind segment 0, then what each segment adds
  float* part_m;          // [seqs][segments - 1][heads][2]: its maximum, the sum of its log forget gates
  int short_shift;        // heads of a short sequence that a CTA walks, as a power of two (as in ssm_umma.cu)
  int o_vec;              // read-outs lie on 16-byte boundaries
  int* error_flag;
  unsigned wait_limit;
  int skip_tile;          // -1 in every launch of the engine: the tile of every CTA whose copies of q and k a test leaves out
};

// Per tile, floats: g_t and a_j in log2 units (two terms each) | exp(m0 - g_t) | exp(a_j - g_C) | exp(a_j - A) with A the largest a of the block of 32 | exp(-m_t) |
// the blocks' A (two terms), and exp(m0 - g_C)
struct Table {
  static constexpr int GH = 0, GL = TOKENS, AH = 2 * TOKENS, AL = 3 * TOKENS, OUT = 4 * TOKENS, IN = 5 * TOKENS, BLOCK = 6 * TOKENS, FLOOR = 7 * TOKENS,
                       TOP = 8 * TOKENS, END = TOP + 8, FLOATS = END + 4;
};

template <int NB> struct Shape {  // NB: the key size in slabs of 64
  static constexpr int C = 0, B = NB * SLAB, X = 2 * NB * SLAB, WX = X + 2 * SLAB, S0 = WX + 3 * SLAB, S_TERM = NB * 64 * 128;
  static constexpr int Y = S0 + 3 * S_TERM;  // columns 0..31 of the read-outs on their way out; the others lie where the tile's v lay
  static constexpr int TABLES = Y + SLAB, NS = TABLES + 2 * Table::FLOATS * 4, SHARES = NS + 2 * TOKENS * 4, BARS = SHARES + 8 * TOKENS * 4, SMEM = BARS + 192 + 1024;
  static_assert(SMEM <= 227 * 1024, "shared memory");
};
// Columns of tensor memory
constexpr int T_G = 0, T_YB = 256, T_YA = 384, T_DS = 448, T_ALL = 512;

// Token range of segment `seg` of a sequence of `tiles` tiles: segment 0 has what the others' even shares leave (a segment without read-outs costs
// 0.45 of one with).
__device__ __forceinline__ void segment_tiles(int tiles, int segments, int seg, int& from, int& to) {
  if (segments == 1) { from = 0; to = tiles; return; }
  const int rest = segments - 1, share = (20 * tiles + 20 * rest + 8) / (20 * rest + 9);
  const int head = max(1, tiles - share * rest);
  from = seg == 0 ? 0 : min(tiles, head + (seg - 1) * share);
  to = min(tiles, head + seg * share);
}

// Columns from_col .. to_col - 1 of a head (dv: n) token after token, COUNT at a time: from the state and maximum in front of token t_from, with read-outs of
// tokens t_emit .. t_end - 1, the state behind them to `to` and its maximum to top_to, a copy per column (or null).  A lane holds every 32nd key row.
template <int COUNT>
__device__ __noinline__ void walk_columns(const Params& p, int head, int from_col, int to_col, const float* from, float m_from, int t_from, int t_emit, int t_end,
                                          float* to, float* top_to) {
  const int lane = threadIdx.x & 31, d = p.d, dv = p.dv, heads = p.heads;
  const float bias_i = p.bias[head], bias_f = p.bias[heads + head], scale = 1.f / sqrtf((float)d);
  for (int c0 = from_col; c0 < to_col; c0 += COUNT) {
    float S[COUNT][4], m = m_from;
#pragma unroll
    for (int c = 0; c < COUNT; ++c)
#pragma unroll
      for (int e = 0; e < 4; ++e) S[c][e] = lane + 32 * e < d ? from[(size_t)(c0 + c) * d + lane + 32 * e] : 0.f;
    for (int t = t_from; t < t_end; ++t) {
      const bf16* row = p.u + (size_t)t * p.u_stride;
      const float li = memory_in_gate(p.gates[(size_t)t * 2 * heads + head] + bias_i, p.cap);
      const float lf = memory_forget_gate(p.gates[(size_t)t * 2 * heads + heads + head] + bias_f, p.cap);
      const float next = fmaxf(lf + m, li), keep = expf(lf + m - next), take = expf(li - next);
      m = next;
      float q[4], k[4], sum[COUNT];
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const bool in = lane + 32 * e < d;
        q[e] = in ? to_float(row[head * d + lane + 32 * e]) : 0.f;
        k[e] = in ? to_float(row[(heads + head) * d + lane + 32 * e]) : 0.f;
      }
#pragma unroll
      for (int c = 0; c < COUNT; ++c) {
        const float w = take * (COUNT > 1 ? to_float(row[2 * heads * d + head * dv + c0 + c]) : 1.f);
        sum[c] = 0.f;
#pragma unroll
        for (int e = 0; e < 4; ++e)
          if (lane + 32 * e < d) {  // (0 times an infinity of a number that is not there must not get through)
            S[c][e] = fmaf(keep, S[c][e], w * k[e]);
            sum[c] = fmaf(q[e], S[c][e], sum[c]);
          }
      }
      sum_over_lanes<COUNT>(sum, lane);
      if (lane % (32 / COUNT) == 0 && t >= t_emit) {
        const size_t at = (size_t)t * heads + head;
        if (COUNT > 1) p.o[at * dv + c0 + lane / (32 / COUNT)] = sum[0] * scale;
        else p.divisor[at] = memory_divisor(sum[0] * scale, m);
      }
    }
    if (to) {
#pragma unroll
      for (int c = 0; c < COUNT; ++c)
#pragma unroll
        for (int e = 0; e < 4; ++e)
          if (lane + 32 * e < d) to[(size_t)(c0 + c) * d + lane + 32 * e] = S[c][e];
      if (top_to && lane < COUNT) top_to[c0 + lane] = m;
    }
  }
}

// SECOND: the second of the two launches over segments.
template <int NB, bool SECOND>
__global__ void __launch_bounds__(THREADS, 1) matrix_memory_umma_kernel(const __grid_constant__ CUtensorMap map, const __grid_constant__ CUtensorMap map_o, const __grid_constant__ Params p) {
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
  const int N = p.d, P = p.dv, inner = p.heads * P, col0 = blockIdx.x * COLS;
  const bool with_n = blockIdx.x == 0;
  const size_t block = (size_t)(P + 1) * N;  // of a head's state
  const size_t slot = (size_t)p.state_slot[seq] * p.heads + head;
  float *slot_state = p.state + slot * block, *slot_top = p.top + slot * (P + 1);
  if (last - first <= SHORT) {  // (one tile, so it is segment 0)
    if (head & ((1 << p.short_shift) - 1)) return;
    const int columns = 4 << p.short_shift, more = warp >> (4 - p.short_shift), from_col = col0 + (warp & ((WARPS >> p.short_shift) - 1)) * columns;
    if (warp < WARPS && head + more < p.heads) {
      float *state = slot_state + more * block, *top = slot_top + more * (P + 1);  // (a warp reads the maximum's copy of its own columns)
      if (from_col < P) {  // (P is a multiple of 8)
        if (columns == 4) walk_columns<4>(p, head + more, from_col, min(P, from_col + 4), state, top[from_col], t0, t0, t1, state, top);
        else walk_columns<8>(p, head + more, from_col, min(P, from_col + columns), state, top[from_col], t0, t0, t1, state, top);
      }
      if (with_n && from_col == 0) walk_columns<1>(p, head + more, P, P + 1, state, top[P], t0, t0, t1, state, top);
    }
    return;
  }

  unsigned char* smem = (unsigned char*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  const uint32_t sm = smem_u32(smem);
  float* tables = reinterpret_cast<float*>(smem + Z::TABLES);
  float* shares = reinterpret_cast<float*>(smem + Z::SHARES);  // [4][TOKENS] of the divisors, [4][TOKENS] of n
  const uint32_t bars = sm + Z::BARS;
  // cb_full, x_full[2], wx_ready, w_ready, y_read, g_done, d_done, y_done, tab_full[2], tile_done[2], tab_done[2], s_ready, yb_done, qk_read
  const uint32_t cb_full = bars, x_full = bars + 8, wx_ready = bars + 24, w_ready = bars + 32, y_read = bars + 40, g_done = bars + 48, d_done = bars + 56,
                 y_done = bars + 64, tab_full = bars + 72, tile_done = bars + 88, tab_done = bars + 104, s_ready = bars + 120, yb_done = bars + 128, qk_read = bars + 136;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(smem + Z::BARS + 144);
  volatile int* failed = reinterpret_cast<volatile int*>(smem + Z::BARS + 148);
  float* first_top = reinterpret_cast<float*>(smem + Z::BARS + 152);  // the maximum where a second walk starts
  if (tid == 0) {
    bar_init(cb_full, 1);
    bar_init(x_full, 1); bar_init(x_full + 8, 1);
    bar_init(wx_ready, WARPS); bar_init(w_ready, WARPS); bar_init(y_read, WARPS);
    bar_init(s_ready, WARPS); bar_init(yb_done, 1); bar_init(qk_read, WARPS);
    bar_init(g_done, 1); bar_init(d_done, 1); bar_init(y_done, 1);
    bar_init(tab_full, 1); bar_init(tab_full + 8, 1);
    bar_init(tile_done, WARPS); bar_init(tile_done + 8, WARPS);
    bar_init(tab_done, WARPS); bar_init(tab_done + 8, WARPS);
    *failed = 0;
    *first_top = SECOND ? p.part_m[((size_t)seq * launched * p.heads + head) * 2] : slot_top[col0];  // (before anybody writes it)
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
  // The maximum in front of the first tile; fn(keep, take, slot) for every segment on the way there.  (The top of column col0: this CTA's own copy.)
  auto start_top = [&](auto&& fn) -> float {
    if (!emit) return -CUDART_INF_F;
    if (!SECOND) return slot_top[col0];
    float m = p.part_m[pbase(0) * 2];
    for (int s = 1; s < seg; ++s) {
      const float mb = m + p.part_m[pbase(s) * 2 + 1], ml = p.part_m[pbase(s) * 2], next = fmaxf(mb, ml);
      fn(expf(mb - next), expf(ml - next), s);
      m = next;
    }
    return m;
  };
  float fin = 0.f;  // 0 while every result was finite, NaN from the first one on that was not
  float S[16], S0_n = 0.f;  // .. and of n (warps 0..3)
  float m_end = 0.f, forgot_end = 0.f;  // (the warp of the tables) the maximum behind the last tile, the sum of the log forget gates
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
        tma_load(sm + Z::X + (i & 1) * SLAB, &map, 2 * p.heads * N + head * P + col0, t0 + i * TOKENS, x_full + 8 * (i & 1));
      }
      ++xs;
      if (i >= 1) {  // q and k have been read
        wait(emit ? yb_done : d_done, (i - 1) & 1, 8);
        if (with_n) wait(qk_read, (i - 1) & 1, 17);
      }
      if (left == 1 || *failed) break;
      if (one) {
        bar_expect(cb_full, (emit ? 2 : 1) * NB * SLAB);
#pragma unroll
        for (int b = 0; b < NB && i != p.skip_tile; ++b) {
          tma_load(sm + Z::B + b * SLAB, &map, (p.heads + head) * N + b * 64, t0 + i * TOKENS, cb_full);
          if (emit) tma_load(sm + Z::C + b * SLAB, &map, head * N + b * 64, t0 + i * TOKENS, cb_full);
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
    const float bias_i = p.bias[head], bias_f = p.bias[p.heads + head];
    unsigned left = p.wait_limit;
    double m0 = (double)start_top([](float, float, int) {}) * LOG2E, forgot = 0.0;  // (log2 units)
    float gi[4], gf[4];
    auto load_raw = [&](int base) {
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        const int t = base + 4 * lane + k;
        const float* g = p.gates + (size_t)(t < t1 ? t : t0) * 2 * p.heads + head;
        gi[k] = g[0];
        gf[k] = g[p.heads];
      }
    };
    load_raw(t0);
    for (int i = 0; i < tiles; ++i) {
      const int base = t0 + i * TOKENS;
      double b[4], a[4], g[4];
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        const bool ok = base + 4 * lane + k < t1;
        b[k] = ok ? (double)memory_forget_gate(gf[k] + bias_f, p.cap) * LOG2E : 0.0;
        a[k] = ok ? (double)memory_in_gate(gi[k] + bias_i, p.cap) * LOG2E : -(double)CUDART_INF_F;
        if (k) b[k] += b[k - 1];
      }
      if (i + 1 < tiles) load_raw(base + TOKENS);
      double incl = b[3];
#pragma unroll
      for (int off = 1; off < 32; off <<= 1) {
        const double other = __shfl_up_sync(0xffffffffu, incl, off);
        if (lane >= off) incl += other;
      }
      const double before = incl - b[3], b_end = __shfl_sync(0xffffffffu, incl, 31);
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        b[k] += before;
        a[k] -= b[k];
        g[k] = k ? fmax(g[k - 1], a[k]) : a[k];
      }
      double top = g[3];
#pragma unroll
      for (int off = 1; off < 32; off <<= 1) {
        const double other = __shfl_up_sync(0xffffffffu, top, off);
        if (lane >= off) top = fmax(top, other);
      }
      double block_top = g[3];  // of 32 tokens
#pragma unroll
      for (int off = 1; off < 8; off <<= 1) block_top = fmax(block_top, __shfl_xor_sync(0xffffffffu, block_top, off));
      double top_before = __shfl_up_sync(0xffffffffu, top, 1);
      top_before = lane == 0 ? m0 : fmax(m0, top_before);
      const double g_end = fmax(m0, __shfl_sync(0xffffffffu, top, 31));
      if (i >= 2) bar_wait(tab_done + 8 * (i & 1), ((i - 2) >> 1) & 1, left, failed, p.error_flag, 9);
      float* tab = tables + (i & 1) * Table::FLOATS;
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        const int t = 4 * lane + k;
        const double gt = fmax(top_before, g[k]);
        const float gh = (float)gt, ah = (float)a[k];
        const bool there = a[k] > -(double)CUDART_INF_F;  // (a NaN is not: its tile is walked)
        tab[Table::GH + t] = gh;
        tab[Table::GL + t] = (float)(gt - (double)gh);
        tab[Table::AH + t] = ah;
        tab[Table::AL + t] = there ? (float)(a[k] - (double)ah) : 0.f;
        tab[Table::OUT + t] = exp2f((float)(m0 - gt));
        tab[Table::IN + t] = exp2f((float)(a[k] - g_end));
        tab[Table::BLOCK + t] = there ? exp2f((float)(a[k] - block_top)) : (a[k] == a[k] ? 0.f : CUDART_NAN_F);
        tab[Table::FLOOR + t] = exp2f((float)-(b[k] + gt));
      }
      if ((lane & 7) == 0) {
        const float h = (float)block_top;
        tab[Table::TOP + (lane >> 3)] = h;
        tab[Table::TOP + 4 + (lane >> 3)] = block_top > -(double)CUDART_INF_F ? (float)(block_top - (double)h) : 0.f;
      }
      if (lane == 0) tab[Table::END] = exp2f((float)(m0 - g_end));
      m0 = b_end + g_end;
      forgot += b_end;
      __syncwarp();
      if (lane == 0) bar_arrive(tab_full + 8 * (i & 1));
    }
    m_end = (float)(m0 / LOG2E);
    forgot_end = (float)(forgot / LOG2E);
  } else {
    // ---- the sixteen warps
#pragma unroll
    for (int e = 0; e < 16; ++e) S[e] = 0.f;
    float n_own = 0.f;  // (warps 0..3 of the CTAs with n) its number of this row
    if (emit) {
      const float* src = SECOND ? p.part + pbase(0) * block : slot_state;
      each_state([&](int e, size_t at) { S[e] = src[at]; });
      if (with_n && cg == 0 && row < N) n_own = src[(size_t)P * N + row];
      start_top([&](float keep, float take, int s) {
        const float* add = p.part + pbase(s) * block;
        each_state([&](int e, size_t at) { S[e] = fmaf(keep, S[e], take * add[at]); });
        if (with_n && cg == 0 && row < N) n_own = fmaf(keep, n_own, take * add[(size_t)P * N + row]);
      });
    }
    const float scale = 1.f / sqrtf((float)N);
    const uint32_t lanes = (uint32_t)(quad * 32) << 16;
    unsigned left = p.wait_limit;
    auto wait = [&](uint32_t bar, uint32_t parity, int code) { bar_wait(bar, parity, left, failed, p.error_flag, code); };
    const bool storer = cg == 0;  // the warp of a quarter of the rows that asks for their way out
    // The weighted values of tile i, and the state at its start, in three terms (their readers of the tile before have ended: d_done, yb_done)
    auto prepare_values = [&](int i) {
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
    };
    auto prepare_state = [&](int i) {
      if (row < NB * 64) store_terms(sm + Z::S0, Z::S_TERM, row, cg, S);
      if (with_n && cg == 0) asm volatile("st.shared.f32 [%0], %1;" ::"r"(sm + Z::NS + ((i & 1) * TOKENS + row) * 4), "f"(n_own) : "memory");
      asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
      __syncwarp();
      if (lane == 0) bar_arrive(s_ready);
    };
    prepare_values(0);
    if (emit) prepare_state(0);
    for (int i = 0; i < tiles; ++i) {
      const uint32_t parity = i & 1;
      const int base = t0 + i * TOKENS, len = min(TOKENS, t1 - base);
      const uint32_t tab = sm + Z::TABLES + parity * Table::FLOATS * 4;
      const uint32_t sx = sm + Z::X + parity * SLAB;
      float scored = 0.f;  // the sum of this thread's weighted scores
      if (emit) {
        // ---- the weighted scores of this row and 32 tokens j
        if (storer && i > 0) {  // the read-outs of the tile before have left shared memory
          asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");
          __syncwarp();
          if (lane == 0) bar_arrive(tile_done + 8 * (parity ^ 1));
        }
        const float th = lds(tab + (Table::GH + row) * 4), tl = lds(tab + (Table::GL + row) * 4);
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
              float v[8] = {f0.x, f0.y, f0.z, f0.w, f1.x, f1.y, f1.z, f1.w};
#pragma unroll
              for (int e = 0; e < 8; ++e) {
                v[e] *= __uint_as_float(g0[e]) + __uint_as_float(g1[e]);
                if (with_n) scored += v[e];
              }
#pragma unroll
              for (int e = 0; e < 4; ++e) split3(v[2 * e], v[2 * e + 1], w[0][e], w[1][e], w[2][e]);
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
        if (cg < quad) {  // a block below the diagonal: exp(a_j - A) exp(A - g_t) with A the block's largest a
          const float behind = ex2((lds(tab + (Table::TOP + cg) * 4) - th) + (lds(tab + (Table::TOP + 4 + cg) * 4) - tl));
          scores([&](int j) {
            const float4 f = lds4(tab + (Table::BLOCK + j) * 4);
            return make_float4(f.x * behind, f.y * behind, f.z * behind, f.w * behind);
          });
        } else if (cg == quad) {
          scores([&](int j) {
            const float4 jh = lds4(tab + (Table::AH + j) * 4), jl = lds4(tab + (Table::AL + j) * 4);
            return make_float4(j <= row ? ex2((jh.x - th) + (jl.x - tl)) : 0.f, j + 1 <= row ? ex2((jh.y - th) + (jl.y - tl)) : 0.f,
                               j + 2 <= row ? ex2((jh.z - th) + (jl.z - tl)) : 0.f, j + 3 <= row ? ex2((jh.w - th) + (jl.w - tl)) : 0.f);
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
      const float out = emit ? lds(tab + (Table::OUT + row) * 4) : 0.f;
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
      const bool more = i + 1 < tiles;
      if (more) prepare_values(i + 1);  // while Ya is made
      if (emit && (more || with_n)) wait(yb_done, parity, 16);  // the state at the tile's start has been read (and everybody's numbers of n are there)
      if (with_n) {
        wait(cb_full, parity, 18);  // (these threads read q and k themselves)
        // ---- n: this row's (as a token) share of 32 keys of its read-out, this row's (as a key) of 32 tokens of what the tile adds
        if (emit) {
          float sum = 0.f;
          if (cg * 32 < N) {
            const uint32_t ns = sm + Z::NS + (parity * TOKENS + cg * 32) * 4, qs = sm + Z::C + (cg >> 1) * SLAB + row * 128;
#pragma unroll
            for (int e = 0; e < 4; ++e)
              if (cg * 32 + e * 8 < N) {
                uint32_t q[4];
                ld_shared16(qs + ((((cg & 1) * 4 + e) ^ (row & 7)) << 4), q);
                const float4 a = lds4(ns + e * 32), b = lds4(ns + e * 32 + 16);
                const float2 q0 = unpack2(q[0]), q1 = unpack2(q[1]), q2 = unpack2(q[2]), q3 = unpack2(q[3]);
                sum = fmaf(q0.x, a.x, fmaf(q0.y, a.y, fmaf(q1.x, a.z, fmaf(q1.y, a.w, sum))));
                sum = fmaf(q2.x, b.x, fmaf(q2.y, b.y, fmaf(q3.x, b.z, fmaf(q3.y, b.w, sum))));
              }
          }
          shares[cg * TOKENS + row] = fmaf(out, sum, scored);
        }
        float sum = 0.f;
        if (row < N) {
          const uint32_t ks = sm + Z::B + (row >> 6) * SLAB + (row & 7) * 2;
#pragma unroll 2
          for (int j = cg * 32; j < cg * 32 + 32; j += 4) {
            const float4 w = lds4(tab + (Table::IN + j) * 4);
            const float ws[4] = {w.x, w.y, w.z, w.w};
#pragma unroll
            for (int e = 0; e < 4; ++e) {
              uint16_t k;
              asm volatile("ld.shared.u16 %0, [%1];" : "=h"(k) : "r"(ks + (j + e) * 128 + ((((row & 63) >> 3) ^ ((j + e) & 7)) << 4)) : "memory");
              sum = fmaf(__uint_as_float((uint32_t)k << 16), ws[e], sum);
            }
          }
        }
        shares[(4 + cg) * TOKENS + row] = sum;
        __syncwarp();
        if (lane == 0) bar_arrive(qk_read);
        asm volatile("bar.sync %0, 128;" ::"r"(1 + quad) : "memory");
        if (cg == 0) {
          n_own = fmaf(lds(tab + Table::END * 4), n_own, (shares[4 * TOKENS + row] + shares[5 * TOKENS + row]) + (shares[6 * TOKENS + row] + shares[7 * TOKENS + row]));
          if (emit) {
            const float all = (shares[row] + shares[TOKENS + row]) + (shares[2 * TOKENS + row] + shares[3 * TOKENS + row]);
            if (row < len && left > 1 && !*failed) {
              fin = fmaf(all, 0.f, fin);
              p.divisor[(size_t)(base + row) * p.heads + head] = fmaxf(fabsf(all * scale), lds(tab + (Table::FLOOR + row) * 4)) + 1e-6f;
            }
          } else {
            asm volatile("bar.sync %0, 128;" ::"r"(1 + quad) : "memory");  // (the next tile's shares go there; with read-outs others stand between)
          }
        } else if (!emit) {
          asm volatile("bar.sync %0, 128;" ::"r"(1 + quad) : "memory");
        }
      }
      __syncwarp();
      if (lane == 0) bar_arrive(tab_done + 8 * parity);
      if (more && emit) prepare_state(i + 1);
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
          if (row < len && 8 * h < there) {
#pragma unroll
            for (int e = 0; e < 8; ++e) fin = fmaf(v[8 * h + e], 0.f, fin);
          }
#pragma unroll
          for (int e = 0; e < 8; ++e) v[8 * h + e] *= scale;
        }
        // through shared memory (columns 32 .. in the place of the tile's v, which nobody needs any more), and from there in copies of 32 rows: stores of a
        // row a thread took 3,300 clocks a tile, and the next fence waited for them
        asm volatile("bar.sync %0, 128;" ::"r"(1 + quad) : "memory");
        const uint32_t half = cg < 2 ? sm + Z::Y : sx;
#pragma unroll
        for (int e = 0; e < 4; ++e)
          st_shared16(half + row * 128 + (((4 * (cg & 1) + e) ^ (row & 7)) << 4), __float_as_uint(v[4 * e]), __float_as_uint(v[4 * e + 1]), __float_as_uint(v[4 * e + 2]),
                      __float_as_uint(v[4 * e + 3]));
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        asm volatile("bar.sync %0, 128;" ::"r"(1 + quad) : "memory");
        const bool whole = p.o_vec && quad * 32 + 32 <= len, ok = left > 1 && !*failed;  // 32 rows of this sequence
        if (ok && whole && storer) {
          if (lane < 2 && P - col0 >= 32 * (lane + 1))
            asm volatile("cp.async.bulk.tensor.2d.global.shared::cta.bulk_group [%0, {%2, %3}], [%1];"
                         ::"l"(&map_o), "r"((lane ? sx : sm + Z::Y) + quad * 32 * 128), "r"(head * P + col0 + 32 * lane), "r"(base + quad * 32) : "memory");
          asm volatile("cp.async.bulk.commit_group;" ::: "memory");
        }
        // the ragged rest: rows of a last tile, columns of a last block
        const int c = (lane & 15) * 4;
        if (ok && c < P - col0 && (!whole || P - col0 < (c & 32) + 32)) {
          float* dst = p.o + (size_t)base * inner + head * P + col0 + c;
#pragma unroll
          for (int k = 0; k < 4; ++k) {
            const int r = quad * 32 + cg * 8 + k * 2 + (lane >> 4);
            if (r < len) {
              uint32_t o[4];
              ld_shared16((c < 32 ? sm + Z::Y : sx) + r * 128 + (((lane & 7) ^ (r & 7)) << 4), o);
              float* at = dst + (size_t)r * inner;
              if (p.o_vec) {
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
    asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");  // (a second walk writes behind these)
    if (with_n && cg == 0) S0_n = n_own;
  }
  float* dst = t1 == last ? slot_state : (SECOND ? nullptr : p.part + pbase(seg) * block);
  if (warp < WARPS && emit && dst) {
    each_state([&](int e, size_t) { fin = fmaf(S[e], 0.f, fin); });
    if (with_n && cg == 0 && row < N) fin = fmaf(S0_n, 0.f, fin);
  }
  const bool again = __syncthreads_or(emit && fin != 0.f);  // (also: nobody writes a read-out behind this)
  if (warp == WARPS) {
    tmem_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(T_ALL) : "memory");
  }
  if (*failed) return;
  if (warp == WARPS + 1) {
    if (t1 == last) {  // a copy for each of this CTA's columns (a second walk stores its own)
      for (int c = lane; c < COLS; c += 32)
        if (!again && col0 + c < P) slot_top[col0 + c] = m_end;
      if (!again && with_n && lane == 0) slot_top[P] = m_end;
    } else if (!SECOND && lane == 0 && with_n) {
      p.part_m[pbase(seg) * 2] = m_end;
      p.part_m[pbase(seg) * 2 + 1] = forgot_end;
    }
  }
  if (again) {
    int second = 0, end = 0;  // segments behind the first start again from the state behind it, the last one that was walked from the slot's
    if (SECOND) segment_tiles((last - first + TOKENS - 1) / TOKENS, p.segments, 1, second, end);
    const float* start = SECOND ? p.part + pbase(0) * block : slot_state;
    if (warp < WARPS) {
      const int from_col = col0 + warp * 4, t_from = first + second * TOKENS;
      walk_columns<4>(p, head, from_col, min(P, from_col + 4), start, *first_top, t_from, t0, t1, dst, t1 == last ? slot_top : nullptr);
      if (with_n && warp == 0) walk_columns<1>(p, head, P, P + 1, start, *first_top, t_from, t0, t1, dst, t1 == last ? slot_top : nullptr);
    }
  } else if (dst && warp < WARPS) {
    each_state([&](int e, size_t at) { dst[at] = S[e]; });
    if (with_n && cg == 0 && row < N) dst[(size_t)P * N + row] = S0_n;
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
int launch(const CUtensorMap& map, const CUtensorMap& map_o, const Params& p, cudaStream_t stream) {
  static OncePerDevice configured;
  if (!configured.here()) {
    cudaError_t e = cudaFuncSetAttribute(matrix_memory_umma_kernel<NB, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, Shape<NB>::SMEM);
    if (e == cudaSuccess) e = cudaFuncSetAttribute(matrix_memory_umma_kernel<NB, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, Shape<NB>::SMEM);
    if (e != cudaSuccess) return (int)e;
    configured.here() = true;
  }
  const dim3 grid(column_blocks(p.dv), p.heads, p.num_seqs * (p.segments > 1 ? p.segments - 1 : 1)), block(THREADS);
  cudaError_t e = launch_pdl((matrix_memory_umma_kernel<NB, false>), grid, block, (size_t)Shape<NB>::SMEM, stream, 1, map, map_o, p);
  if (e == cudaSuccess && p.segments > 1) e = launch_pdl((matrix_memory_umma_kernel<NB, true>), grid, block, (size_t)Shape<NB>::SMEM, stream, 1, map, map_o, p);
  return (int)e;
}

}  // namespace

// Into how many segments the sequences of a step are cut: a launch (of one segment fewer) gives every SM a CTA, and behind the first there is at most one for every
// three tiles of the longest sequence: those have about three tiles or more, the last of them what is left, and the first what they leave, often one (segment_tiles).  Two segments would follow one another: three is the fewest that gain.
DLI_EXPORT int dli_matrix_memory_umma_segments(int num_seqs, int heads, int dv, int max_len) {
  const long long units = (long long)column_blocks(dv) * heads * (num_seqs > 0 ? num_seqs : 1);
  long long fill = sm_count() / (units > 0 ? units : 1);
  const int most = (max_len + TOKENS - 1) / TOKENS / 3;
  if (fill > most) fill = most;
  return fill < 2 ? 1 : (fill > 32 ? 33 : (int)fill + 1);
}

static int run(float* o, float* divisor, const void* u, long long u_stride, const float* gates, const float* bias, float cap, float* state, float* top, const int* q_start,
               const int* state_slot, int num_seqs, int heads, int d, int dv, int n, int segments, float* part, float* part_m, unsigned wait_limit, int skip_tile,
               cudaStream_t stream) {
  if (num_seqs == 0 || n == 0) return 0;
  if (n < 0 || heads < 1 || heads > 65535 || d < 32 || d > 128 || d % 16 || dv < 8 || dv % 8 || segments < 1 || (long long)num_seqs * segments > 65535 || !(cap > 0.f) ||
      ((uintptr_t)u & 15) || u_stride % 8 || ((uintptr_t)o & 7) || (segments > 1 && (!part || !part_m)))
    return DLI_ERR_UNSUPPORTED;
  if (!error_flag_host) {
    if (cudaHostAlloc((void**)&error_flag_host, sizeof(int), cudaHostAllocMapped) != cudaSuccess) return (int)cudaGetLastError();
    *error_flag_host = 0;
    if (cudaHostGetDevicePointer((void**)&error_flag_device, error_flag_host, 0) != cudaSuccess) return (int)cudaGetLastError();
  }
  CUtensorMap map, map_o;
  if (!make_map(&map, u, false, n, (long long)heads * (2 * d + dv), u_stride, TOKENS)) return DLI_ERR_UNSUPPORTED;
  map_o = map;  // (not used where o is not aligned)
  const int o_vec = ((uintptr_t)o & 15) == 0;
  if (o_vec && !make_map(&map_o, o, true, n, (long long)heads * dv, (long long)heads * dv, 32)) return DLI_ERR_UNSUPPORTED;
  Params p;
  p.o = o; p.divisor = divisor; p.u = (const bf16*)u; p.u_stride = u_stride; p.gates = gates; p.bias = bias; p.cap = cap; p.state = state; p.top = top;
  p.q_start = q_start; p.state_slot = state_slot; p.num_seqs = num_seqs; p.heads = heads; p.d = d; p.dv = dv; p.segments = segments; p.part = part;
  p.part_m = part_m; p.o_vec = o_vec; p.short_shift = short_shift((long long)column_blocks(dv) * heads * num_seqs); p.error_flag = error_flag_device;
  p.wait_limit = wait_limit; p.skip_tile = skip_tile;
  return d <= 64 ? launch<1>(map, map_o, p, stream) : launch<2>(map, map_o, p, stream);
}

// n: rows of u.  segments > 1: part [num_seqs (segments - 1) heads (dv + 1) d] and part_m [num_seqs (segments - 1) heads 2] are scratch.
DLI_EXPORT int dli_matrix_memory_umma(float* o, float* divisor, const void* u, long long u_stride, const float* gates, const float* bias, float cap, float* state,
                                      float* top, const int* q_start, const int* state_slot, int num_seqs, int heads, int d, int dv, int n, int segments, float* part,
                                      float* part_m, cudaStream_t stream) {
  return run(o, divisor, u, u_stride, gates, bias, cap, state, top, q_start, state_slot, num_seqs, heads, d, dv, n, segments, part, part_m, WAIT_LIMIT, -1, stream);
}

// For tests: in one segment, with every CTA's copies of q and k of tile `skip_tile` left out and every wait given up after `wait_limit` polls.
DLI_EXPORT int dli_matrix_memory_umma_wait_test(float* o, float* divisor, const void* u, long long u_stride, const float* gates, const float* bias, float cap, float* state,
                                                float* top, const int* q_start, const int* state_slot, int num_seqs, int heads, int d, int dv, int n, unsigned wait_limit,
                                                int skip_tile, cudaStream_t stream) {
  if (wait_limit < 2 || wait_limit > WAIT_LIMIT || skip_tile < 0) return DLI_ERR_UNSUPPORTED;
  return run(o, divisor, u, u_stride, gates, bias, cap, state, top, q_start, state_slot, num_seqs, heads, d, dv, n, 1, nullptr, nullptr, wait_limit, skip_tile, stream);
}

// 0, or the code of the first wait that ran out since the library was loaded or the code was last cleared
DLI_EXPORT int dli_matrix_memory_umma_error() { return error_flag_host ? *error_flag_host : 0; }
DLI_EXPORT int dli_matrix_memory_umma_clear_error() { if (error_flag_host) *error_flag_host = 0; return 0; }
