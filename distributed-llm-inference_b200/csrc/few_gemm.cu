// out[t, f] = sum over k of x[t, k] * W[f, k] for a step of some tokens (up to 128; the engine asks for 9 to 96, kernels/gemm.py: few_max_tokens), bfloat16 in and out, float32 sums, on tcgen05; or the activation of a
// gated feed-forward on such sums.
//
// A step of so few tokens is the reading of the weights: features take the 128-row side of the instruction, all tokens its columns, and every weight
// tile is read once.  A CTA has 128 features and a share of k; the CTAs of a cluster have the same features, exchange their sums through distributed shared
// memory and finish a share of the tokens each, in the same order always.
//
//   * One thread copies (TMA, 128-byte swizzle) a [128 x 128] tile of W and the [tokens x 128] tile of x per step of 128 k, as many steps ahead as shared memory
//     holds; the weights of the first steps are asked for before the kernel in front has ended.  A copy brings both slabs of 64 k (a third dimension of the tensor
//     map): an SM gets a pair of copies each 0.2 us, whatever their size.
//   * A warp issues tcgen05.mma (M = 128, N = the tokens rounded up to 16) into one accumulator.
//   * Eight warps bring the sums to shared memory, token by token, and all write them out, whole rows of 128 features at a time.
//
// What bounds it: the weights' way from HBM where all SMs take part (16,384 features of K 2,048 at 9 tokens: 12.9 us, 5.2 TB/s), otherwise a product's start, the exchange
// and the end, about 3 us (1 to 2 more at 64 tokens).  Figures against the library's products stand beside the rule (kernels/gemm.py).  Before a copy
// brought 128 k, K 8,192 on sixteen SMs took 27 us instead of 18.
//
// Every wait on an mbarrier is bounded: after `wait_limit` polls a code goes to *error_flag, no CTA of the cluster stores anything (the others hear of it in front of
// the barrier behind which sums are added), and the CTA ends when its copies have landed.
#include "umma_tiles.cuh"
#include <type_traits>

using namespace dli;
using namespace dli::umma;
typedef __nv_bfloat16 bf16;

namespace {

constexpr int BF = 128;  // features of a tile
constexpr int BK = 128;  // k of a step: two slabs of 64 for either operand
constexpr int THREADS = 320;  // warp 0: copies, warp 1: products, warps 2..9: sums; all of them write
enum { STORE = 0, SWIGLU = 1 };

struct FewParams {
  bf16* out;
  int tokens, features, K, splits, mode;
  int wide;  // K is a multiple of 128: one copy brings both slabs
  int* error_flag;
  unsigned wait_limit;
  int skip_step;  // -1 in every launch of the engine: the step whose copies of x a test leaves out (dli_few_gemm_wait_test)
};

template <int NT> struct Shape {  // NT: room for tokens
  static constexpr int A_SLAB = BF * 128, B_SLAB = NT * 128, B = 2 * A_SLAB, STAGE = 2 * (A_SLAB + B_SLAB);
  static constexpr int STAGES = NT <= 32 ? 5 : NT == 64 ? 4 : 3;
  static constexpr int COLUMNS = NT < 32 ? 32 : NT;
  static constexpr int SUMS = NT * BF * 4;  // a CTA's sums [tokens][features], in the stages' place
  static constexpr int SMEM = STAGES * STAGE + 256 + 1024;
  static_assert(SMEM <= 227 * 1024 && SUMS <= STAGES * STAGE, "shared memory");
};

template <int NT>
__global__ void __launch_bounds__(THREADS, 1) few_gemm_kernel(const __grid_constant__ CUtensorMap map_x, const __grid_constant__ CUtensorMap map_w,
                                                              const __grid_constant__ FewParams p) {
  using Z = Shape<NT>;
  pdl_launch_dependents();
  extern __shared__ unsigned char smem_raw[];
  unsigned char* smem = (unsigned char*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  const uint32_t sm = smem_u32(smem), full0 = sm + Z::STAGES * Z::STAGE, empty0 = full0 + 8 * Z::STAGES, done = empty0 + 8 * Z::STAGES;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(smem + Z::STAGES * Z::STAGE + 16 * Z::STAGES + 8);
  volatile int* failed = reinterpret_cast<volatile int*>(tmem_slot + 1);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  if (tid == 0) {
    for (int s = 0; s < Z::STAGES; ++s) {
      bar_init(full0 + 8 * s, 1);
      bar_init(empty0 + 8 * s, 1);
    }
    bar_init(done, 1);
    *failed = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)), "r"(Z::COLUMNS) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  tmem_before();
  __syncthreads();
  tmem_after();
  const uint32_t tmem = *tmem_slot;
  const int f0 = blockIdx.x * BF, split = blockIdx.y, all = (p.K + BK - 1) / BK, share = (all + p.splits - 1) / p.splits;
  const int first = min(all, split * share), steps = min(all, first + share) - first;  // (a last split may be empty)
  unsigned left = p.wait_limit;

  if (warp == 0) {
    const uint32_t one = elect_one();
    const int ahead = min(steps, Z::STAGES);
    auto load = [&](uint32_t dst, const CUtensorMap* map, int step, int row, int slab, uint32_t bar) {
      if (p.wide) {
        asm volatile("cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5}], [%2];"
                     ::"r"(dst), "l"(map), "r"(bar), "r"(0), "r"(row), "r"(2 * step) : "memory");
      } else {
        tma_load(dst, map, step * BK, row, bar);
        tma_load(dst + slab, map, step * BK + 64, row, bar);
      }
    };
    if (one) {  // nobody writes the weights: those of the first steps need not wait for the kernel in front
      for (int s = 0; s < ahead; ++s) {
        bar_expect(full0 + 8 * s, Z::STAGE);
        load(sm + s * Z::STAGE, &map_w, first + s, f0, Z::A_SLAB, full0 + 8 * s);
      }
    }
    __syncwarp();
    pdl_wait();
    if (one)
      for (int s = 0; s < ahead; ++s)
        if (first + s != p.skip_step) load(sm + s * Z::STAGE + Z::B, &map_x, first + s, 0, Z::B_SLAB, full0 + 8 * s);
    __syncwarp();
    int asked = ahead;
    for (int s = ahead; s < steps; ++s) {
      const int stage = s % Z::STAGES;
      bar_wait(empty0 + 8 * stage, (s / Z::STAGES - 1) & 1, left, failed, p.error_flag, 1);
      if (left == 1) break;
      if (one) {
        bar_expect(full0 + 8 * stage, Z::STAGE);
        load(sm + stage * Z::STAGE, &map_w, first + s, f0, Z::A_SLAB, full0 + 8 * stage);
        load(sm + stage * Z::STAGE + Z::B, &map_x, first + s, 0, Z::B_SLAB, full0 + 8 * stage);
      }
      __syncwarp();
      asked = s + 1;
    }
    if (*failed)  // what is still on its way lands here, not in the next CTA's shared memory
      for (int s = max(0, asked - Z::STAGES); s < asked; ++s)
        for (unsigned i = 0; i < p.wait_limit && !bar_done(full0 + 8 * (s % Z::STAGES), (s / Z::STAGES) & 1); ++i) {}
  } else if (warp == 1) {
    const uint32_t one = elect_one(), tm = __shfl_sync(0xffffffffu, tmem, 0), idesc = instruction((p.tokens + 15) / 16 * 16, false, false);
    const uint64_t stages = operand(sm);  // (a descriptor counts 16 bytes)
    for (int s = 0; s < steps; ++s) {
      const int stage = s % Z::STAGES;
      bar_wait(full0 + 8 * stage, (s / Z::STAGES) & 1, left, failed, p.error_flag, 2);
      if (left == 1) break;
      tmem_after();
      const uint64_t a = stages + (uint32_t)((stage * Z::STAGE) >> 4), b = a + (Z::B >> 4);
#pragma unroll
      for (int k = 0; k < BK / 16; ++k)
        product(one, tm, a + (((k >> 2) * Z::A_SLAB + (k & 3) * 32) >> 4), b + (((k >> 2) * Z::B_SLAB + (k & 3) * 32) >> 4), idesc, s > 0 || k > 0);
      commit(one, empty0 + 8 * stage);
    }
    commit(one, done);
    __syncwarp();
  } else {
    // ---- the sums to shared memory: lane = feature, column = token
    bar_wait(done, 0, left, failed, p.error_flag, 3);
    tmem_after();
    const int quad = warp & 3;
    float* sums = reinterpret_cast<float*>(smem) + quad * 32 + lane;
    for (int j = warp < 6 ? 0 : 16; j < p.tokens; j += 32) {  // (two warps of a quarter of the features take sixteen tokens in turn)
      uint32_t v[16];
      if (steps > 0) {
        tmem_ld16(tmem + ((uint32_t)(quad * 32) << 16) + j, v);
        tmem_wait_ld();
      } else {
#pragma unroll
        for (int e = 0; e < 16; ++e) v[e] = 0;
      }
#pragma unroll
      for (int e = 0; e < 16; ++e) sums[(j + e) * BF] = __uint_as_float(v[e]);  // (NT is a multiple of 16)
    }
    tmem_before();
  }
  if (left == 1 && lane < p.splits)  // a wait of this warp ran out: every CTA of the cluster would add what is not there
    asm volatile("{\n\t.reg .b32 remote;\n\tmapa.shared::cluster.u32 remote, %0, %1;\n\tst.shared::cluster.u32 [remote], %2;\n\t}"
                 ::"r"(smem_u32(tmem_slot + 1)), "r"(lane), "r"(*failed) : "memory");
  if (p.splits > 1) asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
  else __syncthreads();
  pdl_wait();  // (every thread that writes: the output may alias memory that the kernel in front still reads)

  // ---- this CTA's share of the tokens
  const int per = (p.tokens + p.splits - 1) / p.splits, t_end = min(p.tokens, (split + 1) * per);
  // features f .. f + 3 of the tile and of token t, added over the cluster: COUNT of them, (dt, df) apart, so that their loads are under way together
  auto sums4 = [&](auto count, int t, int dt, int f, int df, float4 (&sum)[decltype(count)::value]) {
    constexpr int COUNT = decltype(count)::value;
    if (p.splits == 1) {
#pragma unroll
      for (int c = 0; c < COUNT; ++c) sum[c] = lds4(sm + (min(t + c * dt, t_end - 1) * BF + f + c * df) * 4);
      return;
    }
    auto add = [&](auto ranks) {
      constexpr int RANKS = decltype(ranks)::value;
      float4 v[COUNT][RANKS];
#pragma unroll
      for (int c = 0; c < COUNT; ++c)
#pragma unroll
        for (int r = 0; r < RANKS; ++r)
          asm volatile("{\n\t.reg .b32 remote;\n\tmapa.shared::cluster.u32 remote, %4, %5;\n\tld.shared::cluster.v4.f32 {%0,%1,%2,%3}, [remote];\n\t}"
                       : "=f"(v[c][r].x), "=f"(v[c][r].y), "=f"(v[c][r].z), "=f"(v[c][r].w) : "r"(sm + (min(t + c * dt, t_end - 1) * BF + f + c * df) * 4), "r"(r) : "memory");
#pragma unroll
      for (int c = 0; c < COUNT; ++c) {
        sum[c] = v[c][0];
#pragma unroll
        for (int r = 1; r < RANKS; ++r) { sum[c].x += v[c][r].x; sum[c].y += v[c][r].y; sum[c].z += v[c][r].z; sum[c].w += v[c][r].w; }
      }
    };
    if (p.splits == 2) add(std::integral_constant<int, 2>());
    else if (p.splits == 4) add(std::integral_constant<int, 4>());
    else add(std::integral_constant<int, 8>());
  };
  const std::integral_constant<int, 2> two;
  if (!*failed) {
    if (p.mode == STORE) {
      const int f = lane * 4;
      if (f0 + f < p.features)  // (a multiple of 4)
        for (int t = split * per + warp; t < t_end; t += 2 * (THREADS / 32)) {
          float4 v[2];
          sums4(two, t, THREADS / 32, f, 0, v);
#pragma unroll
          for (int c = 0; c < 2; ++c)
            if (t + c * (THREADS / 32) < t_end)
              *reinterpret_cast<uint2*>(p.out + (size_t)(t + c * (THREADS / 32)) * p.features + f0 + f) = make_uint2(pack2(v[c].x, v[c].y), pack2(v[c].z, v[c].w));
        }
    } else {  // rows of the tile: 64 gates, then the 64 ups of the same features; the sums as bfloat16 would hold them, as for other numbers of tokens
      const int f = (lane & 15) * 4, I = p.features >> 1;
      for (int t = split * per + warp * 2 + (lane >> 4); t < t_end; t += THREADS / 16) {
        float4 v[2];
        sums4(two, t, 0, f, 64, v);
        auto act = [](float a, float b) {
          a = __bfloat162float(__float2bfloat16_rn(a));
          return a / (1.f + expf(-a)) * __bfloat162float(__float2bfloat16_rn(b));
        };
        *reinterpret_cast<uint2*>(p.out + (size_t)t * I + f0 / 2 + f) =
            make_uint2(pack2(act(v[0].x, v[1].x), act(v[0].y, v[1].y)), pack2(act(v[0].z, v[1].z), act(v[0].w, v[1].w)));
      }
    }
  }
  if (p.splits > 1) asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");  // nobody leaves while its sums are read
  else __syncthreads();
  if (warp == 1) {
    tmem_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(Z::COLUMNS) : "memory");
  }
}

// rows x K bfloat16 numbers, rows `row` apart, as [K / 64][rows][64], in boxes of two of the first, box_rows of the second
bool make_wide_map(CUtensorMap* map, const void* base, long long rows, long long K, long long row, int box_rows) {
  EncodeTiled fn = encode_fn();
  if (!fn) return false;
  cuuint64_t dims[3] = {64, (cuuint64_t)rows, (cuuint64_t)(K / 64)}, strides[2] = {(cuuint64_t)row * 2, 128};
  cuuint32_t box[3] = {64, (cuuint32_t)box_rows, 2}, elem[3] = {1, 1, 1};
  return fn(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, const_cast<void*>(base), dims, strides, box, elem, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
            CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

int* error_flag_device = nullptr;
int* error_flag_host = nullptr;

template <int NT> int launch(const CUtensorMap& map_x, const CUtensorMap& map_w, const FewParams& p, cudaStream_t stream) {
  static OncePerDevice configured;
  if (!configured.here()) {
    const cudaError_t e = cudaFuncSetAttribute(few_gemm_kernel<NT>, cudaFuncAttributeMaxDynamicSharedMemorySize, Shape<NT>::SMEM);
    if (e != cudaSuccess) return (int)e;
    configured.here() = true;
  }
  return (int)launch_pdl((few_gemm_kernel<NT>), dim3((p.features + BF - 1) / BF, p.splits), dim3(THREADS), (size_t)Shape<NT>::SMEM, stream, p.splits, map_x, map_w, p);
}

}  // namespace

static int run(void* out, const void* x, const void* w, int tokens, int features, int K, long long x_row, int swiglu, int splits, unsigned wait_limit, int skip_step,
               cudaStream_t stream) {
  if (tokens < 1 || tokens > 128 || features < 4 || features % 4 || K < 8 || K % 8 || x_row % 8 || (((uintptr_t)x | (uintptr_t)w) & 15) || ((uintptr_t)out & 7) ||
      (swiglu && features % 128) || (splits != 1 && splits != 2 && splits != 4 && splits != 8))
    return DLI_ERR_UNSUPPORTED;
  if (!error_flag_host) {
    if (cudaHostAlloc((void**)&error_flag_host, sizeof(int), cudaHostAllocMapped) != cudaSuccess) return (int)cudaGetLastError();
    *error_flag_host = 0;
    if (cudaHostGetDevicePointer((void**)&error_flag_device, error_flag_host, 0) != cudaSuccess) return (int)cudaGetLastError();
  }
  const int room = tokens <= 16 ? 16 : tokens <= 32 ? 32 : tokens <= 64 ? 64 : 128;
  CUtensorMap map_x, map_w;
  const int wide = K % BK == 0;
  const bool made = wide ? make_wide_map(&map_x, x, tokens, K, x_row, room) && make_wide_map(&map_w, w, features, K, K, BF)
                         : make_map(&map_x, x, false, tokens, K, x_row, room) && make_map(&map_w, w, false, features, K, K, BF);
  if (!made) return DLI_ERR_UNSUPPORTED;
  FewParams p;
  p.out = (bf16*)out; p.tokens = tokens; p.features = features; p.K = K; p.splits = splits; p.mode = swiglu ? SWIGLU : STORE; p.wide = wide; p.error_flag = error_flag_device;
  p.wait_limit = wait_limit; p.skip_step = skip_step;
  if (room == 16) return launch<16>(map_x, map_w, p, stream);
  if (room == 32) return launch<32>(map_x, map_w, p, stream);
  return room == 64 ? launch<64>(map_x, map_w, p, stream) : launch<128>(map_x, map_w, p, stream);
}

// out [tokens][features], or (swiglu) [tokens][features / 2] = silu(gate) * up for weights whose rows are interleaved in blocks of 64 gate rows and the 64 up
// rows of the same features.  x: rows x_row numbers apart.  splits (1, 2, 4 or 8): CTAs that share a tile's k.
DLI_EXPORT int dli_few_gemm(void* out, const void* x, const void* w, int tokens, int features, int K, long long x_row, int swiglu, int splits, cudaStream_t stream) {
  return run(out, x, w, tokens, features, K, x_row, swiglu, splits, WAIT_LIMIT, -1, stream);
}

// For tests: the copies of x of step `skip_step` (of 128 k) are left out and every wait gives up after `wait_limit` polls: the wait for that step runs out (code 2), and
// the one for the sums that depend on it (3).  Every step has a stage of its own.
DLI_EXPORT int dli_few_gemm_wait_test(void* out, const void* x, const void* w, int tokens, int features, int K, int splits, unsigned wait_limit, int skip_step,
                                      cudaStream_t stream) {
  const int steps = (K + BK - 1) / BK;
  if (wait_limit < 2 || wait_limit > WAIT_LIMIT || tokens > 32 || splits < 1 || (steps + splits - 1) / splits > Shape<32>::STAGES || skip_step < 0 || skip_step >= steps)
    return DLI_ERR_UNSUPPORTED;
  return run(out, x, w, tokens, features, K, K, 0, splits, wait_limit, skip_step, stream);
}

// 0, or the code of the first wait that ran out (1 stages, 2 copies, 3 sums)
DLI_EXPORT int dli_few_gemm_error() { return error_flag_host ? *error_flag_host : 0; }
DLI_EXPORT int dli_few_gemm_clear_error() { if (error_flag_host) *error_flag_host = 0; return 0; }
