// Integer GEMM over a batch of samples laid side by side along the contraction axis, each with a pair of scales of its own:
//   out[m, n] = (sum_g ((float)(sum_{k in sample g} a[m, k] * b[n, k]) * scale_a[g (, m)]) * scale_b[g]) * post
// (the weight gradient under the reference's 3-D semantics).  The sum over samples runs in fp32, sample 0 first, so it
// cannot be left to the tensor core: every sample's accumulator is read back, scaled and added.
//
// One CTA per 128 x BN tile.  The tensor core runs up to four samples ahead (four accumulators of at most 128 columns in
// tensor memory); BN / 32 teams of four warps drain them, a thread keeping the running sums of 32 columns of its row in
// registers.
//
// What bounds it at ViT sizes (2304 x 768, 64 samples of 197 tokens: 47.6 us, 62.9 with the drain in eight warps): a sample
// costs a CTA some 1,300 cycles.  Its seven instructions alone take 390 to 450; they share shared memory with the copies
// that fill it (56 to 64 KB a sample) and the issuing thread with the barriers.  The drain keeps up: four warps per 32
// columns, two conversions and three packed operations a pair.  The chain of samples cannot be split over CTAs without
// changing the order of the sum, so BN is chosen for the shortest time of the busiest CTA: 96 where that fills one wave
// (18 x 8 tiles), 32 where few tiles there are.
#include "tc.cuh"

namespace hot {

int device_sm_count();

namespace {

constexpr int kBM = 128, kBK = 128;
constexpr int kSmemMax = 227 * 1024;
constexpr int kBufs = 4;

struct GroupedParams {
  int M, N, groups;
  int n_tiles, num_tiles;
  int blocks;       // k-blocks of 128 per sample
  int last_steps;   // instructions of 32 in a sample's last k-block
  const float* sa;  // [groups] or [groups, M]
  const float* sb;  // [groups]
  int sa_row;
  float post;
  float one;        // 1, where the compiler cannot see it (see the drain)
  int out16;
  uint32_t* status;
  uint64_t wait_ns;
};

template <int BN>
struct Layout {
  static constexpr int kTeams = BN / 32, kEpiWarps = 4 * kTeams, kThreads = (kEpiWarps + 2) * 32;
  static constexpr int kA = kBM * kBK, kB = BN * kBK, kStage = kA + kB;
  static constexpr int kStore = kEpiWarps * 4096;  // a box of 32 rows x 128 bytes per warp
  static constexpr int kFit = (kSmemMax - 2048 - kStore) / kStage;
  static constexpr int kStages = kFit > 8 ? 8 : kFit;
  static constexpr int kOffB = kStages * kA, kOffStore = kOffB + kStages * kB, kOffBar = kOffStore + kStore;
  static constexpr int kBytes = kOffBar + 512 + 1024;
  static constexpr uint32_t kTmemCols = BN * kBufs <= 128 ? 128 : (BN * kBufs <= 256 ? 256 : 512);
  static_assert(kBytes <= kSmemMax && kStages >= 4 && kOffStore % 1024 == 0, "shared-memory plan");
};

template <int BN>
__global__ void __launch_bounds__(Layout<BN>::kThreads, 1)
    gemm_grouped_kernel(const __grid_constant__ CUtensorMap tma_a, const __grid_constant__ CUtensorMap tma_b,
                        const __grid_constant__ CUtensorMap tma_out, const __grid_constant__ GroupedParams p) {
  using L = Layout<BN>;
  constexpr int STAGES = L::kStages;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = smem_raw + ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u);
  uint64_t* full = reinterpret_cast<uint64_t*>(smem + L::kOffBar);
  uint64_t* empty = full + STAGES;
  uint64_t* tmem_full = empty + STAGES;      // [kBufs] a sample's accumulator is complete
  uint64_t* tmem_empty = tmem_full + kBufs;  // [kBufs] drained
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(tmem_empty + kBufs);
  volatile uint32_t* abort_flag = tmem_slot + 1;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  constexpr int kProducer = L::kEpiWarps, kMma = kProducer + 1;

  if (threadIdx.x == 0) {
    for (int s = 0; s < STAGES; ++s) {
      mbar_init(&full[s], 1);
      mbar_init(&empty[s], 1);
    }
    for (int b = 0; b < kBufs; ++b) {
      mbar_init(&tmem_full[b], 1);
      mbar_init(&tmem_empty[b], L::kEpiWarps);
    }
    *abort_flag = 0u;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    tma_prefetch_desc(&tma_a);
    tma_prefetch_desc(&tma_b);
    tma_prefetch_desc(&tma_out);
  }
  if (warp == kMma) tmem_alloc(tmem_slot, L::kTmemCols);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  // launched as a programmatic dependent: the set-up above ran while the kernel before it drained
  asm volatile("griddepcontrol.wait;" ::: "memory");
  const uint32_t tmem_base = *tmem_slot;

  if (warp == kProducer) {
    if (elect_one()) {
      uint32_t s = 0, ph = 0;
      bool ok = true;
      const int total = p.groups * p.blocks;
      for (int tile = blockIdx.x; ok && tile < p.num_tiles; tile += gridDim.x) {
        const int m0 = tile / p.n_tiles * kBM, n0 = tile % p.n_tiles * BN;
        for (int kb = 0; kb < total; ++kb, s = (s + 1 == STAGES ? 0 : s + 1), ph ^= (s == 0 ? 1u : 0u)) {
          ok = mbar_wait(&empty[s], ph ^ 1u, abort_flag, p.wait_ns);
          if (!ok) break;
          mbar_expect_tx(&full[s], L::kStage);
          tma_load_2d(smem + s * L::kA, &tma_a, &full[s], kb * kBK, m0);
          tma_load_2d(smem + L::kOffB + s * L::kB, &tma_b, &full[s], kb * kBK, n0);
        }
      }
    }
  } else if (warp == kMma) {
    if (elect_one()) {
      constexpr uint32_t idesc = instr_desc_i8(BN);
      const uint32_t hi = (uint32_t)(smem_desc_sw128(0) >> 32);
      const uint32_t a_lo0 = (uint32_t)smem_desc_sw128(smem_u32(smem)), b_lo0 = (uint32_t)smem_desc_sw128(smem_u32(smem + L::kOffB));
      uint32_t s = 0, ph = 0, it = 0;
      bool ok = true;
      for (int tile = blockIdx.x; ok && tile < p.num_tiles; tile += gridDim.x) {
        for (int g = 0; ok && g < p.groups; ++g, ++it) {
          const uint32_t buf = it % kBufs, bph = (it / kBufs) & 1u;
          ok = mbar_wait(&tmem_empty[buf], bph ^ 1u, abort_flag, p.wait_ns);
          if (!ok) break;
          tc_fence_after();
          const uint32_t d = tmem_base + buf * BN;
          for (int kb = 0; kb < p.blocks; ++kb, s = (s + 1 == STAGES ? 0 : s + 1), ph ^= (s == 0 ? 1u : 0u)) {
            ok = mbar_wait(&full[s], ph, abort_flag, p.wait_ns);
            if (!ok) break;
            tc_fence_after();
            const uint32_t a_lo = a_lo0 + s * (uint32_t)(L::kA >> 4), b_lo = b_lo0 + s * (uint32_t)(L::kB >> 4);
            const int steps = kb + 1 == p.blocks ? p.last_steps : kBK / 32;
#pragma unroll
            for (int k = 0; k < kBK / 32; ++k)
              if (k < steps) umma_i8(d, ((uint64_t)hi << 32) | (a_lo + 2u * k), ((uint64_t)hi << 32) | (b_lo + 2u * k), idesc, kb > 0 || k > 0 ? 1u : 0u);
            umma_commit(&empty[s]);
          }
          if (ok) umma_commit(&tmem_full[buf]);
        }
      }
    }
  } else {
    const int q = warp & 3, col = (warp >> 2) * 32;  // tensor-memory lane quarter and first column of this warp
    uint8_t* const box = smem + L::kOffStore + warp * 4096;
    uint32_t it = 0;
    bool ok = true;
    for (int tile = blockIdx.x; ok && tile < p.num_tiles; tile += gridDim.x) {
      const int m0 = tile / p.n_tiles * kBM, n0 = tile % p.n_tiles * BN;
      const int row = m0 + q * 32 + lane;
      const float* sa = p.sa + (p.sa_row && row < p.M ? row : 0);
      const int64_t sa_step = p.sa_row ? p.M : 1;
      float2 run[16];
#pragma unroll
      for (int i = 0; i < 16; ++i) run[i] = make_float2(-0.0f, -0.0f);  // (-0 + v is v, also for v = -0)
      float ga = load_result(sa), gb = load_result(p.sb);
      for (int g = 0; g < p.groups; ++g, ++it) {
        const uint32_t buf = it % kBufs, bph = (it / kBufs) & 1u;
        float ga_next = 0.0f, gb_next = 0.0f;
        if (g + 1 < p.groups) {  // in flight during the wait
          ga_next = load_result(sa + (g + 1) * sa_step);
          gb_next = load_result(p.sb + g + 1);
        }
        ok = __all_sync(0xFFFFFFFFu, mbar_wait_parked(&tmem_full[buf], bph, abort_flag, p.wait_ns)) != 0;
        if (!ok) break;
        tc_fence_after();
        uint32_t acc[32];
        tmem_ld32(tmem_base + buf * BN + ((uint32_t)(q * 32) << 16) + col, acc);
        tc_fence_before();
        __syncwarp();
        if (elect_one()) mbar_arrive(&tmem_empty[buf]);
        const float2 a2 = make_float2(ga, ga), b2 = make_float2(gb, gb), one = make_float2(p.one, p.one);
#pragma unroll
        for (int i = 0; i < 16; ++i) {
          const float2 f = make_float2((float)(int)acc[2 * i], (float)(int)acc[2 * i + 1]);
          // the sum as v * 1 + run: the compiler joins a packed addition with the packed product before it, which then rounds
          // once where the reference rounds twice
          run[i] = __ffma2_rn(__fmul2_rn(__fmul2_rn(f, a2), b2), one, run[i]);
        }
        ga = ga_next;
        gb = gb_next;
      }
      if (!ok) break;
      // 32 rows x 32 columns of this warp through a swizzled box
      const float2 post2 = make_float2(p.post, p.post);
      if (elect_one()) bulk_wait_group_read<0>();  // the store of the tile before has left the box
      __syncwarp();
      if (p.out16) {
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          uint32_t w[4];
#pragma unroll
          for (int k = 0; k < 4; ++k) {
            const float2 f = __fmul2_rn(run[4 * j + k], post2);
            const __nv_bfloat162 t = __floats2bfloat162_rn(f.x, f.y);
            w[k] = *reinterpret_cast<const uint32_t*>(&t);
          }
          *reinterpret_cast<uint4*>(box + lane * 64 + ((j ^ ((lane >> 1) & 3)) << 4)) = make_uint4(w[0], w[1], w[2], w[3]);
        }
      } else {
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          const float2 f0 = __fmul2_rn(run[2 * j], post2), f1 = __fmul2_rn(run[2 * j + 1], post2);
          *reinterpret_cast<uint4*>(box + lane * 128 + ((j ^ (lane & 7)) << 4)) =
              make_uint4(__float_as_uint(f0.x), __float_as_uint(f0.y), __float_as_uint(f1.x), __float_as_uint(f1.y));
        }
      }
      fence_proxy_async_smem();
      __syncwarp();
      const int c = n0 + col, y = m0 + q * 32;
      if (elect_one()) {
        if (c < p.N && y < p.M) tma_store_2d(&tma_out, box, c << (p.out16 ? 1 : 2), y);
        bulk_commit_group();
      }
    }
    if (elect_one()) bulk_wait_group<0>();
  }

  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  tc_fence_before();
  __syncthreads();
  if (warp == kMma) {
    tc_fence_after();
    tmem_dealloc(tmem_base, L::kTmemCols);
  }
  if (threadIdx.x == 0 && *abort_flag) {
    if (p.status) atomicOr(p.status, (uint32_t)HOT_STATUS_GEMM);
    const uint64_t t0 = global_timer_ns();  // let bulk copies already issued land before exit
    while (global_timer_ns() - t0 < 100000ull) {
    }
  }
}

template <int BN>
int launch(const void* a, int64_t lda, const void* b, int64_t ldb, void* out, int64_t ldo, int64_t K, GroupedParams& p, int sms, cudaStream_t st) {
  using L = Layout<BN>;
  const int64_t esz = p.out16 ? 2 : 4;
  CUtensorMap ma, mb, mo;
  if (int rc = make_map(&ma, a, p.M, K, lda, kBK, kBM, 128)) return rc;
  if (int rc = make_map(&mb, b, p.N, K, ldb, kBK, BN, 128)) return rc;
  if (int rc = make_map(&mo, out, p.M, p.N * esz, ldo * esz, 32 * (int)esz, 32, 32 * (int)esz)) return rc;
  auto kernel = gemm_grouped_kernel<BN>;
  static PerDeviceOnce once;
  bool done = false;
  const int dev = once.current(&done);
  if (dev < 0) HOT_FAIL(HOT_ERR_CUDA, "hot_gemm_i8_grouped: cannot query the current CUDA device");
  if (!done) {
    HOT_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, L::kBytes));
    once.mark(dev);
  }
  p.n_tiles = (p.N + BN - 1) / BN;
  p.num_tiles = (p.M + kBM - 1) / kBM * p.n_tiles;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)(p.num_tiles < sms ? p.num_tiles : sms));
  cfg.blockDim = dim3(L::kThreads);
  cfg.dynamicSmemBytes = L::kBytes;
  cfg.stream = st;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  HOT_CUDA(cudaLaunchKernelEx(&cfg, kernel, ma, mb, mo, p));
  return HOT_OK;
}

}  // namespace

// hot_gemm_i8_grouped where only the first `len` codes of a sample are not zero.
int gemm_i8_grouped(const void* a, int64_t lda, const void* b, int64_t ldb, int64_t M, int64_t N, int64_t groups, int64_t group_k,
                    int64_t len, const float* scale_a, int scale_a_per_row, const float* scale_b, float post, void* out, int out_dtype,
                    int64_t ldo, uint32_t* status_word, hot_stream_t stream) {
  if (!a || !b || !out || !scale_a || !scale_b) HOT_FAIL(HOT_ERR_ARG, "hot_gemm_i8_grouped: null pointer");
  if (M <= 0 || N <= 0 || groups <= 0 || group_k <= 0 || M > (1 << 30) || N > (1 << 30) || groups * group_k > (1 << 30) || len < 1 || len > group_k)
    HOT_FAIL(HOT_ERR_ARG, "hot_gemm_i8_grouped: bad shape M=%lld N=%lld groups=%lld group_k=%lld", (long long)M, (long long)N,
             (long long)groups, (long long)group_k);
  if (group_k % kBK != 0)
    HOT_FAIL(HOT_ERR_UNSUPPORTED, "hot_gemm_i8_grouped: group_k %lld must be a multiple of %d (pad each group with zero codes)",
             (long long)group_k, kBK);
  const int64_t K = groups * group_k;
  if (lda % 16 || ldb % 16 || lda < K || ldb < K || ((uintptr_t)a) % 16 || ((uintptr_t)b) % 16)
    HOT_FAIL(HOT_ERR_ARG, "hot_gemm_i8_grouped: operand base and pitch must be 16-byte aligned and cover groups * group_k");
  if (out_dtype != HOT_F32 && out_dtype != HOT_BF16) HOT_FAIL(HOT_ERR_UNSUPPORTED, "hot_gemm_i8_grouped: out dtype %d", out_dtype);
  const int64_t esz = out_dtype == HOT_BF16 ? 2 : 4;
  if (ldo < N || ((uintptr_t)out) % 16 != 0 || (ldo * esz) % 16 != 0)
    HOT_FAIL(HOT_ERR_ARG, "hot_gemm_i8_grouped: out and its pitch must be 16-byte aligned, ldo >= N");
  const int sms = device_sm_count();
  if (sms <= 0) return HOT_ERR_CUDA;
  GroupedParams p = {};
  p.M = (int)M;
  p.N = (int)N;
  p.groups = (int)groups;
  p.blocks = (int)(group_k / kBK);
  const int64_t rest = len - (p.blocks - 1) * (int64_t)kBK;  // codes in a sample's last k-block; its padding is not multiplied
  p.last_steps = rest < 1 ? 1 : (int)((rest + 31) / 32);
  p.sa = scale_a;
  p.sb = scale_b;
  p.sa_row = scale_a_per_row ? 1 : 0;
  p.post = post;
  p.one = 1.0f;
  p.out16 = out_dtype == HOT_BF16;
  p.status = status_word;
  p.wait_ns = wait_limit_ns();
  // Tile width: rounds of tiles per SM times a sample's time in a tile, in cycles: its k-blocks or the drain of its
  // accumulators, whichever is longer (of equals the wider, which reads A less often).
  int bn = 128;
  double best = -1.0;
  for (int w : {128, 96, 64, 32}) {
    const int64_t tiles = (M + kBM - 1) / kBM * ((N + w - 1) / w);
    const double mma = p.blocks * (80.0 + 4 * (w > 64 ? w / 2 : 32)), drain = 200.0 + 3.6 * w;
    const double t = (double)((tiles + sms - 1) / sms) * (mma > drain ? mma : drain);
    if (best < 0 || t < 0.98 * best) {
      best = t;
      bn = w;
    }
  }
  cudaStream_t st = (cudaStream_t)stream;
  switch (bn) {
    case 128: return launch<128>(a, lda, b, ldb, out, ldo, K, p, sms, st);
    case 96: return launch<96>(a, lda, b, ldb, out, ldo, K, p, sms, st);
    case 64: return launch<64>(a, lda, b, ldb, out, ldo, K, p, sms, st);
    default: return launch<32>(a, lda, b, ldb, out, ldo, K, p, sms, st);
  }
}

}  // namespace hot

extern "C" int hot_gemm_i8_grouped(const void* a, int64_t lda, const void* b, int64_t ldb, int64_t M, int64_t N, int64_t groups,
                                   int64_t group_k, const float* scale_a, int scale_a_per_row, const float* scale_b, float post, void* out,
                                   int out_dtype, int64_t ldo, uint32_t* status_word, hot_stream_t stream) {
  return hot::gemm_i8_grouped(a, lda, b, ldb, M, N, groups, group_k, group_k, scale_a, scale_a_per_row, scale_b, post, out, out_dtype, ldo,
                              status_word, stream);
}
