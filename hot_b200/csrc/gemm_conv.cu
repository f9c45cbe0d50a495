// Input gradient of a convolution of stride 1 from the codes of grad_output and of the kernel, folded as it is made:
//   grad_x[b, c, h, w] = (sum over taps (i, j) and channels o of  q_go[b, h + ph - i dh, w + pw - j dw, o] * q_w[c, (i, j), o]) * s_go[b] * s_w * post
//
// The product over unfolded rows writes kh * kw values per input element, which a fold then adds up.  All of them carry the same pair
// of scales, so the sum may as well be the contraction: one integer product whose K runs over the taps too, and which leaves
// nothing to fold.  A tile is 128 (or fewer) input positions of one image, whole rows where they fit, by up to 256 channels; for every tap
// the bulk copy fetches the grad_output rows of those positions moved by the tap, with zeros for what lies outside the image, and the kernel's
// rows of that tap, c * kh * kw + tap, are a dimension of their tensor map.  The integer sums are exact and round once, where the taps
// used to round one by one before they were added.
//
// What bounds it: the fill of shared memory (32 to 48 KB per tap and 128 outputs, 200 to 330 ns), and for few channels the start and
// the drain.  32 x 128 x 28 x 28, 3 x 3, 128 outputs, bf16: 15 us, where the product over unfolded rows and the fold took 19 and 27; tiles
// of 128 channels at most made the step of 64 x 256 x 56 x 56 to 512, 1 x 1, 1223 us, 256 make it 1209 (1213 with product and fold).
#include <cstring>

#include "layer.cuh"
#include "tc.cuh"

namespace hot {

int device_sm_count();

namespace {

constexpr int kBM = 128, kBK = 128, kMaxBN = 256;
constexpr int kStages = 4, kStageA = kBM * kBK, kStageB = kMaxBN * kBK;
constexpr int kEpiWarps = 8, kThreads = (kEpiWarps + 2) * 32;
constexpr int kOffB = kStages * kStageA, kOffBar = kOffB + kStages * kStageB;
constexpr int kSmem = kOffBar + 256 + 1024;
constexpr uint32_t kTmemCols = 2 * kMaxBN;

struct FoldParams {
  int H, W, C;
  int bw, bh;               // positions of a tile: bw columns of bh rows
  int tw, th;               // tiles across an image, and down
  int n_tiles, num_tiles, bn;
  int kh, kw, dh, dw, ph, pw;
  int kblocks, last_steps;  // k-blocks of a tap; instructions of 32 in the last of them
  FastDiv by_n, by_tw, by_th, by_bw;
  uint32_t tx;              // bytes of a stage
  const float* sa;
  int sa_batch;             // one scale per image
  const float* sb;
  float post;
  void* out;
  int out16;
  uint32_t* status;
  uint64_t wait_ns;
};

__device__ __forceinline__ void tma_load_3d(void* dst, const CUtensorMap* map, uint64_t* bar, int c0, int c1, int c2) {
  asm volatile("cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5}], [%2];" ::"r"(smem_u32(dst)),
               "l"(reinterpret_cast<uint64_t>(map)), "r"(smem_u32(bar)), "r"(c0), "r"(c1), "r"(c2)
               : "memory");
}
__device__ __forceinline__ void tma_load_4d(void* dst, const CUtensorMap* map, uint64_t* bar, int c0, int c1, int c2, int c3) {
  asm volatile("cp.async.bulk.tensor.4d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5, %6}], [%2];" ::"r"(smem_u32(dst)),
               "l"(reinterpret_cast<uint64_t>(map)), "r"(smem_u32(bar)), "r"(c0), "r"(c1), "r"(c2), "r"(c3)
               : "memory");
}

struct FoldTile {
  int b, h0, w0, n0;
  __device__ __forceinline__ FoldTile(const FoldParams& p, int tile) {
    const int m = tile / p.by_n, row = m / p.by_tw;
    b = row / p.by_th;
    n0 = (tile - m * p.n_tiles) * p.bn;
    w0 = (m - row * p.tw) * p.bw;
    h0 = (row - b * p.th) * p.bh;
  }
};

__global__ void __launch_bounds__(kThreads, 1)
    conv_fold_kernel(const __grid_constant__ CUtensorMap tma_a, const __grid_constant__ CUtensorMap tma_b, const __grid_constant__ FoldParams p) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = smem_raw + ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u);
  uint64_t* full = reinterpret_cast<uint64_t*>(smem + kOffBar);
  uint64_t* empty = full + kStages;
  uint64_t* tmem_full = empty + kStages;  // [2] a tile's accumulator is complete
  uint64_t* tmem_empty = tmem_full + 2;   // [2] drained
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(tmem_empty + 2);
  volatile uint32_t* abort_flag = tmem_slot + 1;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  constexpr int kProducer = kEpiWarps, kMma = kProducer + 1;

  if (threadIdx.x == 0) {
    for (int s = 0; s < kStages; ++s) {
      mbar_init(&full[s], 1);
      mbar_init(&empty[s], 1);
    }
    for (int b = 0; b < 2; ++b) {
      mbar_init(&tmem_full[b], 1);
      mbar_init(&tmem_empty[b], kEpiWarps);
    }
    *abort_flag = 0u;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    tma_prefetch_desc(&tma_a);
    tma_prefetch_desc(&tma_b);
  }
  if (warp == kMma) tmem_alloc(tmem_slot, kTmemCols);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  // launched as a programmatic dependent: the set-up above ran while the kernel before it drained
  asm volatile("griddepcontrol.wait;" ::: "memory");
  const uint32_t tmem_base = *tmem_slot;
  const int taps = p.kh * p.kw;

  if (warp == kProducer) {
    if (elect_one()) {
      uint32_t s = 0, ph = 0;
      bool ok = true;
      for (int tile = blockIdx.x; ok && tile < p.num_tiles; tile += gridDim.x) {
        const FoldTile t(p, tile);
        int i = 0, j = 0;
        for (int tap = 0; ok && tap < taps; ++tap) {
          for (int kb = 0; kb < p.kblocks; ++kb, s = (s + 1 == kStages ? 0 : s + 1), ph ^= (s == 0 ? 1u : 0u)) {
            ok = mbar_wait(&empty[s], ph ^ 1u, abort_flag, p.wait_ns);
            if (!ok) break;
            mbar_expect_tx(&full[s], p.tx);
            tma_load_4d(smem + s * kStageA, &tma_a, &full[s], kb * kBK, t.w0 + p.pw - j * p.dw, t.h0 + p.ph - i * p.dh, t.b);
            tma_load_3d(smem + kOffB + s * kStageB, &tma_b, &full[s], kb * kBK, tap, t.n0);
          }
          if (++j == p.kw) {
            j = 0;
            ++i;
          }
        }
      }
    }
  } else if (warp == kMma) {
    if (elect_one()) {
      const uint32_t idesc = instr_desc_i8(p.bn);
      const uint32_t hi = (uint32_t)(smem_desc_sw128(0) >> 32);
      const uint32_t a_lo0 = (uint32_t)smem_desc_sw128(smem_u32(smem)), b_lo0 = (uint32_t)smem_desc_sw128(smem_u32(smem + kOffB));
      uint32_t s = 0, ph = 0, it = 0;
      bool ok = true;
      for (int tile = blockIdx.x; ok && tile < p.num_tiles; tile += gridDim.x, ++it) {
        const uint32_t buf = it & 1u, bph = (it >> 1) & 1u;
        ok = mbar_wait(&tmem_empty[buf], bph ^ 1u, abort_flag, p.wait_ns);
        if (!ok) break;
        tc_fence_after();
        const uint32_t d = tmem_base + buf * kMaxBN;
        uint32_t accumulate = 0u;
        for (int tap = 0; ok && tap < taps; ++tap)
          for (int kb = 0; kb < p.kblocks; ++kb, s = (s + 1 == kStages ? 0 : s + 1), ph ^= (s == 0 ? 1u : 0u)) {
            ok = mbar_wait(&full[s], ph, abort_flag, p.wait_ns);
            if (!ok) break;
            tc_fence_after();
            const uint32_t a_lo = a_lo0 + s * (uint32_t)(kStageA >> 4), b_lo = b_lo0 + s * (uint32_t)(kStageB >> 4);
            const int steps = kb + 1 == p.kblocks ? p.last_steps : kBK / 32;
#pragma unroll
            for (int k = 0; k < kBK / 32; ++k)
              if (k < steps) {
                umma_i8(d, ((uint64_t)hi << 32) | (a_lo + 2u * k), ((uint64_t)hi << 32) | (b_lo + 2u * k), idesc, accumulate);
                accumulate = 1u;
              }
            umma_commit(&empty[s]);
          }
        if (ok) umma_commit(&tmem_full[buf]);
      }
    }
  } else {
    const int q = warp & 3, team = warp >> 2;  // tensor-memory lane quarter; of the chunks of 32 channels, the even or the odd ones
    const int m = q * 32 + lane, hh = m / p.by_bw, ww = m - hh * p.bw;
    const int chunks = p.bn / 32;
    const int64_t plane = (int64_t)p.H * p.W;
    const float sb = __ldg(p.sb);
    uint32_t it = 0;
    bool ok = true;
    for (int tile = blockIdx.x; ok && tile < p.num_tiles; tile += gridDim.x, ++it) {
      const FoldTile t(p, tile);
      const uint32_t buf = it & 1u, bph = (it >> 1) & 1u;
      const float sa = __ldg(p.sa + (p.sa_batch ? t.b : 0));
      ok = __all_sync(0xFFFFFFFFu, mbar_wait_parked(&tmem_full[buf], bph, abort_flag, p.wait_ns)) != 0;
      if (!ok) break;
      tc_fence_after();
      const bool inside = hh < p.bh && t.h0 + hh < p.H && t.w0 + ww < p.W;
      const int64_t at = ((int64_t)t.b * p.C + t.n0) * plane + (int64_t)(t.h0 + hh) * p.W + t.w0 + ww;
      for (int c = team; c < chunks; c += 2) {
        uint32_t acc[32];
        tmem_ld32(tmem_base + buf * kMaxBN + ((uint32_t)(q * 32) << 16) + c * 32, acc);
        if (!inside) continue;
        const int left = p.C - t.n0 - c * 32;  // channels from this chunk on
        auto value = [&](int i) { return __fmul_rn(__fmul_rn(__fmul_rn((float)(int)acc[i], sa), sb), p.post); };
        if (p.out16) {
          __nv_bfloat16* o = reinterpret_cast<__nv_bfloat16*>(p.out) + at + (int64_t)(c * 32) * plane;
#pragma unroll
          for (int i = 0; i < 32; ++i, o += plane)
            if (i < left) *o = __float2bfloat16_rn(value(i));
        } else {
          float* o = reinterpret_cast<float*>(p.out) + at + (int64_t)(c * 32) * plane;
#pragma unroll
          for (int i = 0; i < 32; ++i, o += plane)
            if (i < left) *o = value(i);
        }
      }
      tc_fence_before();
      __syncwarp();
      if (elect_one()) mbar_arrive(&tmem_empty[buf]);
    }
  }

  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  tc_fence_before();
  __syncthreads();
  if (warp == kMma) {
    tc_fence_after();
    tmem_dealloc(tmem_base, kTmemCols);
  }
  if (threadIdx.x == 0 && *abort_flag) {
    if (p.status) atomicOr(p.status, (uint32_t)HOT_STATUS_GEMM);
    const uint64_t t0 = global_timer_ns();  // let bulk copies already issued land before exit
    while (global_timer_ns() - t0 < 100000ull) {
    }
  }
}

}  // namespace

// Whether conv_grad_input makes the input gradient: stride 1, one scale for the codes of an image, one byte per code, sums that 32 bits
// hold.  (A dilation wider than the output leaves positions that no tap reaches, which have to be 0 whatever the scales.)
bool conv_fold_covered(const hot_layer_t& l, const hot_conv_t& v) {
  const hot_linear_cfg_t& c = l.cfg;
  if (v.B <= 0 || v.C <= 0 || v.H <= 0 || v.W <= 0 || v.kh <= 0 || v.kw <= 0 || v.dh <= 0 || v.dw <= 0 || v.ph < 0 || v.pw < 0 || v.dtype != c.dtype ||
      l.O <= 0 || c.q_w.bits < 2 || c.q_w.bits > 8)
    return false;
  if (v.sh != 1 || v.sw != 1 || c.q_gx.scale_mode != HOT_SCALE_TENSOR || c.q_gx.storage != HOT_STORE_INT8) return false;
  const int64_t oh = v.H + 2 * v.ph - (int64_t)v.dh * (v.kh - 1), ow = v.W + 2 * v.pw - (int64_t)v.dw * (v.kw - 1);
  if (oh < v.dh || ow < v.dw || oh > (1 << 20) || ow > (1 << 20) || v.H > (1 << 20) || v.W > (1 << 20) || v.C > (1 << 20) || v.B > 65535) return false;
  const int64_t k = l.O * (int64_t)v.kh * v.kw;
  return k * 128 * ((1ll << (c.q_w.bits - 1)) - 1) < (1ll << 31) && v.kh * (int64_t)v.kw <= 4096 && l.I == (int64_t)v.C * v.kh * v.kw &&
         (l.batch ? l.batch == v.B && l.L == oh * ow : l.L == v.B * oh * ow);
}

int conv_grad_input(const hot_layer_t& l, const hot_conv_t& v, const void* q_go, int64_t ld_go, const float* s_go, const void* q_w, int64_t ld_w,
                    const float* s_w, float post, void* out, uint32_t* status, cudaStream_t st) {
  if (!conv_fold_covered(l, v)) HOT_FAIL(HOT_ERR_UNSUPPORTED, "hot_layer_backward_conv: this convolution's input gradient is not folded here");
  const int64_t oh = v.H + 2 * v.ph - (int64_t)v.dh * (v.kh - 1), ow = v.W + 2 * v.pw - (int64_t)v.dw * (v.kw - 1), taps = (int64_t)v.kh * v.kw;
  const int sms = device_sm_count();
  if (sms <= 0) return HOT_ERR_CUDA;
  FoldParams p;
  memset(&p, 0, sizeof(p));
  p.H = (int)v.H;
  p.W = (int)v.W;
  p.C = (int)v.C;
  // a tile: as many whole rows as 128 positions hold, evened out over the image, or a stretch of one row
  p.bw = p.W < kBM ? p.W : kBM;
  int rows = kBM / p.bw;
  if (rows > p.H) rows = p.H;
  p.th = (p.H + rows - 1) / rows;
  p.bh = (p.H + p.th - 1) / p.th;
  p.tw = (p.W + p.bw - 1) / p.bw;
  // channels: up to 256, fewer where that leaves SMs idle
  const int64_t m_tiles = (int64_t)v.B * p.th * p.tw;
  p.bn = p.C >= kMaxBN ? kMaxBN : (p.C + 31) / 32 * 32;
  while (p.bn > 32 && m_tiles * ((p.C + p.bn - 1) / p.bn) < sms) p.bn = (p.bn / 2 + 31) / 32 * 32;
  p.n_tiles = (p.C + p.bn - 1) / p.bn;
  if (m_tiles * p.n_tiles >= (1ll << 30)) HOT_FAIL(HOT_ERR_UNSUPPORTED, "hot_layer_backward_conv: too many tiles");
  p.num_tiles = (int)(m_tiles * p.n_tiles);
  p.kh = v.kh; p.kw = v.kw; p.dh = v.dh; p.dw = v.dw; p.ph = v.ph; p.pw = v.pw;
  p.kblocks = (int)((l.O + kBK - 1) / kBK);
  p.last_steps = (int)((l.O - (int64_t)(p.kblocks - 1) * kBK + 31) / 32);
  p.by_n = fast_div(p.n_tiles);
  p.by_tw = fast_div(p.tw);
  p.by_th = fast_div(p.th);
  p.by_bw = fast_div(p.bw);
  p.tx = (uint32_t)((p.bw * p.bh + p.bn) * kBK);
  p.sa = s_go;
  p.sa_batch = l.batch > 0;
  p.sb = s_w;
  p.post = post;
  p.out = out;
  p.out16 = l.cfg.dtype == HOT_BF16;
  p.status = status;
  p.wait_ns = wait_limit_ns();
  CUtensorMap ma, mb;
  const int64_t da[4] = {l.O, ow, oh, v.B}, sa[3] = {ld_go, ld_go * ow, ld_go * ow * oh};
  const int ba[4] = {kBK, p.bw, p.bh, 1};
  if (int rc = make_map_nd(&ma, q_go, 4, da, sa, ba)) return rc;
  const int64_t db[3] = {l.O, taps, v.C}, sb[2] = {ld_w, ld_w * taps};
  const int bb[3] = {kBK, 1, p.bn};
  if (int rc = make_map_nd(&mb, q_w, 3, db, sb, bb)) return rc;
  static PerDeviceOnce once;
  bool done = false;
  const int dev = once.current(&done);
  if (dev < 0) HOT_FAIL(HOT_ERR_CUDA, "hot_layer_backward_conv: cannot query the current CUDA device");
  if (!done) {
    HOT_CUDA(cudaFuncSetAttribute(conv_fold_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmem));
    once.mark(dev);
  }
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)(p.num_tiles < sms ? p.num_tiles : sms));
  cfg.blockDim = dim3(kThreads);
  cfg.dynamicSmemBytes = kSmem;
  cfg.stream = st;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  HOT_CUDA(cudaLaunchKernelEx(&cfg, conv_fold_kernel, ma, mb, p));
  return HOT_OK;
}

}  // namespace hot

extern "C" int hot_conv_folds(const hot_layer_t* layer, const hot_conv_t* conv) {
  return layer && conv && hot::conv_fold_covered(*layer, *conv) ? 1 : 0;
}
