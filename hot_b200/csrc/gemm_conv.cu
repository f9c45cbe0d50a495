// Input gradient of a convolution of stride 1 from the codes of grad_output and of the kernel, folded as it is made:
//   grad_x[b, c, h, w] = sum over taps (i, j) of round(s_go[b] * s_w * post * sum over o of  q_go[b, h + ph - i dh, w + pw - j dw, o] * q_w[c, (i, j), o])
//
// The product over unfolded rows writes kh * kw values per input element, which a fold then reads and adds up.  Here a tile is 128 (or
// fewer) input positions, several images where they are small, by up to 128 channels; for every tap the bulk copy fetches the
// grad_output rows of those positions moved by the tap, with zeros for what lies outside the image, and the kernel's rows of that tap,
// c * kh * kw + tap, are a dimension of their tensor map.  A tap's integer sums are complete in a tensor-memory buffer of their own; the
// epilogue scales and rounds them to the tensors' type as the product over rows would and adds them to its registers in the fold's order, so
// that the result is, bit for bit, what product and fold give (also for scales and gradients that overflow or are infinite): which way a
// size goes, or whether a layer runs natively, changes no value.  Convolutions of one tap keep no sums and take up to 256 channels.
//
// What bounds it: the epilogue (five instructions a value and tap and the conversions; some 550 ns for a tap of 128 x 128), then the fill of
// shared memory (32 KB per tap and 128 outputs, 250 to 330 ns).  The whole training step in bf16, product and fold against this: 32 x 128 x
// 28 x 28, 3 x 3, to 128 outputs 202 and 156 us; 64 x 512 x 7 x 7, 3 x 3, to 512 169 and 144 (tiles of one image: 155); 256 x 2048 x 4 x 4, 1 x 1,
// to 512 341 and 317 (one image: 404); 32 x 256 x 56 x 56, 1 x 1, to 64 369 and 308.  Sixteen warps in the epilogue, chunks of 16 channels, or
// integers converted by an addition were 0 to 6 % slower.  (Summing the taps as integers, rounded once, takes 152 us in the first and
// gives other values.)
#include <cmath>
#include <cstring>
#include <type_traits>

#include "layer.cuh"
#include "tc.cuh"

namespace hot {

int device_sm_count();

namespace {

constexpr int kBM = 128, kBK = 128;
constexpr int kEpiWarps = 8, kTeams = kEpiWarps / 4, kThreads = (kEpiWarps + 2) * 32;
constexpr uint32_t kTmemCols = 512;

// What the choice of a tile, and the choice between this kernel and the product over rows, reckon with (measured): a 128-byte row to shared memory,
// a tap's channel out of tensor memory, for one tap with its store, what a launch takes besides; the two launches over rows, a byte of
// theirs written by the product and read by the fold, a CTA of the fold.
constexpr double kRowNs = 1.05, kDrainNs = 4.7, kDrainOneNs = 3.0, kFoldNs = 4000.0, kRowsNs = 5000.0, kWriteNs = 1 / 3000.0, kReadNs = 1 / 2100.0, kCtaNs = 2.5;
// The product over rows is taken where this kernel would take clearly longer: few tiles of many outputs, whose k-blocks follow one another (the whole
// step of 16 x 64 x 14 x 14, 3 x 3, to 1024, bf16: 83.5 us, 75.6 by product and fold; 1 x 512 x 7 x 7 to 512 51.4 and 47.8).
constexpr double kFoldOver = 1.25;

// ONE: convolutions of one tap
template <bool ONE>
struct Layout {
  static constexpr int kMaxBN = ONE ? 256 : 128;
  static constexpr int kBufs = (int)kTmemCols / kMaxBN;  // accumulators in tensor memory
  static constexpr int kStageA = kBM * kBK, kStageB = kMaxBN * kBK, kStages = ONE ? 4 : 6;
  static constexpr int kOffB = kStages * kStageA, kOffBar = kOffB + kStages * kStageB;
  static constexpr int kSmem = kOffBar + 256 + 1024;
};

struct FoldParams {
  int B, H, W, C;
  int bw, bh, nb;           // positions of a tile: bw columns of bh rows of nb images
  int tw, th;               // tiles across an image, and down
  int n_tiles, num_tiles, bn;
  int OH, OW, kh, kw, dh, dw, ph, pw;
  int kblocks, last_steps;  // k-blocks of a tap; instructions of 32 in the last of them
  FastDiv by_n, by_tw, by_th, by_bw, by_image;  // (by_image: positions of a tile in one image)
  uint32_t tx;              // bytes of a stage
  const float* sa;
  int sa_batch;             // one scale per image
  const float* sb;
  float post;
  int lean;                 // post goes with sb, as in the product over rows whose output begins on 16-byte pieces
  float one;                // 1, in a place where the compiler does not see it
  void* out;
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
    const int images = row / p.by_th;
    b = images * p.nb;
    n0 = (tile - m * p.n_tiles) * p.bn;
    w0 = (m - row * p.tw) * p.bw;
    h0 = (row - images * p.th) * p.bh;
  }
};

template <bool ONE, bool OUT16>
__global__ void __launch_bounds__(kThreads, 1)
    conv_fold_kernel(const __grid_constant__ CUtensorMap tma_a, const __grid_constant__ CUtensorMap tma_b, const __grid_constant__ FoldParams p) {
  using L = Layout<ONE>;
  constexpr int kStages = L::kStages, kStageA = L::kStageA, kStageB = L::kStageB, kOffB = L::kOffB, kBufs = L::kBufs;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = smem_raw + ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u);
  uint64_t* full = reinterpret_cast<uint64_t*>(smem + L::kOffBar);
  uint64_t* empty = full + kStages;
  uint64_t* tmem_full = empty + kStages;     // [kBufs] a tap's sums are complete
  uint64_t* tmem_empty = tmem_full + kBufs;  // [kBufs] drained
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(tmem_empty + kBufs);
  volatile uint32_t* abort_flag = tmem_slot + 1;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  constexpr int kProducer = kEpiWarps, kMma = kProducer + 1;

  if (threadIdx.x == 0) {
    for (int s = 0; s < kStages; ++s) {
      mbar_init(&full[s], 1);
      mbar_init(&empty[s], 1);
    }
    for (int b = 0; b < kBufs; ++b) {
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
        int i = p.kh - 1, j = p.kw - 1;  // (the fold adds ascending output positions)
        for (int tap = taps - 1; ok && tap >= 0; --tap) {
          for (int kb = 0; kb < p.kblocks; ++kb, s = (s + 1 == kStages ? 0 : s + 1), ph ^= (s == 0 ? 1u : 0u)) {
            ok = mbar_wait(&empty[s], ph ^ 1u, abort_flag, p.wait_ns);
            if (!ok) break;
            mbar_expect_tx(&full[s], p.tx);
            tma_load_4d(smem + s * kStageA, &tma_a, &full[s], kb * kBK, t.w0 + p.pw - j * p.dw, t.h0 + p.ph - i * p.dh, t.b);
            tma_load_3d(smem + kOffB + s * kStageB, &tma_b, &full[s], kb * kBK, tap, t.n0);
          }
          if (--j < 0) {
            j = p.kw - 1;
            --i;
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
      for (int tile = blockIdx.x; ok && tile < p.num_tiles; tile += gridDim.x)
        for (int tap = 0; ok && tap < taps; ++tap, ++it) {
          const uint32_t buf = it % kBufs, bph = (it / kBufs) & 1u;
          ok = mbar_wait(&tmem_empty[buf], bph ^ 1u, abort_flag, p.wait_ns);
          if (!ok) break;
          tc_fence_after();
          const uint32_t d = tmem_base + buf * L::kMaxBN;
          for (int kb = 0; kb < p.kblocks; ++kb, s = (s + 1 == kStages ? 0 : s + 1), ph ^= (s == 0 ? 1u : 0u)) {
            ok = mbar_wait(&full[s], ph, abort_flag, p.wait_ns);
            if (!ok) break;
            tc_fence_after();
            const uint32_t a_lo = a_lo0 + s * (uint32_t)(kStageA >> 4), b_lo = b_lo0 + s * (uint32_t)(kStageB >> 4);
            const int steps = kb + 1 == p.kblocks ? p.last_steps : kBK / 32;
#pragma unroll
            for (int k = 0; k < kBK / 32; ++k)
              if (k < steps) umma_i8(d, ((uint64_t)hi << 32) | (a_lo + 2u * k), ((uint64_t)hi << 32) | (b_lo + 2u * k), idesc, kb > 0 || k > 0 ? 1u : 0u);
            umma_commit(&empty[s]);
          }
          if (ok) umma_commit(&tmem_full[buf]);
        }
    }
  } else {
    const int q = warp & 3, team = warp >> 2;  // tensor-memory lane quarter; share of the tile's columns
    const int m = q * 32 + lane, image = m / p.by_image, pos = m - image * (p.bw * p.bh), hh = pos / p.by_bw, ww = pos - hh * p.bw;
    const int per = (p.bn / 32 + kTeams - 1) / kTeams, first = team * per, mine = min(per, p.bn / 32 - first);  // this warp's chunks of 32 channels
    constexpr int kChunks = L::kMaxBN / (32 * kTeams), kSums = ONE ? 1 : kChunks;
    const int64_t plane = (int64_t)p.H * p.W;
    const float sb = load_result(p.sb), fb = p.lean ? __fmul_rn(sb, p.post) : sb;
    const float2 post2 = make_float2(p.post, p.post), one2 = make_float2(p.one, p.one);
    uint32_t it = 0;
    bool ok = true;
    for (int tile = blockIdx.x; ok && tile < p.num_tiles; tile += gridDim.x) {
      const FoldTile t(p, tile);
      const int b = t.b + image, h = t.h0 + hh, w = t.w0 + ww;
      const bool inside = image < p.nb && b < p.B && h < p.H && w < p.W;
      const float sa = load_result(p.sa + (p.sa_batch && inside ? b : 0));
      const int64_t at = ((int64_t)b * p.C + t.n0) * plane + (int64_t)h * p.W + w;
      float2 sum[kSums][16];
      auto open = [&](float2 (&v)[16]) {
#pragma unroll
        for (int i = 0; i < 16; ++i) v[i] = make_float2(0.0f, 0.0f);
      };
      // one tap of 32 channels: scaled and rounded as the product over rows stores it, then added.  (A tap outside the output has sums of
      // zero and comes with scales of zero: it adds nothing.)
      auto add = [&](auto lean, float2 (&v)[16], const uint32_t (&acc)[32], float ta, float tb) {
        const float2 fa2 = make_float2(ta, ta), fb2 = make_float2(tb, tb);
#pragma unroll
        for (int i = 0; i < 16; ++i) {
          float2 f = __fmul2_rn(__fmul2_rn(make_float2((float)(int)acc[2 * i], (float)(int)acc[2 * i + 1]), fa2), fb2);
          if (!decltype(lean)::value) f = __fmul2_rn(f, post2);
          if (OUT16) {
            const __nv_bfloat162 r = __floats2bfloat162_rn(f.x, f.y);
            const uint32_t bits = *reinterpret_cast<const uint32_t*>(&r);
            v[i] = add2(v[i], make_float2(__uint_as_float(bits << 16), __uint_as_float(bits & 0xFFFF0000u)));
          } else {
            v[i] = __ffma2_rn(f, one2, v[i]);  // (as an addition it would be joined with the product before it)
          }
        }
      };
      auto store = [&](const float2 (&v)[16], int c) {
        const int left = p.C - t.n0 - c * 32;  // channels from this chunk on
        if (OUT16) {
          __nv_bfloat16* o = reinterpret_cast<__nv_bfloat16*>(p.out) + at + (int64_t)(c * 32) * plane;
#pragma unroll
          for (int i = 0; i < 32; ++i, o += plane)
            if (i < left) *o = __float2bfloat16_rn(i & 1 ? v[i / 2].y : v[i / 2].x);
        } else {
          float* o = reinterpret_cast<float*>(p.out) + at + (int64_t)(c * 32) * plane;
#pragma unroll
          for (int i = 0; i < 32; ++i, o += plane)
            if (i < left) *o = i & 1 ? v[i / 2].y : v[i / 2].x;
        }
      };
      // the sum of one tap in 16 bits: rounded, and 0 in place of -0
      auto store_one = [&](const uint32_t (&acc)[32], float ta, float tb, int c) {
        const int left = p.C - t.n0 - c * 32;
        const float2 fa2 = make_float2(ta, ta), fb2 = make_float2(tb, tb);
        const __nv_bfloat162 zero = __nv_bfloat162(__ushort_as_bfloat16(0), __ushort_as_bfloat16(0));
        __nv_bfloat16* o = reinterpret_cast<__nv_bfloat16*>(p.out) + at + (int64_t)(c * 32) * plane;
#pragma unroll
        for (int i = 0; i < 16; ++i) {
          float2 f = __fmul2_rn(__fmul2_rn(make_float2((float)(int)acc[2 * i], (float)(int)acc[2 * i + 1]), fa2), fb2);
          if (!p.lean) f = __fmul2_rn(f, post2);
          const __nv_bfloat162 r = __hadd2_rn(__floats2bfloat162_rn(f.x, f.y), zero);
          if (2 * i < left) *o = __low2bfloat16(r);
          o += plane;
          if (2 * i + 1 < left) *o = __high2bfloat16(r);
          o += plane;
        }
      };
      if (!ONE)
#pragma unroll
        for (int k = 0; k < kSums; ++k) open(sum[k]);
      int oh = h + p.ph - (p.kh - 1) * p.dh, ow0 = w + p.pw - (p.kw - 1) * p.dw, ow = ow0, j = p.kw;
      for (int tap = 0; tap < taps; ++tap, ++it) {
        const uint32_t buf = it % kBufs, bph = (it / kBufs) & 1u;
        const bool reached = (unsigned)oh < (unsigned)p.OH && (unsigned)ow < (unsigned)p.OW;
        const float ta = reached ? sa : 0.0f, tb = reached ? fb : 0.0f;
        ok = __all_sync(0xFFFFFFFFu, mbar_wait_parked(&tmem_full[buf], bph, abort_flag, p.wait_ns)) != 0;
        if (!ok) break;
        tc_fence_after();
#pragma unroll
        for (int k = 0; k < kChunks; ++k)
          if (k < mine) {  // (the same in every lane of the warp)
            uint32_t acc[32];
            __syncwarp();
            tmem_ld32(tmem_base + buf * L::kMaxBN + ((uint32_t)(q * 32) << 16) + (first + k) * 32, acc);
            if (ONE && OUT16) {
              if (inside) store_one(acc, ta, tb, first + k);
              continue;
            }
            if (ONE) open(sum[0]);
            if (p.lean) add(std::true_type(), sum[ONE ? 0 : k], acc, ta, tb);
            else add(std::false_type(), sum[ONE ? 0 : k], acc, ta, tb);
            if (ONE && inside) store(sum[0], first + k);
          }
        tc_fence_before();
        __syncwarp();
        if (elect_one()) mbar_arrive(&tmem_empty[buf]);
        ow += p.dw;
        if (--j == 0) {
          j = p.kw;
          ow = ow0;
          oh += p.dh;
        }
      }
      if (!ONE && ok && inside) {
#pragma unroll
        for (int k = 0; k < kSums; ++k)
          if (k < mine) store(sum[k], first + k);
      }
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

// How the positions and channels are cut into tiles, and how long that takes.
struct FoldPlan {
  int bw, bh, nb, tw, th, bn, n_tiles;
  int64_t m_tiles;
  double ns;
};

// A tile: several whole images where 128 positions hold them, else what needs fewest tiles of an image among whole rows and rows in up to
// eight more stretches than they must be cut into, evened out over the image and the batch.  Channels: what takes the busiest SM least.
FoldPlan plan_fold(const hot_layer_t& l, const hot_conv_t& v, int sms) {
  FoldPlan f = {};
  const int taps = v.kh * v.kw, kblocks = (int)((l.O + kBK - 1) / kBK);
  int64_t image_tiles = 0;
  for (int cut = (v.W + kBM - 1) / kBM, last = cut + 8; cut <= last && cut <= v.W; ++cut) {
    const int bw = (v.W + cut - 1) / cut, tw = (v.W + bw - 1) / bw, rows = kBM / bw < v.H ? kBM / bw : v.H, th = (v.H + rows - 1) / rows;
    if (image_tiles && (int64_t)tw * th >= image_tiles) continue;
    image_tiles = (int64_t)tw * th;
    f.bw = bw;
    f.tw = tw;
    f.th = th;
    f.bh = (v.H + th - 1) / th;
  }
  f.nb = image_tiles == 1 ? kBM / (v.W * v.H) : 1;
  if (f.nb > v.B) f.nb = v.B;
  const int64_t batches = (v.B + f.nb - 1) / f.nb;
  f.nb = (int)((v.B + batches - 1) / batches);
  f.m_tiles = batches * image_tiles;
  const int most = taps == 1 ? Layout<true>::kMaxBN : Layout<false>::kMaxBN;
  for (int n = (v.C + most - 1) / most, bn_last = 0; bn_last != 32; ++n) {
    const int bn = ((v.C + n - 1) / n + 31) / 32 * 32, n_tiles = (v.C + bn - 1) / bn;
    if (bn == bn_last) continue;
    bn_last = bn;
    // a tap's copies, or its way out of tensor memory, whichever takes longer; the last one's way out is nobody's cover
    const double copies = kblocks * (kBM + bn) * kRowNs, drain = bn * (taps == 1 ? kDrainOneNs : kDrainNs);
    const double ns = (double)((f.m_tiles * n_tiles + sms - 1) / sms) * taps * (copies > drain ? copies : drain) + drain + kFoldNs;
    if (f.ns && ns >= 0.95 * f.ns) continue;  // (narrower tiles fetch the positions once more each)
    f.ns = ns;
    f.bn = bn;
    f.n_tiles = n_tiles;
  }
  return f;
}

// The same gradient by the product over unfolded rows, tiles of 128 x 256 or the writing of them, and by hot_col2im, which reads them again,
// an image and a few channels to a CTA.
double rows_ns(const hot_layer_t& l, const hot_conv_t& v, int sms) {
  const int taps = v.kh * v.kw, size = v.dtype == HOT_BF16 ? 2 : 4, channels = ((128 / size + taps - 1) / taps + 7) / 8 * 8;
  const double rows = (double)(l.batch ? l.batch * l.L : l.L), bytes = rows * l.I * size;
  const double rounds = ceil(ceil(rows / 128) * ceil(l.I / 256.0) / sms), product = rounds * ((l.O + kBK - 1) / kBK) * (128 + 256) * kRowNs;
  return kRowsNs + (product > bytes * kWriteNs ? product : bytes * kWriteNs) + bytes * kReadNs + v.B * ceil((double)v.C / channels) * kCtaNs;
}

}  // namespace

// Whether conv_grad_input makes the input gradient: stride 1, one scale for the codes of an image, one byte per code, sums of a tap that 32
// bits hold.  (Under a dilation wider than the output most taps reach nothing.)
bool conv_fold_covered(const hot_layer_t& l, const hot_conv_t& v) {
  const hot_linear_cfg_t& c = l.cfg;
  if (v.B <= 0 || v.C <= 0 || v.H <= 0 || v.W <= 0 || v.kh <= 0 || v.kw <= 0 || v.dh <= 0 || v.dw <= 0 || v.ph < 0 || v.pw < 0 || v.dtype != c.dtype ||
      l.O <= 0 || c.q_w.bits < 2 || c.q_w.bits > 8)
    return false;
  if (v.sh != 1 || v.sw != 1 || c.q_gx.scale_mode != HOT_SCALE_TENSOR || c.q_gx.storage != HOT_STORE_INT8) return false;
  const int64_t oh = v.H + 2ll * v.ph - (int64_t)v.dh * (v.kh - 1), ow = v.W + 2ll * v.pw - (int64_t)v.dw * (v.kw - 1);
  if (oh < v.dh || ow < v.dw || oh > (1 << 20) || ow > (1 << 20) || v.H > (1 << 20) || v.W > (1 << 20) || v.ph > (1 << 20) ||
      v.pw > (1 << 20) || v.C > (1 << 20) || v.B > 65535)
    return false;
  return l.O * 128 * ((1ll << (c.q_w.bits - 1)) - 1) < (1ll << 31) && v.kh * (int64_t)v.kw <= 4096 && l.I == (int64_t)v.C * v.kh * v.kw &&
         (l.batch ? l.batch == v.B && l.L == oh * ow : l.L == v.B * oh * ow);
}

int conv_grad_input(const hot_layer_t& l, const hot_conv_t& v, const void* q_go, int64_t ld_go, const float* s_go, const void* q_w, int64_t ld_w,
                    const float* s_w, float post, void* out, uint32_t* status, cudaStream_t st) {
  if (!conv_fold_covered(l, v)) HOT_FAIL(HOT_ERR_UNSUPPORTED, "hot_layer_backward_conv: this convolution's input gradient is not folded here");
  const int64_t oh = v.H + 2ll * v.ph - (int64_t)v.dh * (v.kh - 1), ow = v.W + 2ll * v.pw - (int64_t)v.dw * (v.kw - 1), taps = (int64_t)v.kh * v.kw;
  const int sms = device_sm_count();
  if (sms <= 0) return HOT_ERR_CUDA;
  FoldParams p;
  memset(&p, 0, sizeof(p));
  const FoldPlan f = plan_fold(l, v, sms);
  p.B = (int)v.B;
  p.H = (int)v.H;
  p.W = (int)v.W;
  p.C = (int)v.C;
  p.bw = f.bw;
  p.bh = f.bh;
  p.nb = f.nb;
  p.tw = f.tw;
  p.th = f.th;
  p.bn = f.bn;
  p.n_tiles = f.n_tiles;
  if (f.m_tiles * p.n_tiles >= (1ll << 30)) HOT_FAIL(HOT_ERR_UNSUPPORTED, "hot_layer_backward_conv: too many tiles");
  p.num_tiles = (int)(f.m_tiles * p.n_tiles);
  p.OH = (int)oh; p.OW = (int)ow; p.kh = v.kh; p.kw = v.kw; p.dh = v.dh; p.dw = v.dw; p.ph = v.ph; p.pw = v.pw;
  p.kblocks = (int)((l.O + kBK - 1) / kBK);
  p.last_steps = (int)((l.O - (int64_t)(p.kblocks - 1) * kBK + 31) / 32);
  p.by_n = fast_div(p.n_tiles);
  p.by_tw = fast_div(p.tw);
  p.by_th = fast_div(p.th);
  p.by_bw = fast_div(p.bw);
  p.by_image = fast_div(p.bw * p.bh);
  p.tx = (uint32_t)((p.bw * p.bh * p.nb + p.bn) * kBK);
  p.sa = s_go;
  p.sa_batch = l.batch > 0;
  p.sb = s_w;
  p.post = post;
  p.lean = l.I * (l.cfg.dtype == HOT_BF16 ? 2 : 4) % 16 == 0;
  p.one = 1.0f;
  p.out = out;
  p.status = status;
  p.wait_ns = wait_limit_ns();
  CUtensorMap ma, mb;
  const int64_t da[4] = {l.O, ow, oh, v.B}, sa[3] = {ld_go, ld_go * ow, ld_go * ow * oh};
  const int ba[4] = {kBK, p.bw, p.bh, p.nb};
  if (int rc = make_map_nd(&ma, q_go, 4, da, sa, ba)) return rc;
  const int64_t db[3] = {l.O, taps, v.C}, sb[2] = {ld_w, ld_w * taps};
  const int bb[3] = {kBK, 1, p.bn};
  if (int rc = make_map_nd(&mb, q_w, 3, db, sb, bb)) return rc;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)(p.num_tiles < sms ? p.num_tiles : sms));
  cfg.blockDim = dim3(kThreads);
  cfg.stream = st;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  auto launch = [&](auto kernel, int smem, PerDeviceOnce& once) -> int {
    bool done = false;
    const int dev = once.current(&done);
    if (dev < 0) HOT_FAIL(HOT_ERR_CUDA, "hot_layer_backward_conv: cannot query the current CUDA device");
    if (!done) {
      HOT_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
      once.mark(dev);
    }
    cfg.dynamicSmemBytes = smem;
    HOT_CUDA(cudaLaunchKernelEx(&cfg, kernel, ma, mb, p));
    return HOT_OK;
  };
  static PerDeviceOnce once[4];
  constexpr int kSmem1 = Layout<true>::kSmem, kSmem = Layout<false>::kSmem;
  if (l.cfg.dtype == HOT_BF16) return taps == 1 ? launch(conv_fold_kernel<true, true>, kSmem1, once[0]) : launch(conv_fold_kernel<false, true>, kSmem, once[1]);
  return taps == 1 ? launch(conv_fold_kernel<true, false>, kSmem1, once[2]) : launch(conv_fold_kernel<false, false>, kSmem, once[3]);
}

}  // namespace hot

extern "C" int hot_conv_folds(const hot_layer_t* layer, const hot_conv_t* conv) {
  using namespace hot;
  if (!layer || !conv || !conv_fold_covered(*layer, *conv)) return 0;
  int sms = device_sm_count();
  if (sms <= 0) sms = 148;  // (asked where there is no device)
  return plan_fold(*layer, *conv, sms).ns <= kFoldOver * rows_ns(*layer, *conv, sms) ? 1 : 0;
}
