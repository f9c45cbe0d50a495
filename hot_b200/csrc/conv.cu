// The data movement around a convolution that runs as a linear layer: unfolding the input to one row per output
// position (im2col), folding the gradient of those rows back (col2im), and the two transposes between [positions,
// channels] and [channels, positions].
//
// All three are bound by HBM: the unfolded tensor is kh * kw times the input (57.8 MB for 32 x 128 x 28 x 28, 3 x 3, bf16:
// 9 us to write at the measured 6.5 TB/s).  torch's unfold writes it position-contiguous, one image per launch, and needs
// a transposing copy before the linear layer can read it; its fold reads it with one strided load per tap.  Here a
// CTA stages its part of the smaller side in shared memory, so that both sides of HBM are touched once, in whole sectors.
#include "common.cuh"

namespace hot {
namespace {

constexpr int kThreads = 256;
constexpr int kSmemLimit = 96 * 1024;  // two CTAs per SM
constexpr int kMaxGridY = 65535;

struct ConvGeo {
  int C, H, W, OH, OW, kh, kw, sh, sw, ph, pw, dh, dw;
  int kk;       // kh * kw
  int cc;       // channels per CTA
  int rows;     // im2col: output rows per CTA; col2im: input rows per CTA
  int span_h;   // im2col: staged input rows; col2im: staged output rows (upper bound)
  int span_w;   // im2col: staged input columns
  int pitch;    // col2im: staged elements per position
  FastDiv by_ow, by_w, by_kk, by_kw, by_units;  // OW, W, kh * kw, kw, copies per staged position
};

__device__ __forceinline__ float widen(uint32_t v) { return __uint_as_float(v); }
__device__ __forceinline__ float widen(uint16_t v) { return __uint_as_float((uint32_t)v << 16); }
template <typename R>
__device__ __forceinline__ R narrow(float v);
template <>
__device__ __forceinline__ uint32_t narrow<uint32_t>(float v) {
  return __float_as_uint(v);
}
template <>
__device__ __forceinline__ uint16_t narrow<uint16_t>(float v) {
  return __bfloat16_as_ushort(__float2bfloat16_rn(v));
}

// One CTA: channels c0 .. c0 + cc of one image, output rows oh0 .. oh0 + rows.  The input rows under them go to shared
// memory with the padding as zeros; then a thread gathers V consecutive taps of one position (a warp: four
// neighbouring vectors of eight positions, i.e. 64-byte pieces) through a table of tap offsets and stores them at once.
template <typename R, int V>
__global__ void __launch_bounds__(kThreads) im2col_kernel(const R* __restrict__ x, R* __restrict__ cols, ConvGeo g) {
  extern __shared__ __align__(16) uint8_t smem[];
  const int c0 = blockIdx.x * g.cc, oh0 = blockIdx.y * g.rows;
  const int nc = min(g.cc, g.C - c0), nrows = min(g.rows, g.OH - oh0);
  R* tile = reinterpret_cast<R*>(smem);
  uint16_t* tap = reinterpret_cast<uint16_t*>(smem + (((size_t)g.cc * g.span_h * g.span_w * sizeof(R) + 15) & ~(size_t)15));
  const R* src = x + ((int64_t)blockIdx.z * g.C + c0) * g.H * g.W;
  const int ih0 = oh0 * g.sh - g.ph;
  const int plane = g.span_h * g.span_w;
  for (int c = threadIdx.x >> 5; c < nc; c += kThreads / 32)
    for (int w = threadIdx.x & 31; w < g.span_w; w += 32) {
      const int iw = w - g.pw;
      const bool col_ok = iw >= 0 && iw < g.W;
      const R* from = src + ((int64_t)c * g.H + ih0) * g.W + iw;
      R* to = tile + c * plane + w;
#pragma unroll 4
      for (int r = 0; r < g.span_h; ++r) to[r * g.span_w] = col_ok && (unsigned)(ih0 + r) < (unsigned)g.H ? __ldg(from + r * g.W) : (R)0;
    }
  const int taps = nc * g.kk;
  for (int k = threadIdx.x; k < taps; k += kThreads) {
    const int c = k / g.by_kk, t = k - c * g.kk, i = t / g.by_kw, j = t - i * g.kw;
    tap[k] = (uint16_t)(c * plane + i * g.dh * g.span_w + j * g.dw);
  }
  __syncthreads();
  const int ckk = g.C * g.kk;
  R* dst = cols + ((int64_t)blockIdx.z * g.OH + oh0) * g.OW * ckk + (int64_t)c0 * g.kk;
  const int vecs = taps / V, npos = nrows * g.OW;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int pgroups = (npos + 7) >> 3;
  for (int pg = warp; pg < pgroups; pg += kThreads / 32) {
    const int pos = pg * 8 + (lane >> 2);
    if (pos >= npos) continue;
    const int r = pos / g.by_ow, w = pos - r * g.OW;
    const R* at = tile + r * g.sh * g.span_w + w * g.sw;
    R* to = dst + (int64_t)pos * ckk;
#pragma unroll 2
    for (int v = lane & 3; v < vecs; v += 4) {
      alignas(16) R out[V];
      if constexpr (V == 8) {
        const uint4 o = *reinterpret_cast<const uint4*>(tap + v * 8);
        out[0] = at[o.x & 0xFFFFu]; out[1] = at[o.x >> 16]; out[2] = at[o.y & 0xFFFFu]; out[3] = at[o.y >> 16];
        out[4] = at[o.z & 0xFFFFu]; out[5] = at[o.z >> 16]; out[6] = at[o.w & 0xFFFFu]; out[7] = at[o.w >> 16];
      } else if constexpr (V == 4) {
        const uint2 o = *reinterpret_cast<const uint2*>(tap + v * 4);
        out[0] = at[o.x & 0xFFFFu]; out[1] = at[o.x >> 16]; out[2] = at[o.y & 0xFFFFu]; out[3] = at[o.y >> 16];
      } else {
        out[0] = at[tap[v]];
      }
      if constexpr (V == 1) to[v] = out[0];
      else *reinterpret_cast<uint4*>(to + v * V) = *reinterpret_cast<const uint4*>(out);
    }
  }
}

// Rows too long for shared memory, or too many of them for a launch: one element per thread, read where it lies.
template <typename R>
__global__ void __launch_bounds__(kThreads) im2col_direct_kernel(const R* __restrict__ x, R* __restrict__ cols, ConvGeo g) {
  const int64_t ckk = (int64_t)g.C * g.kk, total = (int64_t)g.OH * g.OW * ckk;
  x += (int64_t)blockIdx.y * g.C * g.H * g.W;
  cols += (int64_t)blockIdx.y * total;
  for (int64_t i = (int64_t)blockIdx.x * kThreads + threadIdx.x; i < total; i += (int64_t)gridDim.x * kThreads) {
    const int64_t pos = i / ckk;
    const int k = (int)(i - pos * ckk), c = k / g.kk, t = k - c * g.kk;
    const int ih = (int)(pos / g.OW) * g.sh - g.ph + t / g.kw * g.dh, iw = (int)(pos % g.OW) * g.sw - g.pw + t % g.kw * g.dw;
    cols[i] = ih >= 0 && ih < g.H && iw >= 0 && iw < g.W ? __ldg(x + ((int64_t)c * g.H + ih) * g.W + iw) : (R)0;
  }
}

// One CTA: channels c0 .. c0 + cc of one image, input rows h0 .. h0 + rows.  The taps of those channels at every
// position that reaches the rows go to shared memory (V elements per load, at an odd pitch of 4-byte words: neighbouring
// positions then lie in different banks), with one more position of zeros for taps outside the output.  A thread
// finds the positions that reach its input element once and then sums the taps of channel after channel in fp32, output row
// by output row.  (STAGED false: rows too long for shared memory; the taps are read where they lie.)
// K: side of a square kernel known at compile time (the taps' addresses stay in registers), 0: any kernel.
template <typename R, int V, bool STAGED, int K>
__global__ void __launch_bounds__(kThreads) col2im_kernel(const R* __restrict__ cols, R* __restrict__ x, ConvGeo g) {
  extern __shared__ __align__(16) uint8_t smem[];
  R* tile = reinterpret_cast<R*>(smem);
  const int c0 = blockIdx.x * g.cc, h0 = blockIdx.y * g.rows;
  const int nc = min(g.cc, g.C - c0), nrows = min(g.rows, g.H - h0);
  const int reach = (g.kh - 1) * g.dh;
  int oh_lo = h0 + g.ph - reach;  // first output row that can reach input row h0
  oh_lo = oh_lo <= 0 ? 0 : (oh_lo + g.sh - 1) / g.sh;
  const int oh_hi = min(g.OH - 1, (h0 + nrows - 1 + g.ph) / g.sh);
  const int npos = oh_hi < oh_lo ? 0 : (oh_hi - oh_lo + 1) * g.OW;
  const int ckk = g.C * g.kk, taps = nc * g.kk;
  const R* src = cols + ((int64_t)blockIdx.z * g.OH + oh_lo) * g.OW * ckk + (int64_t)c0 * g.kk;
  if constexpr (STAGED) {
    const int units = taps / V;
#pragma unroll 4
    for (int i = threadIdx.x; i < npos * units; i += kThreads) {
      const int pos = nc == g.cc ? i / g.by_units : i / units, k = i - pos * units;
      R* to = tile + pos * g.pitch + k * V;
      if constexpr (V * sizeof(R) == 16) {
        const uint4 v = __ldg(reinterpret_cast<const uint4*>(src + (int64_t)pos * ckk) + k);
        uint32_t* w = reinterpret_cast<uint32_t*>(to);
        w[0] = v.x; w[1] = v.y; w[2] = v.z; w[3] = v.w;
      } else {
        *to = __ldg(src + (int64_t)pos * ckk + k);
      }
    }
    for (int k = threadIdx.x; k < g.pitch; k += kThreads) tile[npos * g.pitch + k] = (R)0;
    __syncthreads();
  }
  R* dst = x + ((int64_t)blockIdx.z * g.C + c0) * g.H * g.W + (int64_t)h0 * g.W;
  for (int e = threadIdx.x; e < nrows * g.W; e += kThreads) {
    const int hh = e / g.by_w, w = e - hh * g.W, h = h0 + hh;
    // the output row (column) that reads this element through tap row ki (tap column kj), or -1
    auto out_row = [&](int ki) {
      const int t = h + g.ph - ki * g.dh, o = g.sh == 1 ? t : t / g.sh;
      return t >= 0 && o < g.OH && (g.sh == 1 || o * g.sh == t) ? o - oh_lo : -1;
    };
    auto out_col = [&](int kj) {
      const int t = w + g.pw - kj * g.dw, o = g.sw == 1 ? t : t / g.sw;
      return t >= 0 && o < g.OW && (g.sw == 1 || o * g.sw == t) ? o : -1;
    };
    if constexpr (STAGED && K > 0) {
      int at[K * K];  // tap addresses of channel 0, ascending output rows and columns
#pragma unroll
      for (int i = 0; i < K; ++i)
#pragma unroll
        for (int j = 0; j < K; ++j) {
          const int ki = K - 1 - i, kj = K - 1 - j, r = out_row(ki), c = out_col(kj);
          at[i * K + j] = (r >= 0 && c >= 0 ? r * g.OW + c : npos) * g.pitch + ki * K + kj;
        }
#pragma unroll 4
      for (int c = 0; c < nc; ++c) {
        float sum = 0.0f;
#pragma unroll
        for (int i = 0; i < K * K; ++i) sum += widen(tile[at[i] + c * (K * K)]);
        dst[(int64_t)c * g.H * g.W + e] = narrow<R>(sum);
      }
    } else {
      for (int c = 0; c < nc; ++c) {
        float sum = 0.0f;
        for (int ki = g.kh - 1; ki >= 0; --ki) {
          const int r = out_row(ki);
          if (r < 0) continue;
          for (int kj = g.kw - 1; kj >= 0; --kj) {
            const int o = out_col(kj);
            if (o < 0) continue;
            const int k = c * g.kk + ki * g.kw + kj;
            sum += widen(STAGED ? tile[(r * g.OW + o) * g.pitch + k] : src[((int64_t)r * g.OW + o) * ckk + k]);
          }
        }
        dst[(int64_t)c * g.H * g.W + e] = narrow<R>(sum);
      }
    }
  }
}

// out[b][c][r] = in[b][r][c] (+ bias[c], rounded once more, as a separate addition would): 64 x 64 tiles, neighbouring
// lanes on neighbouring elements on both sides.  VI / VO: 16-bit elements per load / store (pairs where the rows of that
// side begin at whole words: 6.4 MB transposed in 7.3 us one by one).  A CTA takes every gridDim.y-th tile of its columns.
template <typename R, int VI, int VO>
__global__ void __launch_bounds__(kThreads) transpose_kernel(const R* __restrict__ in, const R* __restrict__ bias, R* __restrict__ out,
                                                             int rows, int cols) {
  __shared__ __align__(16) R tile[64][sizeof(R) == 2 ? 66 : 65];
  const int c0 = blockIdx.x * 64;
  in += (int64_t)blockIdx.z * rows * cols;
  out += (int64_t)blockIdx.z * rows * cols;
  constexpr int kLanesI = 64 / VI, kLanesO = 64 / VO;
  for (int r0 = blockIdx.y * 64;;) {
    {
      const int tx = threadIdx.x % kLanesI * VI, ty = threadIdx.x / kLanesI;
#pragma unroll
      for (int i = 0; i < 64 * kLanesI / kThreads; ++i) {
        const int rr = ty + i * (kThreads / kLanesI), r = r0 + rr, c = c0 + tx;
        if (r < rows && c < cols) {
          if constexpr (VI == 2) *reinterpret_cast<uint32_t*>(&tile[rr][tx]) = __ldg(reinterpret_cast<const uint32_t*>(in + (int64_t)r * cols + c));
          else tile[rr][tx] = __ldg(in + (int64_t)r * cols + c);
        }
      }
    }
    __syncthreads();
    const int tx = threadIdx.x % kLanesO * VO, ty = threadIdx.x / kLanesO;
#pragma unroll
    for (int i = 0; i < 64 * kLanesO / kThreads; ++i) {
      const int cc = ty + i * (kThreads / kLanesO), c = c0 + cc, r = r0 + tx;
      if (c < cols && r < rows) {
        R v[VO];
#pragma unroll
        for (int k = 0; k < VO; ++k) {
          v[k] = tile[tx + k][cc];
          if (bias) v[k] = narrow<R>(__fadd_rn(widen(v[k]), widen(bias[c])));
        }
        if constexpr (VO == 2) *reinterpret_cast<uint32_t*>(out + (int64_t)c * rows + r) = (uint32_t)v[0] | ((uint32_t)v[1] << 16);
        else out[(int64_t)c * rows + r] = v[0];
      }
    }
    r0 += (int)gridDim.y * 64;
    if (r0 >= rows) break;
    __syncthreads();
  }
}

int geometry(const hot_conv_t* p, ConvGeo* g, const char* who) {
  if (!p) HOT_FAIL(HOT_ERR_ARG, "%s: null pointer", who);
  if (p->dtype != HOT_F32 && p->dtype != HOT_BF16) HOT_FAIL(HOT_ERR_UNSUPPORTED, "%s: dtype %d", who, p->dtype);
  if (p->B <= 0 || p->B > 65535 || p->C <= 0 || p->H <= 0 || p->W <= 0 || p->kh <= 0 || p->kw <= 0 || p->sh <= 0 || p->sw <= 0 || p->ph < 0 ||
      p->pw < 0 || p->dh <= 0 || p->dw <= 0)
    HOT_FAIL(HOT_ERR_ARG, "%s: bad geometry", who);
  const int64_t oh = p->H + 2ll * p->ph - (int64_t)p->dh * (p->kh - 1) - 1, ow = p->W + 2ll * p->pw - (int64_t)p->dw * (p->kw - 1) - 1;
  if (oh < 0 || ow < 0) HOT_FAIL(HOT_ERR_ARG, "%s: the kernel is larger than the padded input", who);
  g->C = p->C; g->H = p->H; g->W = p->W;
  g->OH = (int)(oh / p->sh + 1); g->OW = (int)(ow / p->sw + 1);
  g->kh = p->kh; g->kw = p->kw; g->sh = p->sh; g->sw = p->sw; g->ph = p->ph; g->pw = p->pw; g->dh = p->dh; g->dw = p->dw;
  g->kk = p->kh * p->kw;
  if ((int64_t)g->OH * g->OW > (1 << 30) || (int64_t)g->C * g->kk > (1 << 30)) HOT_FAIL(HOT_ERR_UNSUPPORTED, "%s: image or kernel too large", who);
  return HOT_OK;
}

template <typename K>
int allow_smem(K kernel, PerDeviceOnce& once) {
  bool done = false;
  const int dev = once.current(&done);
  if (dev < 0) HOT_FAIL(HOT_ERR_CUDA, "cannot query the current CUDA device");
  if (!done) {
    HOT_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmemLimit));
    once.mark(dev);
  }
  return HOT_OK;
}

template <typename R, int V>
int launch_im2col(const R* x, R* cols, const ConvGeo& g, int64_t B, size_t smem, cudaStream_t st) {
  static PerDeviceOnce once;
  if (int rc = allow_smem(im2col_kernel<R, V>, once)) return rc;
  const dim3 grid((g.C + g.cc - 1) / g.cc, (g.OH + g.rows - 1) / g.rows, (unsigned)B);
  im2col_kernel<R, V><<<grid, kThreads, smem, st>>>(x, cols, g);
  HOT_CUDA(cudaGetLastError());
  return HOT_OK;
}

template <typename R>
int im2col_typed(const R* x, R* cols, ConvGeo g, int64_t B, cudaStream_t st) {
  // Channels per CTA: a multiple of 8, so that every CTA's taps begin at a whole vector; output rows: enough for
  // about 192 positions (the rows two neighbouring CTAs both stage are then few).  Both shrink until the staged rows fit and a tap offset fits 16 bits.
  constexpr int kV = 16 / sizeof(R);
  g.span_w = (g.OW - 1) * g.sw + (g.kw - 1) * g.dw + 1;
  g.rows = (191 + g.OW) / g.OW;
  if (g.rows > g.OH) g.rows = g.OH;
  g.cc = g.C < 32 ? g.C : 32;
  auto smem = [&]() {
    g.span_h = (g.rows - 1) * g.sh + (g.kh - 1) * g.dh + 1;
    return (((size_t)g.cc * g.span_h * g.span_w * sizeof(R) + 15) & ~(size_t)15) + ((size_t)g.cc * g.kk + 8) * sizeof(uint16_t);
  };
  auto fits = [&]() { return smem() <= 48 * 1024 && (int64_t)g.cc * g.span_h * g.span_w < 65536; };
  while (!fits() && (g.rows > 1 || g.cc > 1)) {
    if (g.cc > 8) g.cc = (g.cc / 2 + 7) / 8 * 8;
    else if (g.rows > 1) g.rows = (g.rows + 1) / 2;
    else g.cc = (g.cc + 1) / 2;
  }
  if (smem() > (size_t)kSmemLimit || (int64_t)g.cc * g.span_h * g.span_w >= 65536 || (g.OH + g.rows - 1) / g.rows > kMaxGridY) {
    im2col_direct_kernel<R><<<dim3(2048, (unsigned)B), kThreads, 0, st>>>(x, cols, g);
    HOT_CUDA(cudaGetLastError());
    return HOT_OK;
  }
  g.by_ow = fast_div(g.OW);
  g.by_kk = fast_div(g.kk);
  g.by_kw = fast_div(g.kw);
  const bool vec = (int64_t)g.C * g.kk % kV == 0 && (g.cc == g.C || (int64_t)g.cc * g.kk % kV == 0) && ((uintptr_t)cols) % 16 == 0;
  return vec ? launch_im2col<R, kV>(x, cols, g, B, smem(), st) : launch_im2col<R, 1>(x, cols, g, B, smem(), st);
}

template <typename R, int V>
int launch_col2im(const R* cols, R* x, const ConvGeo& g, int64_t B, size_t bytes, bool staged, cudaStream_t st) {
  const dim3 grid((g.C + g.cc - 1) / g.cc, (g.H + g.rows - 1) / g.rows, (unsigned)B);
  auto launch = [&](auto kernel, PerDeviceOnce& once) -> int {
    if (int rc = allow_smem(kernel, once)) return rc;
    kernel<<<grid, kThreads, staged ? bytes : 0, st>>>(cols, x, g);
    HOT_CUDA(cudaGetLastError());
    return HOT_OK;
  };
  static PerDeviceOnce once3, once1, once0, once_direct;
  if (!staged) return launch(col2im_kernel<R, 1, false, 0>, once_direct);
  if (g.kh == 3 && g.kw == 3) return launch(col2im_kernel<R, V, true, 3>, once3);
  if (g.kh == 1 && g.kw == 1) return launch(col2im_kernel<R, V, true, 1>, once1);
  return launch(col2im_kernel<R, V, true, 0>, once0);
}

template <typename R>
int col2im_typed(const R* cols, R* x, ConvGeo g, int64_t B, cudaStream_t st) {
  // Channels per CTA: whole 16-byte vectors, at least 128 contiguous bytes of taps per position.  Rows per CTA: of what
  // fits, the height that loses least to staging rows twice and to a last round of input elements that is not full (at
  // least what keeps the launch within its limits).
  constexpr int kV = 16 / sizeof(R);
  g.cc = (int)((128 / sizeof(R) + g.kk - 1) / g.kk);
  g.cc = (g.cc + kV - 1) / kV * kV;
  if (g.cc > g.C) g.cc = g.C;
  auto smem = [&](int rows) {
    const int words = (int)((g.cc * g.kk * sizeof(R) + 3) / 4) | 1;
    g.pitch = (int)(words * 4 / sizeof(R));
    g.span_h = (rows - 1 + (g.kh - 1) * g.dh) / g.sh + 1;
    if (g.span_h > g.OH) g.span_h = g.OH;
    return ((size_t)g.span_h * g.OW + 1) * words * 4;
  };
  const size_t budget = 72 * 1024;  // three CTAs per SM
  const int least = (g.H + kMaxGridY - 1) / kMaxGridY;
  while (smem(least) > budget && g.cc > 1) g.cc = g.cc > kV ? (g.cc / 2 + kV - 1) / kV * kV : (g.cc + 1) / 2;
  double best = -1.0;
  g.rows = least;
  for (int rows = least; rows <= g.H && (rows == least || smem(rows) <= budget); ++rows) {
    const int tiles = (g.H + rows - 1) / rows, items = rows * g.W;
    const double useful = (double)g.H / ((double)tiles * (rows + (g.kh - 1) * g.dh)) * items / ((items + kThreads - 1) / kThreads * kThreads);
    if (useful > best) {
      best = useful;
      g.rows = rows;
    }
  }
  const size_t bytes = smem(g.rows);
  const bool staged = bytes <= (size_t)kSmemLimit;
  if (!staged) {
    g.cc = g.C < 8 ? g.C : 8;
    g.rows = least;
  }
  g.by_w = fast_div(g.W);
  const bool vec = (int64_t)g.C * g.kk % kV == 0 && (g.cc == g.C || (int64_t)g.cc * g.kk % kV == 0) && ((uintptr_t)cols) % 16 == 0;
  g.by_units = fast_div(g.cc * g.kk / (vec ? kV : 1));
  return vec ? launch_col2im<R, kV>(cols, x, g, B, bytes, staged, st) : launch_col2im<R, 1>(cols, x, g, B, bytes, staged, st);
}

}  // namespace
}  // namespace hot

extern "C" int hot_im2col(const hot_conv_t* conv, const void* x, void* cols, hot_stream_t stream) {
  using namespace hot;
  ConvGeo g = {};
  if (int rc = geometry(conv, &g, "hot_im2col")) return rc;
  if (!x || !cols) HOT_FAIL(HOT_ERR_ARG, "hot_im2col: null pointer");
  cudaStream_t st = (cudaStream_t)stream;
  if (conv->dtype == HOT_F32) return im2col_typed((const uint32_t*)x, (uint32_t*)cols, g, conv->B, st);
  return im2col_typed((const uint16_t*)x, (uint16_t*)cols, g, conv->B, st);
}

extern "C" int hot_col2im(const hot_conv_t* conv, const void* cols, void* x, hot_stream_t stream) {
  using namespace hot;
  ConvGeo g = {};
  if (int rc = geometry(conv, &g, "hot_col2im")) return rc;
  if (!x || !cols || ((uintptr_t)cols) % 4 != 0) HOT_FAIL(HOT_ERR_ARG, "hot_col2im: null or misaligned pointer");
  cudaStream_t st = (cudaStream_t)stream;
  if (conv->dtype == HOT_F32) return col2im_typed((const uint32_t*)cols, (uint32_t*)x, g, conv->B, st);
  return col2im_typed((const uint16_t*)cols, (uint16_t*)x, g, conv->B, st);
}

namespace hot {

int device_sm_count();

namespace {

// y[r, c] += bias[c].  Bound by the two trips over y, of which the reading one mostly hits L2 after the product that wrote it;
// a thread keeps its columns' bias and walks down the rows, four loads in flight (6304 x 3072: torch's broadcast addition
// 49.0 us, this 19.3).  V: columns per thread.
template <typename V>
__global__ void __launch_bounds__(256) add_bias_kernel(V* __restrict__ y, const V* __restrict__ bias, int64_t rows, int nv) {
  const int c = blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= nv) return;
  const V b = bias[c];
  const int64_t step = (int64_t)gridDim.y * blockDim.y;
  int64_t r = (int64_t)blockIdx.y * blockDim.y + threadIdx.y;
  auto add = [&](V& v) {
    float* f = reinterpret_cast<float*>(&v);
    const float* g = reinterpret_cast<const float*>(&b);
#pragma unroll
    for (int i = 0; i < (int)(sizeof(V) / 4); ++i) f[i] = __fadd_rn(f[i], g[i]);
  };
  for (; r + 3 * step < rows; r += 4 * step) {
    V v[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) v[i] = y[(r + i * step) * nv + c];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      add(v[i]);
      y[(r + i * step) * nv + c] = v[i];
    }
  }
  for (; r < rows; r += step) {
    V v = y[r * nv + c];
    add(v);
    y[r * nv + c] = v;
  }
}

}  // namespace
}  // namespace hot

extern "C" int hot_add_bias(float* y, const float* bias, int64_t rows, int64_t cols, hot_stream_t stream) {
  using namespace hot;
  if (!y || !bias) HOT_FAIL(HOT_ERR_ARG, "hot_add_bias: null pointer");
  if (rows <= 0 || cols <= 0 || cols > (1 << 30)) HOT_FAIL(HOT_ERR_ARG, "hot_add_bias: bad shape");
  const int sms = device_sm_count();
  if (sms <= 0) return HOT_ERR_CUDA;
  const bool vec = cols % 4 == 0 && ((uintptr_t)y) % 16 == 0 && ((uintptr_t)bias) % 16 == 0;
  const int nv = (int)(vec ? cols / 4 : cols);
  int bx = 32;
  while (bx < 256 && bx < nv) bx <<= 1;
  const dim3 block((unsigned)bx, (unsigned)(256 / bx));
  const int64_t gx = (nv + bx - 1) / bx;
  // eight CTAs per SM if there are rows for them
  int64_t gy = (sms * 8 + gx - 1) / gx;
  const int64_t most = (rows + block.y - 1) / block.y;
  if (gy > most) gy = most;
  if (gy > 65535) gy = 65535;
  const dim3 grid((unsigned)gx, (unsigned)gy);
  cudaStream_t st = (cudaStream_t)stream;
  if (vec) add_bias_kernel<float4><<<grid, block, 0, st>>>((float4*)y, (const float4*)bias, rows, nv);
  else add_bias_kernel<float><<<grid, block, 0, st>>>(y, bias, rows, nv);
  HOT_CUDA(cudaGetLastError());
  return HOT_OK;
}

extern "C" int hot_transpose(int dtype, int64_t batch, int64_t rows, int64_t cols, const void* in, const void* bias, void* out,
                             hot_stream_t stream) {
  using namespace hot;
  if (!in || !out) HOT_FAIL(HOT_ERR_ARG, "hot_transpose: null pointer");
  if (batch <= 0 || batch > 65535 || rows <= 0 || cols <= 0 || cols > (1 << 30) || rows > (1 << 30))
    HOT_FAIL(HOT_ERR_ARG, "hot_transpose: bad shape");
  const int64_t row_tiles = (rows + 63) / 64;
  const dim3 grid((unsigned)((cols + 63) / 64), (unsigned)(row_tiles < kMaxGridY ? row_tiles : kMaxGridY), (unsigned)batch);
  cudaStream_t st = (cudaStream_t)stream;
  if (dtype == HOT_F32) {
    transpose_kernel<uint32_t, 1, 1><<<grid, kThreads, 0, st>>>((const uint32_t*)in, (const uint32_t*)bias, (uint32_t*)out, (int)rows, (int)cols);
  } else if (dtype == HOT_BF16) {
    const bool vi = cols % 2 == 0 && ((uintptr_t)in) % 4 == 0, vo = rows % 2 == 0 && ((uintptr_t)out) % 4 == 0;
    auto kernel = vi ? (vo ? transpose_kernel<uint16_t, 2, 2> : transpose_kernel<uint16_t, 2, 1>)
                     : (vo ? transpose_kernel<uint16_t, 1, 2> : transpose_kernel<uint16_t, 1, 1>);
    kernel<<<grid, kThreads, 0, st>>>((const uint16_t*)in, (const uint16_t*)bias, (uint16_t*)out, (int)rows, (int)cols);
  }
  else HOT_FAIL(HOT_ERR_UNSUPPORTED, "hot_transpose: dtype %d", dtype);
  HOT_CUDA(cudaGetLastError());
  return HOT_OK;
}
