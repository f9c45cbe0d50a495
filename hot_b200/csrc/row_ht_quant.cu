// Fused block-Hadamard transform along the contiguous dim + INT4/INT8 quantisation.
//
// A thread owns 32 consecutive elements, two runs of 16 held as sixteen packed pairs (r0[i], r1[i]).  Blackwell's packed
// fp32 instructions (add/fma .f32x2, IEEE round-to-nearest per lane) then run the butterfly stages h = 1 to 8 of both runs
// at once; stage h = 16 combines the halves of a pair; only stage h = 32 exchanges with lane ^ 1 through warp shuffles.  Per
// stage the arithmetic is (x + y, x - y) on (i, i + h): the order the CPU oracle fixes.  One Philox block serves the 32
// elements where codes take four random bits.  (With 16 elements per thread, order 32 took 16 shuffles and every thread
// half a block more: the quantising pass was bound by them.)
//
// Where it pays, the elements reach a thread through shared memory: a warp's 1,024 of them arrive by asynchronous copies while it
// works on the ones before, at no registers (prefetching into registers spilled) and in whole lines (a thread's own loads of
// 64 or 128 bytes ask L2 for every sector twice).  16-byte pieces are swizzled so that the eight lanes of a shared-memory phase meet no
// bank twice.
//
// Per-row ("per-token") scale: one launch; a row is held in registers by `tpr` threads, reduced to its abs-max, then
// quantised and stored.
// Per-tensor scale: two launches over the same input (abs-max into a scratch word, then quantise); both are streaming loops.
// The second runs from the end of the input to its start, since the end is what L2 still holds (60 of 134 MB), and is a
// programmatic dependent of the first: its first elements are on their way before that has ended.
// Both launches on inputs that change from call to call, us before and now: 16384 x 4096 bf16 to 4-bit Philox codes, order 32,
// 67.4 and 61.6 (27.3 at 5.7 TB/s, write-backs included, and 34.5 for issue: 65 % of the slots); 65536 x 1024 bf16, nearest, 73.9 and
// 68.0; 8192 x 8192 float32, order 64, nearest, 124.4 and 101.1 (6.0 TB/s over both).
#include "ht_device.cuh"
#include "tma.cuh"

namespace hot {
namespace {

constexpr int kThreads = 256;
constexpr int kMaxPairs = 2;  // 32-element pairs of runs per thread in the per-row kernel: cols <= 2 * 32 * 256

// The pairs of runs of a warp's lanes in shared memory, in order, as 16-byte pieces.
template <typename T>
struct WarpTile {
  static constexpr int kPieces = 2 * (int)sizeof(T);  // per lane
  static constexpr int kBytes = 32 * 16 * kPieces;
  // piece p of the tile lies at slot p ^ twist of its lane
  static __device__ __forceinline__ int twist(int lane) { return sizeof(T) == 2 ? (lane >> 1) & 3 : lane & 7; }
  // where the copy instruction k of this lane puts its piece, k * 32 + lane
  static __device__ __forceinline__ uint32_t to(uint32_t tile, int k, int lane) {
    const int p = k * 32 + lane;
    return tile + (uint32_t)(p ^ twist(p / kPieces)) * 16u;
  }
  static __device__ __forceinline__ void read(uint32_t tile, int lane, float2 (&v)[16]) {
    uint4 r[kPieces];
#pragma unroll
    for (int k = 0; k < kPieces; ++k)
      asm volatile("ld.shared.v4.b32 {%0, %1, %2, %3}, [%4];"
                   : "=r"(r[k].x), "=r"(r[k].y), "=r"(r[k].z), "=r"(r[k].w)
                   : "r"(tile + (uint32_t)(lane * kPieces + (k ^ twist(lane))) * 16u)
                   : "memory");
#pragma unroll
    for (int k = 0; k < kPieces / 2; ++k) {
      const uint4 &p0 = r[k], &p1 = r[k + kPieces / 2];
      const uint32_t a[4] = {p0.x, p0.y, p0.z, p0.w}, b[4] = {p1.x, p1.y, p1.z, p1.w};
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        if (sizeof(T) == 4) {
          v[(4 * k + i) & 15] = make_float2(__uint_as_float(a[i]), __uint_as_float(b[i]));
        } else {
          v[(8 * k + 2 * i) & 15] = make_float2(__uint_as_float(a[i] << 16), __uint_as_float(b[i] << 16));
          v[(8 * k + 2 * i + 1) & 15] = make_float2(__uint_as_float(a[i] & 0xFFFF0000u), __uint_as_float(b[i] & 0xFFFF0000u));
        }
      }
    }
  }
};
__device__ __forceinline__ void launch_dependents() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
__device__ __forceinline__ void wait_for_predecessor() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
// 16 bytes, or zeros
__device__ __forceinline__ void copy_piece(uint32_t dst, const void* src, bool ok) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(ok ? 16 : 0) : "memory");
}
__device__ __forceinline__ void copy_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void copy_wait() {
  asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}

// 32 bytes (32-byte aligned) in one load: half the tag look-ups of two 16-byte loads where lanes lie 64 bytes and more apart.
__device__ __forceinline__ void ldg32(const void* p, uint4& a, uint4& b) {
  asm("ld.global.nc.v8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
      : "=r"(a.x), "=r"(a.y), "=r"(a.z), "=r"(a.w), "=r"(b.x), "=r"(b.y), "=r"(b.z), "=r"(b.w)
      : "l"(p));
}

// Two runs of 16 elements straight from global memory.
template <typename T>
struct Raw32 {
  static constexpr int kWords = (int)sizeof(T);  // 16-byte pieces of a run
  uint4 r[2][kWords];
  // wide: the runs start on 32-byte boundaries
  __device__ __forceinline__ void load(const T* p0, const T* p1, bool ok0, bool ok1, bool wide) {
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const uint4* p = reinterpret_cast<const uint4*>(h ? p1 : p0);
      if (!(h ? ok1 : ok0)) {
#pragma unroll
        for (int k = 0; k < kWords; ++k) r[h][k] = make_uint4(0u, 0u, 0u, 0u);
      } else if (wide) {
#pragma unroll
        for (int k = 0; k < kWords; k += 2) ldg32(p + k, r[h][k], r[h][k + 1]);
      } else {
#pragma unroll
        for (int k = 0; k < kWords; ++k) r[h][k] = __ldg(p + k);
      }
    }
  }
  __device__ __forceinline__ void unpack(float2 (&v)[16]) const {
#pragma unroll
    for (int k = 0; k < kWords; ++k) {
      const uint32_t a[4] = {r[0][k].x, r[0][k].y, r[0][k].z, r[0][k].w}, b[4] = {r[1][k].x, r[1][k].y, r[1][k].z, r[1][k].w};
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        if (sizeof(T) == 4) {
          v[4 * k + i] = make_float2(__uint_as_float(a[i]), __uint_as_float(b[i]));
        } else {
          v[(8 * k + 2 * i) & 15] = make_float2(__uint_as_float(a[i] << 16), __uint_as_float(b[i] << 16));
          v[(8 * k + 2 * i + 1) & 15] = make_float2(__uint_as_float(a[i] & 0xFFFF0000u), __uint_as_float(b[i] & 0xFFFF0000u));
        }
      }
    }
  }
};

// Order-n transform of the pair of runs (N: the order where it is known at compile time, else 0: stages behind a branch
// cost the streaming passes 30 registers).  Must be executed by all lanes of a pair (lane, lane ^ 1) when n = 64.
template <int N>
__device__ __forceinline__ void butterfly32(float2 (&v)[16], int n_run, int lane) {
  const int n = N ? N : n_run;
#pragma unroll
  for (int h = 1; h < 16; h <<= 1) {
    if (n > h) {
#pragma unroll
      for (int i = 0; i < 16; ++i) {
        if ((i & h) == 0) {
          const float2 a = v[i], b = v[i + h];
          v[i] = add2(a, b);
          v[i + h] = sub2(a, b);
        }
      }
    }
  }
  if (n > 16) {
#pragma unroll
    for (int i = 0; i < 16; ++i) v[i] = make_float2(__fadd_rn(v[i].x, v[i].y), __fsub_rn(v[i].x, v[i].y));
  }
  if (n > 32) {
    const float sg = (lane & 1) ? -1.0f : 1.0f;  // upper half: partner - mine; lower: mine + partner
    const float2 sg2 = make_float2(sg, sg);
#pragma unroll
    for (int i = 0; i < 16; ++i) {
      float2 o;
      o.x = __shfl_xor_sync(0xFFFFFFFFu, v[i].x, 1);
      o.y = __shfl_xor_sync(0xFFFFFFFFu, v[i].y, 1);
      v[i] = __ffma2_rn(v[i], sg2, o);  // exact product, one rounding: o +- mine
    }
  }
}

__device__ __forceinline__ float absmax32(const float2 (&v)[16]) {
  float m = 0.0f;
#pragma unroll
  for (int i = 0; i < 16; ++i) asm("max.abs.f32 %0, %1, %2, %3;" : "=f"(m) : "f"(m), "f"(v[i].x), "f"(v[i].y));  // (a NaN is ignored)
  return m;
}

// STORE4: 0 a byte per code, 1 two codes per byte (Philox: of 4 bits, whose offset goes with a flip of one bit), 2 two narrower ones.
// The codes of the pair whose first logical element index is `e0` (a multiple of 16): out[4 * run + ...], two words of a
// run for INT4 (code i | code (i + 8) << 4 in byte i), four for INT8.
// WHOLE: both runs exist and e0 is a multiple of 32.
template <int ROUND, int STORE4, bool WHOLE>
__device__ __forceinline__ void quantise32(const float2 (&v)[16], const ScalePair& sp, const QuantDev& q, uint64_t e0, bool ok0,
                                           bool ok1, uint32_t (&out)[2][4]) {
  if (ROUND == HOT_ROUND_STOCH_PHILOX) {
    const bool rb4 = rand_bits(q.qmax) == 4;
    const float2 mk2 = make_float2(sp.mk, sp.mk), ck2 = make_float2(sp.ck, sp.ck);
    uint32_t k[2][16];  // raw bits of RN(x * mk + ck); the low mantissa bits are K
#pragma unroll
    for (int i = 0; i < 16; ++i) {
      const float2 t = __ffma2_rn(v[i], mk2, ck2);
      k[0][i] = __float_as_uint(t.x);
      k[1][i] = __float_as_uint(t.y);
    }
    uint4 b0, b1;
    if (rb4) {  // a block covers 32 elements: this pair, or the halves of two
      const uint4 b = philox_block(q, e0 >> 5);
      b0 = b;
      b1 = make_uint4(b.z, b.w, 0u, 0u);
      if (!WHOLE && (e0 & 16)) {
        b0 = b1;
        b1 = philox_block(q, (e0 >> 5) + 1);
      }
    } else {
      b0 = philox_block(q, e0 >> 4);
      b1 = philox_block(q, (e0 >> 4) + 1);
    }
    const uint32_t off = (uint32_t)(q.qmax + 1.0f);
#pragma unroll
    for (int r = 0; r < 2; ++r) {
      const uint4 b = r ? b1 : b0;
      uint32_t w[4];  // A (elements 0 to 7) in w[0], w[1], B in w[2], w[3]
      philox_run16_words(k[r], k[r] + 8, STORE4 || rb4, b.x, b.y, b.z, b.w, w[0], w[1], w[2], w[3]);
      if (STORE4) {  // (always 4 random bits)
        out[r][0] = ((w[0] >> 4) & 0x0F0F0F0Fu) | (w[2] & 0xF0F0F0F0u);
        out[r][1] = ((w[1] >> 4) & 0x0F0F0F0Fu) | (w[3] & 0xF0F0F0F0u);
#pragma unroll
        for (int i = 0; i < 2; ++i) out[r][i] = STORE4 == 1 ? out[r][i] ^ 0x88888888u : remove_offset(out[r][i], off, 0x11111111u, 0x10u);
      } else {
#pragma unroll
        for (int i = 0; i < 4; ++i) out[r][i] = remove_offset(rb4 ? (w[i] >> 4) & 0x0F0F0F0Fu : w[i], off, 0x01010101u, 0x100u);
      }
    }
  } else {
    const int qmax = (int)q.qmax;
#pragma unroll
    for (int r = 0; r < 2; ++r) {
      float u[16];
      if (ROUND == HOT_ROUND_STOCH_NOISE) {
        if (WHOLE || (r ? ok1 : ok0)) {
          float ua[8], ub[8];
          Load8<float>::run(q.noise + e0 + 16 * r, ua);
          Load8<float>::run(q.noise + e0 + 16 * r + 8, ub);
#pragma unroll
          for (int i = 0; i < 8; ++i) { u[i] = ua[i]; u[i + 8] = ub[i]; }
        } else {
#pragma unroll
          for (int i = 0; i < 16; ++i) u[i] = 0.0f;
        }
      }
#pragma unroll
      for (int i = 0; i < 4; ++i) out[r][i] = 0u;
#pragma unroll
      for (int i = 0; i < 16; ++i) {
        const int c = quantise_one<ROUND>(r ? v[i].y : v[i].x, sp, ROUND == HOT_ROUND_STOCH_NOISE ? u[i] : 0.0f, qmax);
        if (STORE4) out[r][(i & 7) >> 2] |= (uint32_t)(c & 0xF) << (8 * (i & 3) + 4 * (i >> 3));
        else out[r][i >> 2] |= (uint32_t)(c & 0xFF) << (8 * (i & 3));
      }
    }
  }
}

template <int STORE4>
__device__ __forceinline__ void store_run(uint8_t* dst, const uint32_t (&w)[4]) {
  if (STORE4) *reinterpret_cast<uint2*>(dst) = make_uint2(w[0], w[1]);
  else *reinterpret_cast<uint4*>(dst) = make_uint4(w[0], w[1], w[2], w[3]);
}

// ---------------------------------------------------------------------------------------
// per-row scale: one pass, row resident in registers
// ---------------------------------------------------------------------------------------
// Two kernels.  Rows straight from global memory, a CTA for each row or few, or, for 4-byte elements alone, through shared memory to
// persistent CTAs of whole warps per row.  The copies pay where a row fills those warps (up to four lanes of its last may idle) or where
// the direct kernel's threads, a power of two of them, are more (float32, order 16, 4-bit Philox codes, us, direct and staged: 40000 x 2560
// 107.1 and 99.5, 1024 columns 33.4 and 33.1, but 528 29.3 and 33.4, 1088 60.0 and 64.1); for codes that take little arithmetic they pay beside
// the exchanges of order 64 whatever idles (640 columns, nearest, 39.1 and 35.3; 1088 74.5 and 73.5).  Rows of 2-byte elements are bound
// by issue, and the copies only add to it (16384 x 4096 bf16 47.3 and 47.2, 58932 x 384 22.7 and 25.1, 32768 x 8192 213 and 217).
//
// kPairs: pairs of runs per thread (1 or 2).  tpr, the threads of a row: the power of two that gives each one pair, from 4 to
// the CTA: short rows share a warp.
template <typename T, int ROUND, int STORE4, int kPairs, int N>
__global__ void __launch_bounds__(kThreads) row_ht_quant_rowscale_kernel(
    const T* __restrict__ x, int64_t rows, int cols, int64_t ldx, int n, QuantDev q, uint8_t* __restrict__ codes,
    int64_t ld_codes, float* __restrict__ scales, int tpr, bool wide) {
  __shared__ float s_part[kThreads / 32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int rows_per_cta = kThreads / tpr;
  const int64_t row = (int64_t)blockIdx.x * rows_per_cta + threadIdx.x / tpr;
  const int t = threadIdx.x % tpr;
  const int nrun = cols >> 4;
  const bool row_ok = row < rows;
  const T* xr = x + (row_ok ? row : 0) * ldx;

  float2 v[kPairs][16];
  float mx = 0.0f;
#pragma unroll
  for (int j = 0; j < kPairs; ++j) {
    const int ri = 2 * (t + j * tpr);
    const T* p = xr + (int64_t)ri * 16;
    Raw32<T> raw;
    raw.load(p, p + 16, row_ok && ri < nrun, row_ok && ri + 1 < nrun, wide);
    raw.unpack(v[j]);
  }
#pragma unroll
  for (int j = 0; j < kPairs; ++j) {
    butterfly32<N>(v[j], n, lane);
    mx = fmaxf(mx, absmax32(v[j]));
  }
  for (int m = (tpr < 32 ? tpr : 32) >> 1; m; m >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xFFFFFFFFu, mx, m));
  if (tpr > 32) {
    if (lane == 0) s_part[warp] = mx;
    __syncthreads();
    const int w0 = (threadIdx.x / tpr) * (tpr / 32);
    mx = 0.0f;
    for (int w = 0; w < tpr / 32; ++w) mx = fmaxf(mx, s_part[w0 + w]);
  }
  const ScalePair sp = scale_from_absmax(mx, q.qmax);
  if (!row_ok) return;
  if (t == 0) scales[row] = sp.s;
  uint8_t* cr = codes + row * ld_codes;
#pragma unroll
  for (int j = 0; j < kPairs; ++j) {
    const int ri = 2 * (t + j * tpr);
    if (ri < nrun) {
      const bool ok1 = ri + 1 < nrun;
      uint32_t w[2][4];
      const uint64_t e0 = (uint64_t)row * (uint64_t)cols + (uint64_t)ri * 16u;
      quantise32<ROUND, STORE4, false>(v[j], sp, q, e0, true, ok1, w);
      uint8_t* dst = cr + (int64_t)ri * (STORE4 ? 8 : 16);
      if (STORE4 && ok1 && ((uintptr_t)dst & 15) == 0) {
        *reinterpret_cast<uint4*>(dst) = make_uint4(w[0][0], w[0][1], w[1][0], w[1][1]);
      } else {
        store_run<STORE4>(dst, w[0]);
        if (ok1) store_run<STORE4>(dst + (STORE4 ? 8 : 16), w[1]);
      }
    }
  }
}

// tpr: from a warp per row on as many whole warps as give each thread one pair, up to the CTA.
template <typename T, int ROUND, int STORE4, int kPairs, int N>
__global__ void __launch_bounds__(kThreads, kPairs == 1 ? 3 : 1) row_ht_quant_rowscale_staged_kernel(
    const T* __restrict__ x, int64_t rows, int cols, int64_t ldx, int n, QuantDev q, uint8_t* __restrict__ codes,
    int64_t ld_codes, float* __restrict__ scales, int tpr, int rows_per_cta) {
  using W = WarpTile<T>;
  extern __shared__ __align__(16) uint8_t smem[];
  __shared__ float s_part[2][kThreads / 32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int in_cta = threadIdx.x / tpr, t = threadIdx.x - in_cta * tpr;
  const int nrun = cols >> 4;
  const uint32_t tile = smem_u32(smem) + (uint32_t)(warp * kPairs * W::kBytes);
  const int shift = 31 - __clz(tpr), warp_row = warp * 32 / tpr;  // (below a warp per row, tpr is a power of two)
  const int row_bytes = cols * (int)sizeof(T);
  // the next row or rows of this warp; pieces past a row's end are zeros
  auto fetch = [&](int64_t row0) {
    const int64_t row_w = row0 + warp_row;
    if (tpr >= 32) {
      const int at0 = (warp * 32 - warp_row * tpr) * W::kPieces * 16 + lane * 16;  // the warp's pieces lie one after the other
      const char* src = reinterpret_cast<const char*>(x + row_w * ldx) + at0;
      const int left = row_w < rows ? row_bytes - at0 : 0;
#pragma unroll
      for (int j = 0; j < kPairs; ++j)
#pragma unroll
        for (int k = 0; k < W::kPieces; ++k) {
          const int off = j * kThreads * W::kPieces * 16 + k * 512;  // (two pairs per thread: tpr is the CTA)
          const bool ok = off < left;
          copy_piece(W::to(tile + j * W::kBytes, k, lane), ok ? src + off : reinterpret_cast<const char*>(x), ok);
        }
    } else {
#pragma unroll
      for (int k = 0; k < W::kPieces; ++k) {
        const int p = k * 32 + lane, owner = p / W::kPieces, at = ((owner & (tpr - 1)) * W::kPieces + p % W::kPieces) * 16;
        const int64_t row = row_w + (owner >> shift);
        const bool ok = row < rows && at < row_bytes;
        copy_piece(W::to(tile, k, lane), reinterpret_cast<const char*>(x) + (ok ? row * ldx * (int64_t)sizeof(T) + at : 0), ok);
      }
    }
    copy_commit();
  };

  const int64_t step = (int64_t)gridDim.x * rows_per_cta;
  int64_t row0 = (int64_t)blockIdx.x * rows_per_cta;
  fetch(row0);
#pragma unroll 1
  for (int turn = 0; row0 < rows; row0 += step, turn ^= 1) {
    const int64_t row = row0 + in_cta;
    const bool row_ok = row < rows;
    float2 v[kPairs][16];
    copy_wait<0>();
    __syncwarp();
#pragma unroll
    for (int j = 0; j < kPairs; ++j) W::read(tile + j * W::kBytes, lane, v[j]);
    __syncwarp();
    fetch(row0 + step);
    float mx = 0.0f;
#pragma unroll
    for (int j = 0; j < kPairs; ++j) {
      butterfly32<N>(v[j], n, lane);
      mx = fmaxf(mx, absmax32(v[j]));
    }
    for (int m = (tpr < 32 ? tpr : 32) >> 1; m; m >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xFFFFFFFFu, mx, m));
    if (tpr > 32) {
      if (lane == 0) s_part[turn][warp] = mx;
      __syncthreads();  // (one barrier a turn: the other half of s_part is the next turn's)
      const int w0 = in_cta * (tpr >> 5);
      mx = 0.0f;
      for (int w = 0; w < tpr >> 5; ++w) mx = fmaxf(mx, s_part[turn][w0 + w]);
    }
    const ScalePair sp = scale_from_absmax(mx, q.qmax);
    if (!row_ok) continue;
    if (t == 0) scales[row] = sp.s;
    uint8_t* cr = codes + row * ld_codes;
#pragma unroll
    for (int j = 0; j < kPairs; ++j) {
      const int ri = 2 * (t + j * tpr);
      if (ri < nrun) {
        const bool ok1 = ri + 1 < nrun;
        uint32_t w[2][4];
        const uint64_t e0 = (uint64_t)row * (uint64_t)cols + (uint64_t)ri * 16u;
        quantise32<ROUND, STORE4, false>(v[j], sp, q, e0, true, ok1, w);
        uint8_t* dst = cr + (int64_t)ri * (STORE4 ? 8 : 16);
        if (STORE4 && ok1 && ((uintptr_t)dst & 15) == 0) {
          *reinterpret_cast<uint4*>(dst) = make_uint4(w[0][0], w[0][1], w[1][0], w[1][1]);
        } else {
          store_run<STORE4>(dst, w[0]);
          if (ok1) store_run<STORE4>(dst + (STORE4 ? 8 : 16), w[1]);
        }
      }
    }
  }
  copy_wait<0>();
}

// ---------------------------------------------------------------------------------------
// per-tensor scale: pass 1 (abs-max) and pass 2 (quantise), streaming over pairs of runs
// ---------------------------------------------------------------------------------------
// A warp takes 32 neighbouring pairs at a time and has the next ones on their way.
template <typename T>
struct Stream {
  static constexpr int kCtasPerSm = 3;  // (80 registers a thread; 48 or 64 KB of tiles a CTA)
  static constexpr int kStages = sizeof(T) == 2 ? 3 : 2;
  static constexpr int kBytes = kThreads / 32 * kStages * WarpTile<T>::kBytes;
};

// The streamed tensor, row-major over rows x nrun runs; contig, contig_q: the rows of x, of the codes, follow one another without a gap,
// so that no division is needed.
struct Runs {
  int64_t total, ldx, ld_codes;
  int nrun;
  FastDiv by_nrun;
  bool contig, contig_q, wide;  // wide: runs start on 32-byte boundaries
  // A run in the tensor, worked out once for a warp's 64 neighbouring ones.  (With a quotient of its own for every 16-byte piece and
  // every run of codes, on both sides where only one had gaps, 40000 x 1040 float32 to 4-bit codes took 100.4 us; now 60.8.)
  struct Spot {
    int64_t row;
    int run;
  };
  __device__ __forceinline__ Spot spot(int64_t item) const {
    const int64_t row = item >> 31 ? item / nrun : (int64_t)((int)item / by_nrun);
    return {row, (int)(item - row * nrun)};
  }
  // where the run `ahead` (0 .. 63) behind that one begins, for rows of `ld` elements and runs of `size`
  __device__ __forceinline__ int64_t at(const Spot& s, int ahead, int64_t ld, int size) const {
    const int run = s.run + ahead, rows = run / by_nrun;
    return (s.row + rows) * ld + (int64_t)((run - rows * nrun) * size);
  }
};

// The 64 runs from `first` on to this warp's tile (runs outside 0 .. total: zeros)
template <typename T>
__device__ __forceinline__ void fetch_runs(uint32_t tile, const T* __restrict__ x, int64_t first, const Runs& t, int lane) {
  using W = WarpTile<T>;
  constexpr int kPerRun = W::kPieces / 2;
  if (t.contig && first >= 0 && first + 64 <= t.total) {
    const char* src = reinterpret_cast<const char*>(x + first * 16) + lane * 16;
#pragma unroll
    for (int k = 0; k < W::kPieces; ++k)
      asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(W::to(tile, k, lane)), "l"(src + k * 512) : "memory");
  } else if (first >= 0 && first < t.total) {  // (a loop: unrolled, it costs the streaming loop registers that it spills)
    const Runs::Spot s = t.spot(first);
    const int left = (int)(t.total - first < 64 ? t.total - first : 64);
#pragma unroll 1
    for (int k = 0; k < W::kPieces; ++k) {
      const int p = k * 32 + lane, ahead = p / kPerRun;
      const bool ok = ahead < left;
      copy_piece(W::to(tile, k, lane), reinterpret_cast<const char*>(x + (ok ? t.at(s, ahead, t.ldx, 16) : 0)) + (ok ? p % kPerRun * 16 : 0), ok);
    }
  }
  copy_commit();
}

// 2-byte elements come straight from global memory here: the pass is at what HBM gives, and the copies through shared memory only cost
// it CTAs (16384 x 4096 bf16 27.3 us, 29.5 with them, at 134 MB read and 20 MB of an earlier call's codes written back).
template <typename T, int N>
__global__ void __launch_bounds__(kThreads, sizeof(T) == 2 ? 4 : 3) row_ht_absmax_kernel(const T* __restrict__ x, Runs t, int64_t sample, int n,
                                                                                               uint32_t* __restrict__ absmax) {
  launch_dependents();  // (the second pass's CTAs come in as these leave, and wait for all of them)
  // blockIdx.y: sample of a batched call (one abs-max word per sample)
  extern __shared__ __align__(16) uint8_t smem[];
  using W = WarpTile<T>;
  constexpr int kStages = Stream<T>::kStages;
  x += (int64_t)blockIdx.y * sample;
  absmax += blockIdx.y;
  const int lane = threadIdx.x & 31;
  const int64_t step = (int64_t)gridDim.x * (2 * kThreads);
  int64_t first = (int64_t)blockIdx.x * (2 * kThreads) + (int64_t)(threadIdx.x >> 5) * 64;  // this warp's next 64 runs
  float mx = 0.0f;
  if constexpr (sizeof(T) == 2) {
    for (; first < t.total; first += step) {
      const int64_t item = first + 2 * lane;
      const bool ok0 = item < t.total, ok1 = item + 1 < t.total;
      const T *p0 = x + item * 16, *p1 = p0 + 16;
      if (!t.contig) {
        const Runs::Spot s = t.spot(first);
        p0 = x + t.at(s, 2 * lane, t.ldx, 16);
        p1 = x + t.at(s, 2 * lane + 1, t.ldx, 16);
      }
      Raw32<T> raw;
      raw.load(ok0 ? p0 : x, ok1 ? p1 : x, ok0, ok1, t.wide);
      float2 v[16];
      raw.unpack(v);
      butterfly32<N>(v, n, lane);
      mx = fmaxf(mx, absmax32(v));
    }
    mx = warp_max(mx);
    if (lane == 0) atomic_absmax(absmax, mx);
    return;
  }
  const uint32_t ring = smem_u32(smem) + (threadIdx.x >> 5) * (uint32_t)(kStages * W::kBytes);
#pragma unroll
  for (int k = 0; k < kStages - 1; ++k) fetch_runs(ring + k * W::kBytes, x, first + k * step, t, lane);
  int stage = 0;
  for (; first < t.total; first += step) {
    fetch_runs(ring + (stage == 0 ? kStages - 1 : stage - 1) * W::kBytes, x, first + (kStages - 1) * step, t, lane);
    copy_wait<kStages - 1>();
    __syncwarp();
    float2 v[16];
    W::read(ring + stage * W::kBytes, lane, v);
    __syncwarp();
    butterfly32<N>(v, n, lane);
    mx = fmaxf(mx, absmax32(v));
    stage = stage + 1 == kStages ? 0 : stage + 1;
  }
  copy_wait<0>();
  mx = warp_max(mx);
  if (lane == 0) atomic_absmax(absmax, mx);
}

template <typename T, int ROUND, int STORE4, int N>
__global__ void __launch_bounds__(kThreads, Stream<T>::kCtasPerSm) row_ht_quant_tensorscale_kernel(
    const T* __restrict__ x, Runs t, int64_t sample, int64_t sample_codes, int n, QuantDev q, uint8_t* __restrict__ codes,
    float* __restrict__ scales, const uint32_t* absmax) {
  // blockIdx.y: sample of a batched call; the Philox / noise element index runs on across samples
  extern __shared__ __align__(16) uint8_t smem[];
  using W = WarpTile<T>;
  constexpr int kStages = Stream<T>::kStages;
  x += (int64_t)blockIdx.y * sample;
  codes += (int64_t)blockIdx.y * sample_codes;
  const uint64_t e_base = (uint64_t)blockIdx.y * (uint64_t)t.total * 16u;
  constexpr int kRunBytes = STORE4 ? 8 : 16;
  const int lane = threadIdx.x & 31;
  const int64_t step = (int64_t)gridDim.x * (2 * kThreads);
  const int64_t last = (t.total - 1) & ~63ll;  // the tensor's last 64 runs, where this pass begins
  int64_t first = last - ((int64_t)blockIdx.x * (2 * kThreads) + (int64_t)(threadIdx.x >> 5) * 64);
  const uint32_t ring = smem_u32(smem) + (threadIdx.x >> 5) * (uint32_t)(kStages * W::kBytes);
#pragma unroll
  for (int k = 0; k < kStages - 1; ++k) fetch_runs(ring + k * W::kBytes, x, first - k * step, t, lane);
  wait_for_predecessor();  // (x is no work of the first pass: its copies were under way before)
  const ScalePair sp = scale_from_absmax(__uint_as_float(load_result(absmax + blockIdx.y)), q.qmax);
  if (blockIdx.x == 0 && threadIdx.x == 0) scales[blockIdx.y] = sp.s;
  const bool flat = t.contig_q && (e_base & 31) == 0 && ((uintptr_t)codes & 15) == 0;
  int stage = 0;
  for (; first >= 0; first -= step) {
    fetch_runs(ring + (stage == 0 ? kStages - 1 : stage - 1) * W::kBytes, x, first - (kStages - 1) * step, t, lane);
    copy_wait<kStages - 1>();
    __syncwarp();
    const int64_t item = first + 2 * lane;
    const bool ok0 = item < t.total, ok1 = item + 1 < t.total;
    float2 v[16];
    W::read(ring + stage * W::kBytes, lane, v);
    __syncwarp();
    butterfly32<N>(v, n, lane);
    uint32_t w[2][4];
    // logical element index of the pair: row * cols + col == item * 16 in either layout; whole tiles need no look at the halves of
    // Philox blocks, or, in codes without gaps, at where their runs lie
    const uint64_t e0 = e_base + (uint64_t)item * 16u;
    if (flat && first + 64 <= t.total) {
      quantise32<ROUND, STORE4, true>(v, sp, q, e0, true, true, w);
      uint8_t* dst = codes + item * kRunBytes;
      if (STORE4) {
        *reinterpret_cast<uint4*>(dst) = make_uint4(w[0][0], w[0][1], w[1][0], w[1][1]);
      } else {
        store_run<STORE4>(dst, w[0]);
        store_run<STORE4>(dst + 16, w[1]);
      }
    } else {
      quantise32<ROUND, STORE4, false>(v, sp, q, e0, ok0, ok1, w);
      const Runs::Spot s = t.spot(first);
      if (ok0) store_run<STORE4>(codes + t.at(s, 2 * lane, t.ld_codes, kRunBytes), w[0]);
      if (ok1) store_run<STORE4>(codes + t.at(s, 2 * lane + 1, t.ld_codes, kRunBytes), w[1]);
    }
    stage = stage + 1 == kStages ? 0 : stage + 1;
  }
  copy_wait<0>();
}

template <typename K>
int allow_smem(K kernel, int bytes, PerDeviceOnce& once) {
  bool done = false;
  const int dev = once.current(&done);
  if (dev < 0) HOT_FAIL(HOT_ERR_CUDA, "hot_row_ht_quant: cannot query the current CUDA device");
  if (!done) {
    HOT_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes));
    once.mark(dev);
  }
  return HOT_OK;
}

int grid_for(int64_t total_runs, int device_sms, int ctas_per_sm) {
  int64_t want = ((total_runs + 1) / 2 + kThreads - 1) / kThreads;
  const int64_t cap = (int64_t)device_sms * ctas_per_sm;
  if (want > cap) want = cap;
  if (want < 1) want = 1;
  return (int)want;
}

template <typename T, int ROUND, int STORE4>
int launch_typed(const T* x, int64_t rows, int cols, int64_t ldx, int n, const hot_quant_t& hq, uint8_t* codes,
                 int64_t ld_codes, float* scales, uint32_t* absmax_ws, cudaStream_t st, int sms, int batch) {
  const QuantDev q = make_quant_dev(hq);
  if (hq.scale_mode == HOT_SCALE_ROW) {
    const int npair = ((cols >> 4) + 1) / 2;
    int tpr = 4;
    while (tpr < kThreads && tpr < npair) tpr <<= 1;  // one pair per thread while a CTA can hold the row
    const int warps_tpr = npair >= kThreads ? kThreads : (npair + 31) / 32 * 32;
    // (see above the kernels; rows of more than kThreads pairs are the staged kernel's alone)
    const bool light = n == 64 && ROUND != HOT_ROUND_STOCH_NOISE && (STORE4 || ROUND == HOT_ROUND_NEAREST);
    const bool staged = sizeof(T) == 4 && npair > 16 && (warps_tpr < tpr || npair + 4 >= warps_tpr || light);
    if (staged) tpr = warps_tpr;
    if (npair > kMaxPairs * tpr)
      HOT_FAIL(HOT_ERR_UNSUPPORTED, "hot_row_ht_quant: per-row scale supports cols <= %d (got %d)", kMaxPairs * 32 * kThreads, cols);
    const int rows_per_cta = kThreads / tpr;
    const int64_t groups = (rows + rows_per_cta - 1) / rows_per_cta;
    if constexpr (sizeof(T) == 4) {
      if (staged) {
        auto run = [&](auto kernel, int pairs, PerDeviceOnce& once) -> int {
          const int warp_bytes = pairs * WarpTile<T>::kBytes, threads = rows_per_cta * tpr;
          if (int rc = allow_smem(kernel, kThreads / 32 * warp_bytes, once)) return rc;
          const int64_t most = (int64_t)sms * (pairs == 1 ? 3 * kThreads / threads : 1);
          kernel<<<(unsigned)(groups < most ? groups : most), threads, threads / 32 * warp_bytes, st>>>(x, rows, cols, ldx, n, q, codes, ld_codes, scales, tpr,
                                                                                                        rows_per_cta);
          HOT_CUDA(cudaGetLastError());
          return HOT_OK;
        };
        static PerDeviceOnce once2, once16, once32, once64, once0;
        return npair > tpr ? run(row_ht_quant_rowscale_staged_kernel<T, ROUND, STORE4, 2, 0>, 2, once2)
               : n == 16   ? run(row_ht_quant_rowscale_staged_kernel<T, ROUND, STORE4, 1, 16>, 1, once16)
               : n == 32   ? run(row_ht_quant_rowscale_staged_kernel<T, ROUND, STORE4, 1, 32>, 1, once32)
               : n == 64   ? run(row_ht_quant_rowscale_staged_kernel<T, ROUND, STORE4, 1, 64>, 1, once64)
                           : run(row_ht_quant_rowscale_staged_kernel<T, ROUND, STORE4, 1, 0>, 1, once0);
      }
    }
    const bool wide = (uintptr_t)x % 32 == 0 && ldx * sizeof(T) % 32 == 0;
    auto direct = [&](auto kernel) { kernel<<<(unsigned)groups, kThreads, 0, st>>>(x, rows, cols, ldx, n, q, codes, ld_codes, scales, tpr, wide); };
    if constexpr (sizeof(T) == 2) {  // (4-byte rows this long are staged)
      if (npair > tpr) direct(row_ht_quant_rowscale_kernel<T, ROUND, STORE4, 2, 0>);
    }
    if (npair <= tpr) {
      if (n == 16) direct(row_ht_quant_rowscale_kernel<T, ROUND, STORE4, 1, 16>);
      else if (n == 32) direct(row_ht_quant_rowscale_kernel<T, ROUND, STORE4, 1, 32>);
      else if (n == 64) direct(row_ht_quant_rowscale_kernel<T, ROUND, STORE4, 1, 64>);
      else direct(row_ht_quant_rowscale_kernel<T, ROUND, STORE4, 1, 0>);
    }
  } else {
    const Runs t = {rows * (cols >> 4), ldx, ld_codes, cols >> 4, fast_div(cols >> 4), ldx == cols, ld_codes == (STORE4 ? cols / 2 : cols),
                    (uintptr_t)x % 32 == 0 && ldx * sizeof(T) % 32 == 0};
    const int sms_per_sample = (sms + batch - 1) / batch;
    const dim3 grid((unsigned)grid_for(t.total, sms_per_sample, Stream<T>::kCtasPerSm), (unsigned)batch);
    constexpr bool kDirect = sizeof(T) == 2;  // (the first pass)
    const dim3 grid_s((unsigned)grid_for(t.total, sms_per_sample, kDirect ? 4 : Stream<T>::kCtasPerSm), (unsigned)batch);
    HOT_CUDA(cudaMemsetAsync(absmax_ws, 0, sizeof(uint32_t) * (size_t)batch, st));
    constexpr int kSmem = Stream<T>::kBytes;
    auto run = [&](auto stats, auto quantise, PerDeviceOnce& once_s, PerDeviceOnce& once_q) -> int {
      if (!kDirect)
        if (int rc = allow_smem(stats, kSmem, once_s)) return rc;
      if (int rc = allow_smem(quantise, kSmem, once_q)) return rc;
      stats<<<grid_s, kThreads, kDirect ? 0 : kSmem, st>>>(x, t, rows * ldx, n, absmax_ws);
      cudaLaunchAttribute attr[1];
      attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
      attr[0].val.programmaticStreamSerializationAllowed = 1;
      cudaLaunchConfig_t cfg = {};
      cfg.gridDim = grid;
      cfg.blockDim = dim3(kThreads);
      cfg.dynamicSmemBytes = kSmem;
      cfg.stream = st;
      cfg.attrs = attr;
      cfg.numAttrs = 1;
      HOT_CUDA(cudaLaunchKernelEx(&cfg, quantise, x, t, rows * ldx, rows * ld_codes, n, q, codes, scales, (const uint32_t*)absmax_ws));
      return HOT_OK;
    };
    static PerDeviceOnce once[8];
    int rc;
    switch (n) {
      case 16: rc = run(row_ht_absmax_kernel<T, 16>, row_ht_quant_tensorscale_kernel<T, ROUND, STORE4, 16>, once[0], once[1]); break;
      case 32: rc = run(row_ht_absmax_kernel<T, 32>, row_ht_quant_tensorscale_kernel<T, ROUND, STORE4, 32>, once[2], once[3]); break;
      case 64: rc = run(row_ht_absmax_kernel<T, 64>, row_ht_quant_tensorscale_kernel<T, ROUND, STORE4, 64>, once[4], once[5]); break;
      default: rc = run(row_ht_absmax_kernel<T, 0>, row_ht_quant_tensorscale_kernel<T, ROUND, STORE4, 0>, once[6], once[7]);
    }
    if (rc) return rc;
  }
  HOT_CUDA(cudaGetLastError());
  return HOT_OK;
}

template <typename T>
int launch_modes(const T* x, int64_t rows, int cols, int64_t ldx, int n, const hot_quant_t& q, uint8_t* codes,
                 int64_t ld_codes, float* scales, uint32_t* ws, cudaStream_t st, int sms, int batch) {
#define HOT_CASE(R, S)                                                                              \
  if (q.rounding == (R) && q.storage == (S))                                                        \
    return launch_typed<T, (R), (S)>(x, rows, cols, ldx, n, q, codes, ld_codes, scales, ws, st, sms, batch);
  HOT_CASE(HOT_ROUND_NEAREST, HOT_STORE_INT8)
  HOT_CASE(HOT_ROUND_NEAREST, HOT_STORE_INT4)
  HOT_CASE(HOT_ROUND_STOCH_PHILOX, HOT_STORE_INT8)
  if (q.rounding == HOT_ROUND_STOCH_PHILOX && q.bits < 4)
    return launch_typed<T, HOT_ROUND_STOCH_PHILOX, 2>(x, rows, cols, ldx, n, q, codes, ld_codes, scales, ws, st, sms, batch);
  HOT_CASE(HOT_ROUND_STOCH_PHILOX, HOT_STORE_INT4)
  HOT_CASE(HOT_ROUND_STOCH_NOISE, HOT_STORE_INT8)
  HOT_CASE(HOT_ROUND_STOCH_NOISE, HOT_STORE_INT4)
#undef HOT_CASE
  HOT_FAIL(HOT_ERR_ARG, "hot_row_ht_quant: bad rounding/storage %d/%d", q.rounding, q.storage);
}

}  // namespace

int device_sm_count();

}  // namespace hot

namespace hot {
namespace {
int row_ht_quant_impl(const void* x, int dtype, int64_t rows, int64_t cols, int64_t ldx, int order, const hot_quant_t* q,
                      void* codes, int64_t ld_codes, float* scales, uint32_t* absmax_ws, hot_stream_t stream, int batch) {
  if (rows == 0 && cols > 0 && q) return HOT_OK;  // nothing to do (and the pointers may be null)
  if (!x || !q || !codes || !scales) HOT_FAIL(HOT_ERR_ARG, "hot_row_ht_quant: null pointer");
  if (rows < 0 || cols <= 0) HOT_FAIL(HOT_ERR_ARG, "hot_row_ht_quant: bad shape %lld x %lld", (long long)rows, (long long)cols);
  if (int rc = validate_quant(q, "hot_row_ht_quant")) return rc;
  if (order < 1 || order > 64 || (order & (order - 1)))
    HOT_FAIL(HOT_ERR_UNSUPPORTED, "hot_row_ht_quant: order %d not a power of two in [1, 64]", order);
  if (cols % 16 != 0 || cols % order != 0 || cols > (1 << 30))
    HOT_FAIL(HOT_ERR_UNSUPPORTED, "hot_row_ht_quant: cols %lld must be a multiple of 16 and of the order %d",
             (long long)cols, order);
  const int esz = dtype == HOT_F32 ? 4 : 2;
  if (ldx < cols || (ldx * esz) % 16 != 0 || ((uintptr_t)x) % 16 != 0)
    HOT_FAIL(HOT_ERR_ARG, "hot_row_ht_quant: x and its pitch must be 16-byte aligned, ldx >= cols");
  const int64_t row_bytes = q->storage == HOT_STORE_INT4 ? cols / 2 : cols;
  if (ld_codes < row_bytes || ld_codes % 8 != 0 || (q->storage == HOT_STORE_INT8 && ld_codes % 16 != 0) ||
      ((uintptr_t)codes) % 16 != 0)
    HOT_FAIL(HOT_ERR_ARG, "hot_row_ht_quant: codes pitch %lld must be >= %lld and 16-byte aligned (8 for INT4)",
             (long long)ld_codes, (long long)row_bytes);
  if (q->scale_mode == HOT_SCALE_TENSOR && !absmax_ws) HOT_FAIL(HOT_ERR_ARG, "hot_row_ht_quant: absmax_ws is null");
  if (q->rounding == HOT_ROUND_STOCH_NOISE && ((uintptr_t)q->noise) % 16 != 0)
    HOT_FAIL(HOT_ERR_ARG, "hot_row_ht_quant: noise must be 16-byte aligned");
  cudaStream_t st = (cudaStream_t)stream;
  const int sms = device_sm_count();
  if (sms <= 0) return HOT_ERR_CUDA;
  if (dtype == HOT_F32)
    return launch_modes<float>((const float*)x, rows, (int)cols, ldx, order, *q, (uint8_t*)codes, ld_codes, scales,
                               absmax_ws, st, sms, batch);
  if (dtype == HOT_BF16)
    return launch_modes<__nv_bfloat16>((const __nv_bfloat16*)x, rows, (int)cols, ldx, order, *q, (uint8_t*)codes,
                                       ld_codes, scales, absmax_ws, st, sms, batch);
  HOT_FAIL(HOT_ERR_UNSUPPORTED, "hot_row_ht_quant: dtype %d", dtype);
}
}  // namespace
}  // namespace hot

extern "C" int hot_row_ht_quant(const void* x, int dtype, int64_t rows, int64_t cols, int64_t ldx, int order,
                                const hot_quant_t* q, void* codes, int64_t ld_codes, float* scales,
                                uint32_t* absmax_ws, hot_stream_t stream) {
  return hot::row_ht_quant_impl(x, dtype, rows, cols, ldx, order, q, codes, ld_codes, scales, absmax_ws, stream, 1);
}

extern "C" int hot_row_ht_quant_batched(const void* x, int dtype, int64_t batch, int64_t rows, int64_t cols, int64_t ldx,
                                        int order, const hot_quant_t* q, void* codes, int64_t ld_codes, float* scales,
                                        uint32_t* absmax_ws, hot_stream_t stream) {
  using namespace hot;
  if (batch < 1 || batch > 65535) HOT_FAIL(HOT_ERR_ARG, "hot_row_ht_quant_batched: batch %lld outside [1, 65535]", (long long)batch);
  if (!q) HOT_FAIL(HOT_ERR_ARG, "hot_row_ht_quant_batched: null pointer");
  if (q->scale_mode != HOT_SCALE_TENSOR)
    HOT_FAIL(HOT_ERR_UNSUPPORTED, "hot_row_ht_quant_batched: one scale per sample is HOT_SCALE_TENSOR; per-row scales do not depend on the batch");
  return row_ht_quant_impl(x, dtype, rows, cols, ldx, order, q, codes, ld_codes, scales, absmax_ws, stream, (int)batch);
}
