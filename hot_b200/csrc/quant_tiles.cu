// The quantisers of a layer, several tensors in one pair of launches: statistics, then codes.
//
// A job is one tensor [batch, rows, channels] with a row side (Hadamard along the channels, codes as they lie: grad_output
// for g_x), a column side (low-rank or Hadamard basis along the rows, codes transposed: grad_output for g_w, the weight, the
// activation buffer), or both, and optionally the sum over all rows (the bias gradient).  Every CTA of either launch takes
// one tile of one job: 64 channels (lane = a channel pair) by 64 to 256 rows, so that a small layer is two launches
// instead of a clear, an abs-max and a quantise launch per operand, and a large one has thousands of equal tiles.
//
//   row side     a thread takes 16 channels of a row, straight from global memory (32- or 64-byte pieces, four lanes
//                per 128-byte line), butterflies and quantises them in registers.
//   column side  a warp takes 16 rows (32 for the basis of 8 of 16) of 32 channel pairs, one 128-byte line per load,
//                butterflies on packed pairs.  Bases that keep every row, and the 8 of 16, leave 16 consecutive
//                positions of each channel in a thread's registers; other bases go through a float tile
//                [position][channel] in shared memory to the same form.  Codes leave as 16-byte pieces of the output
//                rows, straight from registers (half a sector each; a transpose through shared memory that made them
//                whole lines cost two barriers and more instructions than the stores).
// When both sides are on, the tile is read twice, the second time from L1.
//
// What bounds them: instruction issue (about 8 warp instructions per 32 row-side codes of 4 bits and 7 per 32 column-side
// codes of 8, Philox included, beside the butterflies), not HBM.  The separate kernels they stand in for (row_ht_quant,
// col_ht_quant) took 110 us for both sides of grad_output [64, 197, 2304] in bf16 and 15 us for the transposed codes
// of a 49 x 3072 tensor, whose 24 CTAs each ran a long serial tile.
//
// Statistics reach the second launch as one partial per CTA (no atomics, nothing to clear, the same every time): the
// abs-max of either side, per sample; per channel where the column side has a scale of its own for each; two doubles
// for the two-moment clip; and the row sums, whose chains (over 16 rows at a time, over warps, over partials) run in double: in
// float32 they were up to 3.7 times as far from the exact sum as torch's (8192 samples of 16 tokens), now they are nearer.
//
// The arithmetic is that of row_ht_quant / col_ht_quant (same butterflies, rounding and Philox indexing), so the codes are
// bit-identical to theirs; those kernels keep what is not covered here (explicit noise, orders above 16, odd columns).
#include "quant_tiles.cuh"

#include <cstring>
#include <type_traits>

namespace hot {

int device_sm_count();

namespace {

constexpr int kThreads = 128;
constexpr int kWarps = kThreads / 32;
constexpr int kRowLanes = kThreads / 4;  // rows a pass of the row side takes (four runs of 16 channels each)
constexpr int kCh = 64;                  // channels per tile

enum ColMode { kColNone = 0, kColAll = 1, kColHalf16 = 2, kColKept = 3 };
enum RowStore { kRowBytes8 = 0, kRowPacked4 = 1, kRowTimes16 = 2 };

struct DevJob {
  const void* x;
  int64_t ldx;
  int L, C;                 // rows per sample, channels
  int cblocks;              // 64-channel blocks
  int tt, tiles;            // rows per tile and tiles per sample (second launch)
  int ts, stiles;           // the same of the first launch
  FastDiv by_cblocks, by_tiles, by_stiles;
  // row side
  int row_on, n_row, row_philox, row_store;
  QuantDev qr;
  uint8_t* q_row;
  int64_t ld_row;
  float* s_row;
  float* part_row;          // [batch][stiles * cblocks]
  // column side
  int col_mode, n_col, col_philox, scale_mode;
  int group_pos;            // positions a group of 16 rows leaves (kColKept)
  int plain_stats;          // the row-side threads also take the column side's abs-max (order 1: no transform to do)
  signed char slot[16];     // position within the group of natural row i of the group, or -1 (kColKept)
  QuantDev qc;
  uint8_t* q_col;
  int64_t ld_col, sample_pitch;  // bytes; sample_pitch 0: one sample, rows of out_len codes
  int64_t row_codes;        // codes from one output row to the next in the Philox index
  int out_len;              // positions per sample
  float* s_col;
  float* part_col;          // [batch][stiles * cblocks], per channel [batch][stiles][C], two-moment: pairs of doubles
  // row sums
  float* part_sum;          // [batch * stiles][C], or null
  void* sum_out;            // [C] of the tensor's type
  int batch;
};

// The second job is always a weight: column side only, every row kept, one sample.
struct DevJobs {
  DevJob job[3];            // the main job, the weight, and another job of the main one's kind
  int third, sthird;        // first CTA of job[2], whose CTAs come after the main job's, in the second / first launch ...
  int first, sfirst;        // ... and of the weight, whose come last (beyond the grid: there is none)
  int sums;                 // CTAs of the second launch that add up row sums, before all of these (0: the first tiles' do)
};

template <typename T>
struct Pair;
template <>
struct Pair<float> {
  static __device__ __forceinline__ float2 load(const char* p) { return load_result(reinterpret_cast<const float2*>(p)); }
};
template <>
struct Pair<__nv_bfloat16> {
  static __device__ __forceinline__ float2 load(const char* p) {
    const uint32_t w = load_result(reinterpret_cast<const uint32_t*>(p));
    return make_float2(__uint_as_float(w << 16), __uint_as_float(w & 0xFFFF0000u));
  }
};

// 16 rows of a channel pair, `pitch` bytes apart (a row's address is then one multiply-add); rows at or past `valid` read
// as zeros.
// (FULL: there are 16).
template <typename T, bool FULL = false>
__device__ __forceinline__ void load_rows16(const char* at, uint32_t pitch, int valid, float2 (&v)[16]) {
#pragma unroll
  for (int t = 0; t < 16; ++t) v[t] = FULL || t < valid ? Pair<T>::load(at + (uint64_t)(uint32_t)t * pitch) : make_float2(0.0f, 0.0f);
}

// Order-n butterflies (n <= 16) on the blocks of n rows among 16, stages h = 1, 2, 4, 8 as everywhere
__device__ __forceinline__ void butterfly_rows16(float2 (&v)[16], int n) {
#pragma unroll
  for (int h = 1; h < 16; h <<= 1) {
    if (n <= h) break;
#pragma unroll
    for (int i = 0; i < 16; ++i)
      if ((i & h) == 0) {
        const float2 a = v[i], b = v[i + h];
        v[i] = add2(a, b);
        v[i + h] = sub2(a, b);
      }
  }
}

// maximum over a warp of non-negative values (their bit patterns order like integers)
__device__ __forceinline__ float warp_max_abs(float v) { return __uint_as_float(__reduce_max_sync(0xFFFFFFFFu, __float_as_uint(v))); }
// maximum of n non-negative partials, the same in every lane of every warp
__device__ __forceinline__ float max_of_partials(const float* p, int n) {
  float m = 0.0f;
  for (int i = threadIdx.x & 31; i < n; i += 32) m = fmaxf(m, load_result(p + i));
  return warp_max_abs(m);
}
__device__ __forceinline__ int warp_index() { return __shfl_sync(0xFFFFFFFFu, (int)(threadIdx.x >> 5), 0); }  // warp-uniform

__device__ __forceinline__ void launch_dependents() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
__device__ __forceinline__ void wait_for_predecessor() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

// abs-max of 16 raw elements as they lie in memory
template <typename T>
struct RawMax;
template <>
struct RawMax<float> {
  float m = 0.0f;
  __device__ __forceinline__ void add(const float2 (&v)[8], const float*) {
#pragma unroll
    for (int i = 0; i < 8; ++i) m = fmaxf(m, fmaxf(fabsf(v[i].x), fabsf(v[i].y)));
  }
  __device__ __forceinline__ float get() const { return m; }
};
template <>
struct RawMax<__nv_bfloat16> {  // on packed pairs, re-read from L1
  __nv_bfloat162 m = __nv_bfloat162(__ushort_as_bfloat16(0), __ushort_as_bfloat16(0));
  __device__ __forceinline__ void add(const float2 (&)[8], const __nv_bfloat16* p) {
    const uint4 a = load_result(reinterpret_cast<const uint4*>(p)), b = load_result(reinterpret_cast<const uint4*>(p) + 1);
    const uint32_t w[8] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w};
#pragma unroll
    for (int i = 0; i < 8; ++i) m = __hmax2(m, __habs2(*reinterpret_cast<const __nv_bfloat162*>(&w[i])));
  }
  __device__ __forceinline__ float get() const { return fmaxf(__low2float(m), __high2float(m)); }
};

// ---- first launch: statistics ---------------------------------------------------------------------
// WEIGHT: the second job's form (see DevJobs), so that its code is small and its parameters have fixed addresses.
template <typename T, int MODE, bool WEIGHT>
__device__ __forceinline__ void stats_tile(const DevJob& j, int at) {
  __shared__ float s_red[2][kWarps];
  __shared__ double s_mom[2][kWarps];
  __shared__ float s_ch[kWarps][kCh + 2];
  __shared__ __align__(16) float s_sum[kRowLanes][kCh + 4];
  const int rest = at / j.by_cblocks, cb = at - rest * j.cblocks;
  const int b = WEIGHT ? 0 : rest / j.by_stiles, tile = WEIGHT ? rest : rest - b * j.stiles;
  const int t0 = tile * j.ts, t1 = min(j.L, t0 + j.ts), c0 = cb * kCh;
  const int lane = threadIdx.x & 31, warp = warp_index();
  const T* x = reinterpret_cast<const T*>(j.x) + (int64_t)b * j.L * j.ldx;
  wait_for_predecessor();

  float max_row = 0.0f, max_col = 0.0f;
  const bool row_on = !WEIGHT && j.row_on;
  const bool sums = !WEIGHT && j.part_sum != nullptr;
  const bool col_part = WEIGHT || (MODE != kColNone && !(row_on && j.plain_stats));
  if (row_on) {
    const int run = threadIdx.x & 3, ch = c0 + run * 16;
    float2 sum[8];
    zero16(sum);
    RawMax<T> raw;
    if (ch < j.C) {
      const T* p = x + ch + (int64_t)(t0 + (int)(threadIdx.x >> 2)) * j.ldx;
#pragma unroll 2
      for (int t = t0 + (threadIdx.x >> 2); t < t1; t += kRowLanes, p += kRowLanes * j.ldx) {
        float2 v[8];
        Load16<T>::run(p, v);
        if (j.plain_stats) raw.add(v, p);
        if (sums && !col_part) {
#pragma unroll
          for (int i = 0; i < 8; ++i) sum[i] = add2(sum[i], v[i]);
        }
        butterfly16(v, j.n_row, lane);
        max_row = fmaxf(max_row, absmax16(v));
      }
    }
    max_col = raw.get();
    if (sums && !col_part) {
      float* to = &s_sum[threadIdx.x >> 2][run * 16];
#pragma unroll
      for (int i = 0; i < 8; i += 4) {
        *reinterpret_cast<float4*>(to + i) = make_float4(sum[i].x, sum[i + 1].x, sum[i + 2].x, sum[i + 3].x);
        *reinterpret_cast<float4*>(to + 8 + i) = make_float4(sum[i].y, sum[i + 1].y, sum[i + 2].y, sum[i + 3].y);
      }
      __syncthreads();
      const int c = threadIdx.x & 63, q = threadIdx.x >> 6;
      double s = 0.0;
#pragma unroll
      for (int i = 0; i < kRowLanes / 2; ++i) s += (double)s_sum[q * (kRowLanes / 2) + i][c];
      s_ch[q][c] = (float)s;
      __syncthreads();
      if (threadIdx.x < kCh && c0 + (int)threadIdx.x < j.C)
        j.part_sum[((int64_t)b * j.stiles + tile) * j.C + c0 + threadIdx.x] = s_ch[0][threadIdx.x] + s_ch[1][threadIdx.x];
    }
  }
  if (col_part || (sums && !row_on)) {
    const int ch = c0 + 2 * lane;
    const bool ok = ch < j.C;
    const bool sawb = MODE != kColNone && j.scale_mode == HOT_SCALE_SAWB;
    float2 m2 = make_float2(0.0f, 0.0f);
    double acc0 = 0.0, acc1 = 0.0;  // the two moments, or the sums of the two channels (no job has both)
    const uint32_t pitch = (uint32_t)j.ldx * (uint32_t)sizeof(T);
    const char* rows = reinterpret_cast<const char*>(x + (ok ? ch : 0));
    const bool whole = c0 + kCh <= j.C;
    for (int t = t0 + warp * 16; t < t1; t += kWarps * 16) {
      float2 v[16];
      const char* at = rows + (uint64_t)(uint32_t)t * pitch;
      if (whole && t1 - t >= 16) load_rows16<T, true>(at, pitch, 16, v);
      else load_rows16<T>(at, pitch, ok ? t1 - t : 0, v);
      if (sums) {
        float2 s4[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) s4[i] = add2(add2(v[4 * i], v[4 * i + 1]), add2(v[4 * i + 2], v[4 * i + 3]));
        const float2 s16 = add2(add2(s4[0], s4[1]), add2(s4[2], s4[3]));
        acc0 += (double)s16.x;
        acc1 += (double)s16.y;
      }
      if (MODE == kColNone) continue;
      constexpr int kN = MODE == kColHalf16 ? 8 : 16;
      float2 e[kN];
      if constexpr (MODE == kColHalf16) {
        butterfly_tokens16_even(v, e);
      } else {
        butterfly_rows16(v, j.n_col);
#pragma unroll
        for (int i = 0; i < 16; ++i) e[i] = MODE == kColKept && j.slot[i] < 0 ? make_float2(0.0f, 0.0f) : v[i];
      }
      if (sawb) {
        // in double throughout (the squares are exact there), so that the two means round to float once
#pragma unroll
        for (int i = 0; i < kN; ++i) {
          acc0 = fma((double)e[i].x, (double)e[i].x, fma((double)e[i].y, (double)e[i].y, acc0));
          acc1 += fabs((double)e[i].x) + fabs((double)e[i].y);
        }
      } else {
#pragma unroll
        for (int i = 0; i < kN; ++i) m2 = make_float2(fmaxf(m2.x, fabsf(e[i].x)), fmaxf(m2.y, fabsf(e[i].y)));
      }
    }
    max_col = fmaxf(max_col, fmaxf(m2.x, m2.y));
    if (sums) {
      s_ch[warp][2 * lane] = (float)acc0;
      s_ch[warp][2 * lane + 1] = (float)acc1;
      __syncthreads();
      if (threadIdx.x < kCh && c0 + (int)threadIdx.x < j.C) {
        double s = 0.0;
#pragma unroll
        for (int w = 0; w < kWarps; ++w) s += (double)s_ch[w][threadIdx.x];
        j.part_sum[((int64_t)b * j.stiles + tile) * j.C + c0 + threadIdx.x] = (float)s;
      }
      __syncthreads();
    }
    if (MODE != kColNone && j.scale_mode == HOT_SCALE_ROW) {
      s_ch[warp][2 * lane] = m2.x;
      s_ch[warp][2 * lane + 1] = m2.y;
      __syncthreads();
      if (threadIdx.x < kCh && c0 + (int)threadIdx.x < j.C) {
        float m = 0.0f;
#pragma unroll
        for (int w = 0; w < kWarps; ++w) m = fmaxf(m, s_ch[w][threadIdx.x]);
        j.part_col[((int64_t)b * j.stiles + tile) * j.C + c0 + threadIdx.x] = m;
      }
    } else if (sawb) {
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) {
        acc0 += __shfl_xor_sync(0xFFFFFFFFu, acc0, o);
        acc1 += __shfl_xor_sync(0xFFFFFFFFu, acc1, o);
      }
      if (lane == 0) {
        s_mom[0][warp] = acc0;
        s_mom[1][warp] = acc1;
      }
      __syncthreads();
      if (threadIdx.x < 2) {
        double s = 0.0;
        for (int w = 0; w < kWarps; ++w) s += s_mom[threadIdx.x][w];
        reinterpret_cast<double*>(j.part_col)[2 * (((int64_t)b * j.stiles + tile) * j.cblocks + cb) + threadIdx.x] = s;
      }
    }
  }
  max_row = warp_max_abs(max_row);
  max_col = warp_max_abs(max_col);
  if (lane == 0) {
    s_red[0][warp] = max_row;
    s_red[1][warp] = max_col;
  }
  __syncthreads();
  if (threadIdx.x < 2) {
    float m = s_red[threadIdx.x][0];
#pragma unroll
    for (int w = 1; w < kWarps; ++w) m = fmaxf(m, s_red[threadIdx.x][w]);
    const int64_t slot = ((int64_t)b * j.stiles + tile) * j.cblocks + cb;
    if (threadIdx.x == 0 && row_on) j.part_row[slot] = m;
    if (threadIdx.x == 1 && MODE != kColNone && j.scale_mode == HOT_SCALE_TENSOR) j.part_col[slot] = m;
  }
  launch_dependents();
}

template <typename T, int MODE>
__global__ void __launch_bounds__(kThreads, 6) tile_stats_kernel(const __grid_constant__ DevJobs jobs) {
  if ((int)blockIdx.x < jobs.sthird) stats_tile<T, MODE, false>(jobs.job[0], blockIdx.x);
  else if ((int)blockIdx.x < jobs.sfirst) stats_tile<T, MODE, false>(jobs.job[2], (int)blockIdx.x - jobs.sthird);
  else stats_tile<T, kColAll, true>(jobs.job[1], (int)blockIdx.x - jobs.sfirst);
}

// ---- second launch: codes ---------------------------------------------------------------------------
// the 16 random bytes of codes e0 .. e0 + 15 where e0 is not a multiple of 16: parts of two blocks
__device__ __forceinline__ uint4 philox_bytes_unaligned(const QuantDev& q, uint64_t e0) {
  const uint4 a = philox_block(q, e0 >> 4), b = philox_block(q, (e0 >> 4) + 1);
  const uint32_t o = (uint32_t)(e0 & 15u);
  uint32_t w[8] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w};
  if (o & 8u) {
#pragma unroll
    for (int i = 0; i < 6; ++i) w[i] = w[i + 2];
  }
  if (o & 4u) {
#pragma unroll
    for (int i = 0; i < 5; ++i) w[i] = w[i + 1];
  }
  const uint32_t s = 8u * (o & 3u);
  return make_uint4(__funnelshift_r(w[0], w[1], s), __funnelshift_r(w[1], w[2], s), __funnelshift_r(w[2], w[3], s),
                    __funnelshift_r(w[3], w[4], s));
}

// How a column side turns 16 values into codes, chosen once per tile so that the loop over its chunks has no choices left:
// Philox with 8-bit or 4-bit codes whose runs begin at whole runs of the random stream, to nearest, to nearest of values within
// a positive, finite clip, or anything.
enum CodeKind { kCodeAny = 0, kCode8 = 1, kCode4 = 2, kCodeNearest = 3, kCodeClipped = 4 };

// offset codes of 4 bits, one per byte -> sign-extended codes
__device__ __forceinline__ uint32_t finish_nibbles(uint32_t w) {
  w ^= 0x08080808u;
  return w | (((w & 0x08080808u) >> 3) * 0xF0u);
}

template <int KIND>
__device__ __forceinline__ uint4 philox_codes16(const uint32_t (&k)[16], const QuantDev& q, uint64_t e0) {
  if constexpr (KIND == kCode8) {
    const uint4 r = philox_block(q, e0 >> 4);
    return make_uint4(offset_codes4_rb8(k[0], k[1], k[2], k[3], r.x) ^ 0x80808080u, offset_codes4_rb8(k[4], k[5], k[6], k[7], r.y) ^ 0x80808080u,
                      offset_codes4_rb8(k[8], k[9], k[10], k[11], r.z) ^ 0x80808080u,
                      offset_codes4_rb8(k[12], k[13], k[14], k[15], r.w) ^ 0x80808080u);
  } else if constexpr (KIND == kCode4) {
    uint32_t r0, r1, w[4];
    philox_run_words4(q, e0, r0, r1);
    philox_run16_words(k, k + 8, true, r0, r1, 0u, 0u, w[0], w[1], w[2], w[3]);
#pragma unroll
    for (int i = 0; i < 4; ++i) w[i] = finish_nibbles((w[i] >> 4) & 0x0F0F0F0Fu);
    return make_uint4(w[0], w[1], w[2], w[3]);
  } else {
    // Sums in packed lanes on runs of 8, one by one elsewhere, as col_ht_quant does: the two differ in what the overflowing sum
    // of a NaN leaves.
    uint32_t w[4];
    const uint32_t off = (uint32_t)(q.qmax + 1.0f);
    const bool runs8 = (e0 & 7u) == 0;
    if (rand_bits(q.qmax) == 8) {
      const uint4 r = (e0 & 15u) == 0 ? philox_block(q, e0 >> 4) : philox_bytes_unaligned(q, e0);
      const uint32_t rw[4] = {r.x, r.y, r.z, r.w};
      if (runs8) {
#pragma unroll
        for (int i = 0; i < 4; ++i) w[i] = offset_codes4_rb8(k[4 * i], k[4 * i + 1], k[4 * i + 2], k[4 * i + 3], rw[i]);
      } else {
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          auto one = [&](int j) { return ((k[4 * i + j] & 0xFFFFu) + ((rw[i] >> (8 * j)) & 0xFFu)) >> 8; };
          w[i] = gather_low_bytes(one(0), one(1), one(2), one(3));
        }
      }
    } else {
      const uint4 a = philox_block(q, e0 >> 5), b = philox_block(q, (e0 + 15) >> 5);
      if (runs8) {
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const uint64_t e = e0 + (uint64_t)(4 * i);
          const uint4 blk = (e >> 5) == (e0 >> 5) ? a : b;
          const uint32_t word = (e & 16u) ? ((i & 1) ? blk.w : blk.z) : ((i & 1) ? blk.y : blk.x);
          w[i] = (offset_sums4_rb4(k[4 * i], k[4 * i + 1], k[4 * i + 2], k[4 * i + 3], (word >> ((e & 8u) ? 4 : 0)) & 0x0F0F0F0Fu) >> 4) & 0x0F0F0F0Fu;
        }
      } else {
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          auto one = [&](int j) {
            const uint64_t e = e0 + (uint64_t)(4 * i + j);
            return ((k[4 * i + j] & 0xFFFFu) + philox_r4((e >> 5) == (e0 >> 5) ? a : b, e)) >> 4;
          };
          w[i] = gather_low_bytes(one(0), one(1), one(2), one(3));
        }
      }
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) w[i] = __vsub4(w[i], off * 0x01010101u);
    return make_uint4(w[0], w[1], w[2], w[3]);
  }
}

// max(|a|, |b|, |c|), NaN if any of them is
__device__ __forceinline__ float absmax3_nan(float a, float b, float c) {
  float m;
  asm("max.NaN.abs.f32 %0, %1, %2, %3;" : "=f"(m) : "f"(a), "f"(b), "f"(c));
  return m;
}

__device__ __forceinline__ float code_range(float v, float qmax) { return v == v ? fminf(fmaxf(v, -qmax), qmax) : 0.0f; }

// 16 consecutive codes of two neighbouring channels: y[i] = (value i of channel c, value i of channel c + 1); e_a / e_b:
// Philox index of the first code of either.
// Nearest: the quotient (exact, as everywhere) plus 1.5 * 2^23 rounds half to even and leaves the code in the low byte.  The
// largest quotient is qmax within an ulp unless the tensor holds NaN or the scale is none (infinite, or the clip of a tensor of
// constant magnitude, which is negative): where one of the 32 is beyond, they are clamped, and a NaN gives code 0.  (Clipped
// values need no look: the moments behind the clip carry a NaN or an infinity, and the clip is then neither positive nor finite.)
template <int KIND>
__device__ __forceinline__ void quantise_pair16(float2 (&y)[16], const ScalePair& sa, const ScalePair& sb, const QuantDev& q, uint64_t e_a,
                                                uint64_t e_b, uint4& out_a, uint4& out_b) {
  uint32_t ka[16], kb[16];
  if constexpr (KIND != kCodeNearest && KIND != kCodeClipped) {
    const float2 mk2 = make_float2(sa.mk, sb.mk), ck2 = make_float2(sa.ck, sb.ck);
#pragma unroll
    for (int i = 0; i < 16; ++i) {
      const float2 t = __ffma2_rn(y[i], mk2, ck2);
      ka[i] = __float_as_uint(t.x);
      kb[i] = __float_as_uint(t.y);
    }
    out_a = philox_codes16<KIND>(ka, q, e_a);
    out_b = philox_codes16<KIND>(kb, q, e_b);
  } else {
    const float2 r2 = make_float2(sa.dv.r, sb.dv.r), nd2 = make_float2(-sa.dv.d, -sb.dv.d), magic = make_float2(kKMagic, kKMagic);
    auto quotient = [&](float2 v) {
      const float2 q0 = __fmul2_rn(v, r2);
      return __ffma2_rn(__ffma2_rn(q0, nd2, v), r2, q0);
    };
    if constexpr (KIND == kCodeNearest) {
      float largest = 0.0f;
#pragma unroll
      for (int i = 0; i < 16; ++i) {
        y[i] = quotient(y[i]);
        largest = absmax3_nan(largest, y[i].x, y[i].y);
      }
      if (!(largest < q.qmax + 0.5f)) {
#pragma unroll
        for (int i = 0; i < 16; ++i) y[i] = make_float2(code_range(y[i].x, q.qmax), code_range(y[i].y, q.qmax));
      }
    }
#pragma unroll
    for (int i = 0; i < 16; ++i) {
      const float2 t = add2(KIND == kCodeNearest ? y[i] : quotient(y[i]), magic);
      ka[i] = __float_as_uint(t.x);
      kb[i] = __float_as_uint(t.y);
    }
    out_a = make_uint4(gather_low_bytes(ka[0], ka[1], ka[2], ka[3]), gather_low_bytes(ka[4], ka[5], ka[6], ka[7]),
                       gather_low_bytes(ka[8], ka[9], ka[10], ka[11]), gather_low_bytes(ka[12], ka[13], ka[14], ka[15]));
    out_b = make_uint4(gather_low_bytes(kb[0], kb[1], kb[2], kb[3]), gather_low_bytes(kb[4], kb[5], kb[6], kb[7]),
                       gather_low_bytes(kb[8], kb[9], kb[10], kb[11]), gather_low_bytes(kb[12], kb[13], kb[14], kb[15]));
  }
}

template <typename T>
__device__ __forceinline__ void store_sum(void* out, int c, float v);
template <>
__device__ __forceinline__ void store_sum<float>(void* out, int c, float v) {
  reinterpret_cast<float*>(out)[c] = v;
}
template <>
__device__ __forceinline__ void store_sum<__nv_bfloat16>(void* out, int c, float v) {
  reinterpret_cast<__nv_bfloat16*>(out)[c] = __float2bfloat16_rn(v);
}

// The row side of a tile with 4-bit Philox codes stored as 16 * code.  A Philox block serves two neighbouring runs, i.e. the
// runs of lanes l and l ^ 1: over two rows, the even lane makes the block of the first, the odd lane that of the second,
// and they swap halves (SHARED: C is a multiple of 32, so that the two runs do lie in one block).
// N: the transform's order where it is 16, else 0.  FULL: both rows of every lane exist.
template <typename T, int N, bool SHARED, bool FULL>
__device__ __forceinline__ void row_pass_times16(const DevJob& j, const T* p, uint64_t e0, uint8_t* dst, bool ok0, bool ok1, const ScalePair& sp) {
  const bool odd = (threadIdx.x & 1) != 0;
  float2 v[2][8];
  if (FULL || ok0) Load16<T>::run(p, v[0]);
  else zero16(v[0]);
  if (FULL || ok1) Load16<T>::run(p + kRowLanes * j.ldx, v[1]);
  else zero16(v[1]);
  const uint64_t e1 = e0 + (uint64_t)kRowLanes * (uint64_t)j.C;
  uint32_t r[2][2];
  if (SHARED) {
    const uint4 blk = philox_block(j.qr, (odd ? e1 : e0) >> 5);
    // the words of my own run of the row whose block I made, and of my partner's run of it
    const uint32_t mine0 = odd ? blk.z : blk.x, mine1 = odd ? blk.w : blk.y;
    const uint32_t other0 = __shfl_xor_sync(0xFFFFFFFFu, odd ? blk.x : blk.z, 1), other1 = __shfl_xor_sync(0xFFFFFFFFu, odd ? blk.y : blk.w, 1);
    r[0][0] = odd ? other0 : mine0;
    r[0][1] = odd ? other1 : mine1;
    r[1][0] = odd ? mine0 : other0;
    r[1][1] = odd ? mine1 : other1;
  } else {
    philox_run_words4(j.qr, e0, r[0][0], r[0][1]);
    philox_run_words4(j.qr, e1, r[1][0], r[1][1]);
  }
  const float2 mk2 = make_float2(sp.mk, sp.mk), ck2 = make_float2(sp.ck, sp.ck);
#pragma unroll
  for (int u = 0; u < 2; ++u) {
    butterfly16(v[u], N ? N : j.n_row, 0);
    uint32_t ka[8], kb[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const float2 k = __ffma2_rn(v[u][i], mk2, ck2);
      ka[i] = __float_as_uint(k.x);
      kb[i] = __float_as_uint(k.y);
    }
    uint32_t wa0, wa1, wb0, wb1;
    philox_run16_words(ka, kb, true, r[u][0], r[u][1], 0u, 0u, wa0, wa1, wb0, wb1);
    // the sums' high nibbles are the offset codes: with the top bit flipped and the low nibble cleared a byte is 16 * code
    constexpr uint32_t keep = 0xF0F0F0F0u, flip = 0x80808080u;
    if (FULL || (u == 0 ? ok0 : ok1))
      *reinterpret_cast<uint4*>(dst + (u ? kRowLanes * j.ld_row : 0)) =
          make_uint4((wa0 & keep) ^ flip, (wa1 & keep) ^ flip, (wb0 & keep) ^ flip, (wb1 & keep) ^ flip);
  }
}
template <typename T, int N, bool SHARED>
__device__ __forceinline__ void row_side_times16(const DevJob& j, const T* x, int b, int t0, int c0, const ScalePair& sp) {
  const int ch = c0 + (threadIdx.x & 3) * 16, lane_row = threadIdx.x >> 2, t1 = min(j.L, t0 + j.tt);
  const int64_t row = (int64_t)b * j.L + t0 + lane_row;
  const T* p = x + (int64_t)(t0 + lane_row) * j.ldx + ch;
  uint64_t e0 = (uint64_t)row * (uint64_t)j.C + (uint64_t)ch;
  uint8_t* dst = j.q_row + row * j.ld_row + ch;
  const bool whole = c0 + kCh <= j.C;
  for (int t = t0; t < t1; t += 2 * kRowLanes) {
    if (whole && t + 2 * kRowLanes <= t1)
      row_pass_times16<T, N, SHARED, true>(j, p, e0, dst, true, true, sp);
    else
      row_pass_times16<T, N, SHARED, false>(j, p, e0, dst, ch < j.C && t + lane_row < t1, ch < j.C && t + lane_row + kRowLanes < t1, sp);
    p += 2 * kRowLanes * j.ldx;
    e0 += 2ull * kRowLanes * (uint64_t)j.C;
    dst += 2 * kRowLanes * j.ld_row;
  }
}

// The other forms of the row side: a run at a time.
template <typename T>
__device__ __forceinline__ void row_side_any(const DevJob& j, const T* x, int b, int t0, int c0, const ScalePair& sp) {
  const int ch = c0 + (threadIdx.x & 3) * 16, lane = threadIdx.x & 31, t1 = min(j.L, t0 + j.tt);
  if (ch >= j.C) return;
  const int code_bytes = j.row_store == kRowPacked4 ? 8 : 16;
  for (int t = t0 + (int)(threadIdx.x >> 2); t < t1; t += kRowLanes) {
    float2 v[8];
    Load16<T>::run(x + (int64_t)t * j.ldx + ch, v);
    butterfly16(v, j.n_row, lane);
    const int64_t row = (int64_t)b * j.L + t;
    const uint64_t e0 = (uint64_t)row * (uint64_t)j.C + (uint64_t)ch;
    uint8_t* dst = j.q_row + row * j.ld_row + (int64_t)(ch >> 4) * code_bytes;
    if (j.row_philox) {
      if (j.row_store == kRowPacked4) quantise_store16<HOT_ROUND_STOCH_PHILOX, 1>(v, sp, j.qr, e0, dst);
      else quantise_store16<HOT_ROUND_STOCH_PHILOX, 0>(v, sp, j.qr, e0, dst);
    } else if (j.row_store == kRowPacked4) {
      quantise_store16<HOT_ROUND_NEAREST, 1>(v, sp, j.qr, e0, dst);
    } else {
      quantise_store16<HOT_ROUND_NEAREST, 0>(v, sp, j.qr, e0, dst);
    }
  }
}

template <typename T, int MODE, bool APART, bool WEIGHT>
__device__ __forceinline__ void quant_tile(const DevJob& j, int at, uint8_t* smem) {
  __shared__ double s_mom[2][kWarps];
  const int rest = at / j.by_cblocks, cb = at - rest * j.cblocks;
  const int b = WEIGHT ? 0 : rest / j.by_tiles, tile = WEIGHT ? rest : rest - b * j.tiles;
  const int t0 = tile * j.tt, c0 = cb * kCh;
  const int lane = threadIdx.x & 31, warp = warp_index();
  const T* x = reinterpret_cast<const T*>(j.x) + (int64_t)b * j.L * j.ldx;
  const int parts = j.stiles * j.cblocks;
  wait_for_predecessor();

  if (!WEIGHT && j.row_on) {
    const ScalePair sp = scale_from_absmax(max_of_partials(j.part_row + (int64_t)b * parts, parts), j.qr.qmax);
    // (16 * code goes with a sixteenth of the scale, exact wherever a code is not 0: their product is the unstored one's, so it
    // overflows where that does)
    if (tile == 0 && cb == 0 && threadIdx.x == 0) j.s_row[b] = j.row_store == kRowTimes16 ? 0.0625f * sp.s : sp.s;
    if (j.row_store != kRowTimes16) row_side_any<T>(j, x, b, t0, c0, sp);
    else if (j.n_row == 16 && (j.C & 31) == 0) row_side_times16<T, 16, true>(j, x, b, t0, c0, sp);
    else row_side_times16<T, 0, false>(j, x, b, t0, c0, sp);
  }

  if (MODE != kColNone) {
    ScalePair sa, sb;
    float clip = 0.0f;
    const int ch = c0 + 2 * lane;
    const bool ok = ch < j.C;
    if (j.scale_mode == HOT_SCALE_TENSOR) {
      sa = scale_from_absmax(max_of_partials(j.part_col + (int64_t)b * parts, parts), j.qc.qmax);
      sb = sa;
      if (tile == 0 && cb == 0 && threadIdx.x == 0) j.s_col[b] = sa.s;
    } else if (j.scale_mode == HOT_SCALE_ROW) {
      float2 m2 = make_float2(0.0f, 0.0f);
      if (ok)
        for (int i = 0; i < j.stiles; ++i) {
          const float* p = j.part_col + ((int64_t)b * j.stiles + i) * j.C + ch;
          m2 = make_float2(fmaxf(m2.x, load_result(p)), fmaxf(m2.y, load_result(p + 1)));
        }
      sa = scale_from_absmax(m2.x, j.qc.qmax);
      sb = scale_from_absmax(m2.y, j.qc.qmax);
      if (tile == 0 && warp == 0 && ok) {
        j.s_col[(int64_t)b * j.C + ch] = sa.s;
        j.s_col[(int64_t)b * j.C + ch + 1] = sb.s;
      }
    } else {
      // clip = 12.1 * sqrt(mean(y^2)) - 12.2 * mean(|y|) over the transformed tensor (of this sample), the partials added
      // in a fixed order
      double sq = 0.0, ab = 0.0;
      const double* part = reinterpret_cast<const double*>(j.part_col) + 2 * (int64_t)b * parts;
      for (int i = threadIdx.x; i < parts; i += kThreads) {
        sq += load_result(part + 2 * i);
        ab += load_result(part + 2 * i + 1);
      }
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) {
        sq += __shfl_xor_sync(0xFFFFFFFFu, sq, o);
        ab += __shfl_xor_sync(0xFFFFFFFFu, ab, o);
      }
      if (lane == 0) {
        s_mom[0][warp] = sq;
        s_mom[1][warp] = ab;
      }
      __syncthreads();
      double tq = 0.0, ta = 0.0;
      for (int w = 0; w < kWarps; ++w) {
        tq += s_mom[0][w];
        ta += s_mom[1][w];
      }
      const double count = (double)j.out_len * (double)j.C;
      clip = __fsub_rn(__fmul_rn(12.1f, __fsqrt_rn((float)(tq / count))), __fmul_rn(12.2f, (float)(ta / count)));
      sa = scale_from_absmax(clip, j.qc.qmax);
      sb = sa;
      if (tile == 0 && cb == 0 && threadIdx.x == 0) j.s_col[b] = sa.s;
    }
    const int tile_pos = MODE == kColHalf16 ? j.tt / 2 : (MODE == kColAll ? j.tt : j.tt / 16 * j.group_pos);
    const int64_t pos0 = (int64_t)tile * tile_pos;  // first position of the tile
    const uint64_t e_ch = (uint64_t)ch * (uint64_t)j.row_codes + (uint64_t)b * (uint64_t)j.sample_pitch + (uint64_t)pos0;
    const uint32_t pitch = (uint32_t)j.ldx * (uint32_t)sizeof(T);
    const char* rows = reinterpret_cast<const char*>(x + (ok ? ch : 0)) + (uint64_t)(uint32_t)t0 * pitch;
    const int left = ok ? j.L - t0 : 0;  // rows of the sample from the tile on
    float* kept = reinterpret_cast<float*>(smem);
    if constexpr (MODE == kColKept) {
      const int groups = min(j.tt, j.L - t0 + 15) / 16;
      for (int g = warp; g < j.tt / 16; g += kWarps) {
        float2 v[16];
        if (g < groups) {
          const char* at = rows + (uint64_t)(uint32_t)(g * 16) * pitch;
          if (c0 + kCh <= j.C && left - g * 16 >= 16) load_rows16<T, true>(at, pitch, 16, v);
          else load_rows16<T>(at, pitch, left - g * 16, v);
          butterfly_rows16(v, j.n_col);
        } else {
#pragma unroll
          for (int i = 0; i < 16; ++i) v[i] = make_float2(0.0f, 0.0f);
        }
#pragma unroll
        for (int i = 0; i < 16; ++i) {
          const int s = j.slot[i];
          if (s >= 0) *reinterpret_cast<float2*>(kept + (g * j.group_pos + s) * kCh + 2 * lane) = v[i];
        }
      }
      __syncthreads();
    }
    // a sample's positions past its rows, up to the next sample, are zeros: chunks with no rows at all are not made
    const int64_t limit = !WEIGHT && j.sample_pitch > 0 ? j.sample_pitch : (int64_t)j.out_len;
    const int live = (int)min((int64_t)tile_pos, (int64_t)j.out_len - pos0);  // positions of the tile that have rows
    const int chunks = (live + 15) / 16;
    uint8_t* const out = j.q_col + (WEIGHT ? 0 : (int64_t)b * j.sample_pitch) + pos0 + (int64_t)(ok ? ch : 0) * j.ld_col;
    auto make_chunk = [&](auto kind, auto full, int chunk) {
      constexpr bool kFull = decltype(full)::value;
      float2 y[16];
      if constexpr (MODE == kColAll) {
        load_rows16<T, kFull>(rows + (uint64_t)(uint32_t)(chunk * 16) * pitch, pitch, left - chunk * 16, y);
        if (WEIGHT || j.n_col > 1) butterfly_rows16(y, j.n_col);
      } else if constexpr (MODE == kColHalf16) {
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          float2 v[16], e[8];
          load_rows16<T, kFull>(rows + (uint64_t)(uint32_t)(chunk * 32 + 16 * h) * pitch, pitch, left - chunk * 32 - 16 * h, v);
          butterfly_tokens16_even(v, e);
#pragma unroll
          for (int i = 0; i < 8; ++i) y[8 * h + kHalf16SlotOfEvenRow[i]] = e[i];
        }
      } else {
#pragma unroll
        for (int i = 0; i < 16; ++i) y[i] = *reinterpret_cast<const float2*>(kept + (chunk * 16 + i) * kCh + 2 * lane);
      }
      if (kind.value == kCodeClipped || (kind.value == kCodeNearest && j.scale_mode == HOT_SCALE_SAWB)) {
#pragma unroll
        for (int i = 0; i < 16; ++i) y[i] = make_float2(fminf(fmaxf(y[i].x, -clip), clip), fminf(fmaxf(y[i].y, -clip), clip));
      }
      uint4 qa, qb;
      const uint64_t e = e_ch + (uint64_t)(chunk * 16);
      quantise_pair16<kind.value>(y, sa, sb, j.qc, e, e + (uint64_t)j.row_codes, qa, qb);
      if (ok) {
        *reinterpret_cast<uint4*>(out + chunk * 16) = qa;
        *reinterpret_cast<uint4*>(out + chunk * 16 + j.ld_col) = qb;
      }
    };
    // whole chunks without bounds checks, then the one that may be ragged
    const int whole = c0 + kCh <= j.C ? (MODE == kColKept ? chunks : (j.L - t0) / (MODE == kColHalf16 ? 32 : 16)) : 0;
    auto make = [&](auto kind) {
      int chunk = warp;
      for (; chunk < min(chunks, whole); chunk += kWarps) make_chunk(kind, std::true_type(), chunk);
      for (; chunk < chunks; chunk += kWarps) make_chunk(kind, std::false_type(), chunk);
    };
    if (!j.col_philox && j.scale_mode == HOT_SCALE_SAWB && clip > 0.0f && clip <= 3.4028234e38f) make(std::integral_constant<int, kCodeClipped>());
    else if (!j.col_philox) make(std::integral_constant<int, kCodeNearest>());
    else if (j.qc.qmax == 127.0f && (j.row_codes & 15) == 0) make(std::integral_constant<int, kCode8>());
    else if (j.qc.qmax == 7.0f && (j.row_codes & 15) == 0) make(std::integral_constant<int, kCode4>());
    else make(std::integral_constant<int, kCodeAny>());
    if (!WEIGHT && j.sample_pitch > 0) {
      const int64_t end = tile == j.tiles - 1 ? limit : min(limit, pos0 + tile_pos);
      for (int chunk = chunks + warp; ok && pos0 + chunk * 16 < end; chunk += kWarps) {
        *reinterpret_cast<uint4*>(out + chunk * 16) = make_uint4(0u, 0u, 0u, 0u);
        *reinterpret_cast<uint4*>(out + chunk * 16 + j.ld_col) = make_uint4(0u, 0u, 0u, 0u);
      }
    }
  }

  if (!WEIGHT && !APART && j.part_sum && tile == 0 && b == 0) {  // the row sums of this channel block, partials in a fixed order
    __syncthreads();
    double* part = reinterpret_cast<double*>(smem);
    const int c = threadIdx.x & 63, q = threadIdx.x >> 6, n = j.batch * j.stiles;
    double s[4] = {0.0, 0.0, 0.0, 0.0};
    if (c0 + c < j.C) {
      const float* p = j.part_sum + c0 + c;
      for (int i = q; i < n; i += 8) {
        float v[4];
#pragma unroll
        for (int k = 0; k < 4; ++k) v[k] = load_result(p + (int64_t)(i + 2 * k < n ? i + 2 * k : i) * j.C);
#pragma unroll
        for (int k = 0; k < 4; ++k) s[k] += i + 2 * k < n ? (double)v[k] : 0.0;
      }
    }
    part[threadIdx.x] = (s[0] + s[1]) + (s[2] + s[3]);
    __syncthreads();
    if (threadIdx.x < kCh && c0 + c < j.C) store_sum<T>(j.sum_out, c0 + c, (float)(part[c] + part[64 + c]));
  }
  launch_dependents();
}

// Row sums of many partials (samples x tiles) come from CTAs of their own (APART): 16 channels each, the partials of every sample and
// tile in a fixed order, eight loads of a thread in flight.  Summed by the CTAs of the first tiles, half a channel's partials to a thread,
// they are a tail behind the codes: [32, 784, 128] in bf16, 416 partials, 26.9 us for both launches, 14.2 apart.  Few partials
// stay there: [64, 197, 2304] and its 64 take 64.7 us, 65.7 apart.  Between the two, steps of layers with 100 to 512 partials of 384 to 3072
// channels are within 1.5 % of one another either way.  (A slice of the channels to each of the first 8 or 16 CTAs, in one kernel: the
// same layers 0.99 to 1.01, the convolution's step 4 us of 157 slower.)
constexpr int kManyPartials = 128, kSumCh = 16;
template <typename T>
__device__ __forceinline__ void add_row_sums(const DevJob& j, int block, uint8_t* smem) {
  wait_for_predecessor();
  double2* const part = reinterpret_cast<double2*>(smem);
  constexpr int pairs = kSumCh / 2, lines = kThreads / pairs;
  const int pair = threadIdx.x % pairs, line = threadIdx.x / pairs, ch = 2 * (block * pairs + pair), n = j.batch * j.stiles;
  double2 s = make_double2(0.0, 0.0);
  if (ch < j.C) {
    const float* p = j.part_sum + (int64_t)line * j.C + ch;
    const int64_t step = (int64_t)lines * j.C;
    for (int i = line; i < n; i += 8 * lines, p += 8 * step) {
      float2 v[8];
#pragma unroll
      for (int k = 0; k < 8; ++k) v[k] = load_result(reinterpret_cast<const float2*>(i + k * lines < n ? p + k * step : p));  // (no branches)
#pragma unroll
      for (int k = 0; k < 8; ++k) {
        const bool in = i + k * lines < n;
        s.x += in ? (double)v[k].x : 0.0;
        s.y += in ? (double)v[k].y : 0.0;
      }
    }
  }
  part[threadIdx.x] = s;
  __syncthreads();
  const int c = block * kSumCh + (int)threadIdx.x;
  if ((int)threadIdx.x < kSumCh && c < j.C) {
    const double* q = reinterpret_cast<const double*>(part) + threadIdx.x;
    double t = 0.0;
#pragma unroll
    for (int k = 0; k < lines; ++k) t += q[k * kSumCh];
    store_sum<T>(j.sum_out, c, (float)t);
  }
  launch_dependents();
}

// CTAs per SM: six, whose 80 registers spill some words, but five where kept rows go through shared memory and for float32 with the
// basis of 8 of 16 (the extension call's three tensors of 6304 tokens: 44.0 us for both launches with six, 43.4 with five).
template <typename T, int MODE, bool APART>
__global__ void __launch_bounds__(kThreads, MODE == kColKept || (MODE == kColHalf16 && sizeof(T) == 4) ? 5 : 6) tile_quant_kernel(const __grid_constant__ DevJobs jobs) {
  extern __shared__ __align__(16) uint8_t smem[];  // kept rows as floats [position][64 channels]
  const int cta = (int)blockIdx.x - (APART ? jobs.sums : 0);  // (the row sums' CTAs come first)
  if (APART && cta < 0) add_row_sums<T>(jobs.job[0], blockIdx.x, smem);
  else if (cta < jobs.third) quant_tile<T, MODE, APART, false>(jobs.job[0], cta, smem);
  else if (cta < jobs.first) quant_tile<T, MODE, APART, false>(jobs.job[2], cta - jobs.third, smem);
  else quant_tile<T, kColAll, APART, true>(jobs.job[1], cta - jobs.first, smem);
}

// ---- host side --------------------------------------------------------------------------------------
#ifndef HOT_TILES_F32
bool is_half16(const TileJob& t) {
  if (!t.sel || t.order_col != 16 || t.rank != 8) return false;
  for (int i = 0; i < 8; ++i)
    if (t.sel[i] != kHalf16Sel[i]) return false;
  return true;
}
bool keeps_all(const TileJob& t) {
  if (t.rank != t.order_col) return false;
  for (int i = 0; t.sel && i < t.rank; ++i)
    if (t.sel[i] != i) return false;
  return true;
}

struct Geometry {
  int col_mode, cblocks, tt, tiles, ts, stiles, group_pos, tile_pos;
};

Geometry geometry_of(const TileJob& t) {
  Geometry g = {};
  g.col_mode = !t.col ? kColNone : (keeps_all(t) ? kColAll : (is_half16(t) ? kColHalf16 : kColKept));
  g.cblocks = (int)((t.channels + kCh - 1) / kCh);
  g.group_pos = g.col_mode == kColKept ? 16 / t.order_col * t.rank : 0;
  // Rows per tile of the second launch: 256, so that a CTA's four warps have a few groups of 16 rows each for the scales and
  // addresses they set up (with one group per warp that set-up was half of the instructions); fewer where the tensor is
  // so small that the chip would stand idle.  A tile's positions are whole runs of 16 codes: with an odd number per group
  // of rows only 256 will do.
  const int least = (g.group_pos & 1) ? 256 : (g.group_pos & 2) ? 128 : (g.col_mode == kColHalf16 ? 128 : 64);
  g.tt = g.col_mode == kColKept && least <= 128 ? 128 : 256;  // (kept rows are staged as floats: shorter tiles, more CTAs per SM)
  while (g.tt > least && t.batch * g.cblocks * ((t.rows + g.tt - 1) / g.tt) < 592) g.tt /= 2;
  g.tiles = (int)((t.rows + g.tt - 1) / g.tt);
  g.tile_pos = g.col_mode == kColHalf16 ? g.tt / 2 : (g.col_mode == kColKept ? g.tt / 16 * g.group_pos : g.tt);
  // Statistics: tall enough that the reductions at a tile's end cost little and the second launch has at most a few
  // hundred partials per sample to read, short enough that a small tensor still spreads over the chip.
  g.ts = 64;
  auto ctas = [&]() { return t.batch * g.cblocks * ((t.rows + g.ts - 1) / g.ts); };
  while (g.ts < t.rows && (ctas() > 1776 || (int64_t)g.cblocks * ((t.rows + g.ts - 1) / g.ts) > 768)) g.ts *= 2;
  g.stiles = (int)((t.rows + g.ts - 1) / g.ts);
  return g;
}

size_t align16(size_t v) { return (v + 15) / 16 * 16; }

// Lays the job's partials out behind `base` (null: only measures); returns the bytes they take.
size_t place_partials(const TileJob& t, const Geometry& g, uint8_t* base, DevJob* d) {
  size_t at = 0;
  auto take = [&](size_t bytes) {
    uint8_t* p = base ? base + at : nullptr;
    at += align16(bytes);
    return p;
  };
  const size_t parts = (size_t)t.batch * g.stiles * g.cblocks;
  uint8_t* pr = t.row ? take(parts * sizeof(float)) : nullptr;
  uint8_t* pc = nullptr;
  if (t.col) {
    if (t.q_col.scale_mode == HOT_SCALE_ROW) pc = take((size_t)t.batch * g.stiles * t.channels * sizeof(float));
    else if (t.q_col.scale_mode == HOT_SCALE_SAWB) pc = take(parts * 2 * sizeof(double));
    else pc = take(parts * sizeof(float));
  }
  uint8_t* ps = t.sum ? take((size_t)t.batch * g.stiles * t.channels * sizeof(float)) : nullptr;
  if (d) {
    d->part_row = (float*)pr;
    d->part_col = (float*)pc;
    d->part_sum = (float*)ps;
  }
  return at;
}

#endif  // HOT_TILES_F32

template <typename T, int MODE>
int launch_mode(const DevJobs& jobs, int stats_ctas, int quant_ctas, size_t smem, cudaStream_t st) {
  static PerDeviceOnce once;
  bool done = false;
  const int dev = once.current(&done);
  if (dev < 0) HOT_FAIL(HOT_ERR_CUDA, "quant_tiles: cannot query the current CUDA device");
  if (!done) {
    for (auto kernel : {tile_quant_kernel<T, MODE, false>, tile_quant_kernel<T, MODE, true>})
      HOT_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, 256 * kCh * (int)sizeof(float)));
    once.mark(dev);
  }
  // both may start while their predecessor on the stream drains; they wait for it before they touch memory
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t cfg = {};
  cfg.blockDim = dim3(kThreads);
  cfg.stream = st;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  cfg.gridDim = dim3((unsigned)stats_ctas);
  HOT_CUDA(cudaLaunchKernelEx(&cfg, tile_stats_kernel<T, MODE>, jobs));
  cfg.gridDim = dim3((unsigned)quant_ctas);
  cfg.dynamicSmemBytes = smem;
  HOT_CUDA(cudaLaunchKernelEx(&cfg, jobs.sums ? tile_quant_kernel<T, MODE, true> : tile_quant_kernel<T, MODE, false>, jobs));
  return HOT_OK;
}

template <typename T>
int launch_typed(const DevJobs& jobs, int stats_ctas, int quant_ctas, size_t smem, cudaStream_t st) {
  switch (jobs.job[0].col_mode) {
    case kColAll: return launch_mode<T, kColAll>(jobs, stats_ctas, quant_ctas, smem, st);
    case kColHalf16: return launch_mode<T, kColHalf16>(jobs, stats_ctas, quant_ctas, smem, st);
    case kColKept: return launch_mode<T, kColKept>(jobs, stats_ctas, quant_ctas, smem, st);
    default: return launch_mode<T, kColNone>(jobs, stats_ctas, quant_ctas, smem, st);
  }
}

}  // namespace

// The float32 instances are compiled from this file once more, by quant_tiles_f32.cu: half of what was by far the longest compilation.
int launch_tiles_f32(const void* jobs, int stats_ctas, int quant_ctas, size_t smem, cudaStream_t st);
#ifdef HOT_TILES_F32
int launch_tiles_f32(const void* jobs, int stats_ctas, int quant_ctas, size_t smem, cudaStream_t st) {
  return launch_typed<float>(*static_cast<const DevJobs*>(jobs), stats_ctas, quant_ctas, smem, st);
}
#else

// Whether a job is covered: Philox or nearest rounding, transforms of order up to 16, channel pairs that can be loaded at
// once, one byte per code on the column side; the row side takes one scale per sample and whole runs of 16 channels.
bool tile_job_covered(const TileJob& t, int dtype) {
  const int esz = dtype == HOT_F32 ? 4 : 2;
  if (dtype != HOT_F32 && dtype != HOT_BF16) return false;
  if (!t.x || t.batch < 1 || t.rows < 1 || t.rows >= (1ll << 30) || t.channels < 2 || t.channels % 2 || t.channels >= (1 << 30) || t.ldx < t.channels ||
      t.ldx % 2 || t.ldx * esz >= (1ll << 31) || ((uintptr_t)t.x) % (2 * esz))
    return false;
  const Geometry g = geometry_of(t);
  if (t.batch * (int64_t)g.cblocks * g.tiles >= (1ll << 30)) return false;
  if (t.row) {
    const hot_quant_t& q = t.q_row;
    if (q.scale_mode != HOT_SCALE_TENSOR || (q.rounding != HOT_ROUND_STOCH_PHILOX && q.rounding != HOT_ROUND_NEAREST) || q.bits < 2 || q.bits > 8 ||
        (q.storage == HOT_STORE_INT4 && q.bits > 4) || t.order_row < 1 || t.order_row > 16 || (t.order_row & (t.order_row - 1)) || t.channels % 16 ||
        (t.ldx * esz) % 16 || ((uintptr_t)t.x) % 16 || t.ld_row % 16 || ((uintptr_t)t.codes_row) % 16)
      return false;
  }
  if (t.col) {
    const hot_quant_t& q = t.q_col;
    if ((q.rounding != HOT_ROUND_STOCH_PHILOX && q.rounding != HOT_ROUND_NEAREST) ||
        (q.scale_mode == HOT_SCALE_SAWB && (q.rounding != HOT_ROUND_NEAREST || t.sum)) ||
        q.bits < 2 || q.bits > 8 || q.storage != HOT_STORE_INT8 || t.order_col < 1 || t.order_col > 16 || (t.order_col & (t.order_col - 1)) || t.rank < 1 ||
        t.rank > t.order_col || t.rows % t.order_col || t.ld_col % 16 || t.sample_pitch % 16 || ((uintptr_t)t.codes_col) % 16)
      return false;
    const int64_t len = t.rows / t.order_col * t.rank;
    if (t.sample_pitch ? (t.sample_pitch < len || t.ld_col < t.sample_pitch * t.batch) : (t.batch != 1 || t.ld_col < len)) return false;
  }
  return t.row || t.col || t.sum;
}

size_t tile_scratch_bytes(const TileJob* jobs, int count) {
  size_t total = 0;
  for (int i = 0; i < count; ++i) total += place_partials(jobs[i], geometry_of(jobs[i]), nullptr, nullptr);
  return total;
}

bool tile_jobs_alike(const TileJob& a, const TileJob& b) { return geometry_of(a).col_mode == geometry_of(b).col_mode; }

int launch_tile_jobs(const TileJob* jobs, int count, int dtype, void* scratch, size_t scratch_bytes, cudaStream_t st, const TileJob* third,
                     void* third_scratch) {
  if (count < 1 || count > kMaxTileJobs) HOT_FAIL(HOT_ERR_ARG, "quant_tiles: %d jobs", count);
  if (tile_scratch_bytes(jobs, count) > scratch_bytes || ((uintptr_t)scratch) % 16) HOT_FAIL(HOT_ERR_WORKSPACE, "quant_tiles: scratch too small or misaligned");
  DevJobs dev;
  memset(&dev, 0, sizeof(dev));
  dev.first = dev.sfirst = dev.third = dev.sthird = 1 << 30;
  int stats_ctas = 0, quant_ctas = 0;
  size_t smem = kThreads * sizeof(double2);
  uint8_t* at = (uint8_t*)scratch;
  for (int i : {0, 2, 1}) {
    if (i == 2 ? !third : i >= count) continue;
    const TileJob& t = i == 2 ? *third : jobs[i];
    if (!tile_job_covered(t, dtype)) HOT_FAIL(HOT_ERR_UNSUPPORTED, "quant_tiles: job %d is not covered", i);
    const Geometry g = geometry_of(t);
    DevJob& d = dev.job[i];
    d.x = t.x;
    d.ldx = t.ldx;
    d.L = (int)t.rows;
    d.C = (int)t.channels;
    d.batch = (int)t.batch;
    d.cblocks = g.cblocks;
    d.tt = g.tt;
    d.tiles = g.tiles;
    d.ts = g.ts;
    d.stiles = g.stiles;
    d.by_cblocks = fast_div(g.cblocks);
    d.by_tiles = fast_div(g.tiles);
    d.by_stiles = fast_div(g.stiles);
    if (i == 1) {
      if (t.row || t.sum || t.batch != 1 || t.sample_pitch || g.col_mode != kColAll)
        HOT_FAIL(HOT_ERR_UNSUPPORTED, "quant_tiles: the second job is a weight (columns only, every row kept, one sample)");
      dev.first = quant_ctas;
      dev.sfirst = stats_ctas;
      if (!third) {
        dev.third = quant_ctas;
        dev.sthird = stats_ctas;
      }
    } else if (i == 2) {
      if (!tile_jobs_alike(jobs[0], t)) HOT_FAIL(HOT_ERR_UNSUPPORTED, "quant_tiles: the third job is unlike the first");
      dev.third = quant_ctas;
      dev.sthird = stats_ctas;
    }
    stats_ctas += (int)(t.batch * g.cblocks * g.stiles);
    quant_ctas += (int)(t.batch * g.cblocks * g.tiles);
    d.row_on = t.row;
    if (t.row) {
      d.n_row = t.order_row;
      d.row_philox = t.q_row.rounding == HOT_ROUND_STOCH_PHILOX;
      d.row_store = t.q_row.storage == HOT_STORE_INT4 ? kRowPacked4 : (t.times16 ? kRowTimes16 : kRowBytes8);
      d.qr = make_quant_dev(t.q_row);
      d.q_row = (uint8_t*)t.codes_row;
      d.ld_row = t.ld_row;
      d.s_row = t.scale_row;
    }
    d.col_mode = g.col_mode;
    d.scale_mode = HOT_SCALE_TENSOR;
    if (t.col) {
      d.n_col = t.order_col;
      d.col_philox = t.q_col.rounding == HOT_ROUND_STOCH_PHILOX;
      d.scale_mode = t.q_col.scale_mode;
      d.plain_stats = t.order_col == 1 && t.q_col.scale_mode == HOT_SCALE_TENSOR;
      d.group_pos = g.group_pos;
      for (int r = 0; r < 16; ++r) d.slot[r] = -1;
      if (g.col_mode == kColKept)
        for (int blk = 0; blk < 16 / t.order_col; ++blk)
          for (int s = 0; s < t.rank; ++s) {
            const int natural = t.sel ? t.sel[s] : s;
            if (natural < 0 || natural >= t.order_col || d.slot[blk * t.order_col + natural] >= 0)
              HOT_FAIL(HOT_ERR_ARG, "quant_tiles: kept row %d = %d out of range or repeated", s, natural);
            d.slot[blk * t.order_col + natural] = (signed char)(blk * t.rank + s);
          }
      d.qc = make_quant_dev(t.q_col);
      d.q_col = (uint8_t*)t.codes_col;
      d.ld_col = t.ld_col;
      d.sample_pitch = t.sample_pitch;
      d.out_len = (int)(t.rows / t.order_col * t.rank);
      d.row_codes = t.sample_pitch ? t.sample_pitch * t.batch : d.out_len;
      d.s_col = t.scale_col;
      const size_t need = g.col_mode == kColKept ? (size_t)g.tile_pos * kCh * sizeof(float) : 0;
      if (need > smem) smem = need;
    }
    if (i == 2) place_partials(t, g, (uint8_t*)third_scratch, &d);
    else at += place_partials(t, g, at, &d);
    d.sum_out = t.sum;
    if (t.sum && t.batch * g.stiles > kManyPartials) dev.sums = (int)((t.channels + kSumCh - 1) / kSumCh);
  }
  quant_ctas += dev.sums;
  if (dtype == HOT_F32) return launch_tiles_f32(&dev, stats_ctas, quant_ctas, smem, st);
  return launch_typed<__nv_bfloat16>(dev, stats_ctas, quant_ctas, smem, st);
}
#endif  // HOT_TILES_F32

}  // namespace hot
