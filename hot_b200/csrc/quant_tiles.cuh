// Host interface of the tiled quantisers (quant_tiles.cu): what a job is, whether it is covered, and the pair of launches.
#pragma once

#include "ht_device.cuh"

namespace hot {

constexpr int kMaxTileJobs = 2;

struct TileJob {
  const void* x = nullptr;  // [batch, rows, channels], pitch ldx elements
  int64_t ldx = 0, batch = 1, rows = 0, channels = 0;
  // row side: codes like x at pitch ld_row bytes, one scale per sample
  bool row = false;
  int order_row = 1;
  hot_quant_t q_row = {};
  bool times16 = false;     // 4-bit Philox codes one per byte, stored as 16 * code with the scale / 16
  void* codes_row = nullptr;
  int64_t ld_row = 0;
  float* scale_row = nullptr;
  // column side: codes [channels, ...] one per byte at pitch ld_col bytes, sample b at byte b * sample_pitch (0: one sample)
  bool col = false;
  int order_col = 1, rank = 1;
  const int32_t* sel = nullptr;  // kept natural rows; null: all of them in order
  hot_quant_t q_col = {};
  void* codes_col = nullptr;
  int64_t ld_col = 0, sample_pitch = 0;
  float* scale_col = nullptr;
  // sum over all rows of all samples, in the type of x
  void* sum = nullptr;
};

bool tile_job_covered(const TileJob& job, int dtype);
size_t tile_scratch_bytes(const TileJob* jobs, int count);
// One pair of launches: jobs[0], and with count 2 a weight (columns only, every row kept, one sample).  third: one more job
// that is like jobs[0] (tile_jobs_alike), with scratch of its own (tile_scratch_bytes(third, 1)).
bool tile_jobs_alike(const TileJob& a, const TileJob& b);
int launch_tile_jobs(const TileJob* jobs, int count, int dtype, void* scratch, size_t scratch_bytes, cudaStream_t st,
                     const TileJob* third = nullptr, void* third_scratch = nullptr);

}  // namespace hot
