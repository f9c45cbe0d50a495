// The float32 instances of the tiled quantisers (see the end of quant_tiles.cu).
#define HOT_TILES_F32
#include "quant_tiles.cu"
