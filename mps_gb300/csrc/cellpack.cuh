// A grid cell's coordinates in one 32-bit word (the split V-cycle's tables, solver.cu):
// 16 bits each, so grids of up to 65,536 cells per axis.  Callers keep plain cell
// indices where a grid is wider (packs() false): an index costs a division when read,
// which every cell of the cycle's chain of phases would wait for.
#pragma once

#include <cstdint>

#ifdef __CUDACC__
#define MPS_CELL_FN __host__ __device__ __forceinline__
#else
#define MPS_CELL_FN inline
#endif

namespace mpsg {

MPS_CELL_FN bool packs(int nx, int ny) { return nx <= 65536 && ny <= 65536; }
MPS_CELL_FN uint32_t pack_cell(int x, int y) { return (uint32_t)x << 16 | (uint32_t)y; }
MPS_CELL_FN int cell_x(uint32_t c) { return (int)(c >> 16); }
MPS_CELL_FN int cell_y(uint32_t c) { return (int)(c & 0xffffu); }

}  // namespace mpsg
