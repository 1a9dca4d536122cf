// One-launch stage over every degree group of an hp mesh with four lanes per cell
// (compiled once per stage-input type: OC_CELL_HP_FP64 1 for stage 0).  The grid is the
// concatenation of the groups' block ranges, as in stage_kernel_hp.
#include "oc_cell.cuh"

#define OC_CAT2(a, b) a##b
#define OC_CAT(a, b) OC_CAT2(a, b)
#ifndef OC_CELL_HP_FP64
#error "OC_CELL_HP_FP64 must be defined"
#endif

namespace oc {

#if OC_CELL_HP_FP64
using CellHpIn = double;
#else
using CellHpIn = float;
#endif

// resident blocks per SM (register cap of the degree-4 body)
#ifndef OC_CELL_HP_BLOCKS
#define OC_CELL_HP_BLOCKS 8
#endif
template <typename RIN>
__global__ void __launch_bounds__(32 * kCellWarps, OC_CELL_HP_BLOCKS) cell_kernel_hp(const StageArgs a) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int b = blockIdx.x;
#define OC_HP_CASE(P)                                                                          \
  if (b >= a.hp_first_block[P] && b < a.hp_first_block[P] + a.hp_blocks[P]) {                 \
    cell_body<P, RIN, 0, false, 4>(a, smem_raw, b - a.hp_first_block[P], a.hp_n[P],              \
                                a.hp_cells[P], 0);                                            \
    return;                                                                                    \
  }
  OC_HP_CASE(4)
  OC_HP_CASE(3)
  OC_HP_CASE(2)
  OC_HP_CASE(1)
#undef OC_HP_CASE
}

static constexpr int kBlockBytes = CellDims<4, 0, 4>::warp_bytes * kCellWarps;  // the largest of the degrees
static_assert(CellDims<1, 0, 4>::warp_bytes * kCellWarps <= kBlockBytes &&
                  CellDims<2, 0, 4>::warp_bytes * kCellWarps <= kBlockBytes &&
                  CellDims<3, 0, 4>::warp_bytes * kCellWarps <= kBlockBytes,
              "a block holds the cells of any degree");

cudaError_t OC_CAT(configure_cell_hp_v, OC_CELL_HP_FP64)() {
  return cudaFuncSetAttribute(cell_kernel_hp<CellHpIn>,
                              cudaFuncAttributeMaxDynamicSharedMemorySize,
                              kBlockBytes);
}

cudaError_t OC_CAT(launch_cell_hp_v, OC_CELL_HP_FP64)(const StageArgs &a, int grid,
                                                      cudaStream_t st) {
  return launch_programmatic(cell_kernel_hp<CellHpIn>, grid, 32 * kCellWarps, kBlockBytes, st, a);
}

cudaError_t OC_CAT(upload_cell_tables_hp_v, OC_CELL_HP_FP64)(const DegTables<double> *td,
                                                             const DegTables<float> *tf) {
  cudaError_t e = cudaMemcpyToSymbol(c_tabd, td, sizeof(DegTables<double>) * OC_MAXDEG);
  if (e != cudaSuccess) return e;
  return cudaMemcpyToSymbol(c_tabf, tf, sizeof(DegTables<float>) * OC_MAXDEG);
}

}  // namespace oc
