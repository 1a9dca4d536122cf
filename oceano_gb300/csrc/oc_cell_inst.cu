// Instantiations of the four-lanes-per-cell stage kernel for one degree and one cell
// Gauss rule (compiled once per (degree, rule), like oc_stage_inst.cu).
#include "oc_cell.cuh"

#ifndef OC_DEGREE
#error "OC_DEGREE must be defined"
#endif
#ifndef OC_CELL_RULE
#define OC_CELL_RULE 0
#endif
#define OC_CAT2(a, b) a##b
#define OC_CAT(a, b) OC_CAT2(a, b)
#if OC_CELL_RULE == 1
#define OC_NAME(base) OC_CAT(OC_CAT(base, OC_DEGREE), _r1)
#else
#define OC_NAME(base) OC_CAT(base, OC_DEGREE)
#endif

namespace oc {

template <int LPC>
static constexpr int block_bytes() {
  return CellDims<OC_DEGREE, OC_CELL_RULE, LPC>::warp_bytes * kCellWarps;
}

template <typename RIN, bool CONF, int LPC>
static cudaError_t configure_one() {
  return cudaFuncSetAttribute(cell_kernel<OC_DEGREE, RIN, OC_CELL_RULE, CONF, LPC>,
                              cudaFuncAttributeMaxDynamicSharedMemorySize, block_bytes<LPC>());
}

template <int LPC>
static cudaError_t configure_lanes() {
  cudaError_t e = configure_one<float, false, LPC>();
  if (e == cudaSuccess) e = configure_one<double, false, LPC>();
  if (e == cudaSuccess) e = configure_one<float, true, LPC>();
  if (e == cudaSuccess) e = configure_one<double, true, LPC>();
  return e;
}

cudaError_t OC_NAME(configure_cell_p)() {
  cudaError_t e = configure_lanes<4>();
#if OC_DEGREE == 1
  if (e == cudaSuccess) e = configure_lanes<2>();
#elif OC_DEGREE == 4
  if (e == cudaSuccess) e = configure_lanes<8>();
#endif
  return e;
}

template <typename RIN, bool CONF, int LPC>
static cudaError_t launch_one(const StageArgs &a, int grid, cudaStream_t st) {
  return launch_programmatic(cell_kernel<OC_DEGREE, RIN, OC_CELL_RULE, CONF, LPC>, grid,
                             32 * kCellWarps, block_bytes<LPC>(), st, a);
}

template <int LPC>
static cudaError_t launch_lanes(const StageArgs &a, bool conforming, int grid, cudaStream_t st) {
  if (conforming)
    return a.r_is_float ? launch_one<float, true, LPC>(a, grid, st)
                        : launch_one<double, true, LPC>(a, grid, st);
  return a.r_is_float ? launch_one<float, false, LPC>(a, grid, st)
                      : launch_one<double, false, LPC>(a, grid, st);
}

// conforming: every cell of this degree, no hanging face, standard orientation; lanes: of a
// cell, 4, or 2 (degree 1) or 8 (degree 4)
cudaError_t OC_NAME(launch_cell_p)(const StageArgs &a, bool conforming, int lanes, int grid,
                                   cudaStream_t st) {
  if (lanes == 4) return launch_lanes<4>(a, conforming, grid, st);
#if OC_DEGREE == 1
  if (lanes == 2) return launch_lanes<2>(a, conforming, grid, st);
#elif OC_DEGREE == 4
  if (lanes == 8) return launch_lanes<8>(a, conforming, grid, st);
#endif
  return cudaErrorInvalidValue;
}

cudaError_t OC_NAME(upload_cell_tables_p)(const DegTables<double> *td,
                                          const DegTables<float> *tf) {
  cudaError_t e = cudaMemcpyToSymbol(c_tabd, td, sizeof(DegTables<double>) * OC_MAXDEG);
  if (e != cudaSuccess) return e;
  return cudaMemcpyToSymbol(c_tabf, tf, sizeof(DegTables<float>) * OC_MAXDEG);
}

}  // namespace oc
