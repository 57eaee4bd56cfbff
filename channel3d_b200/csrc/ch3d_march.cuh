// ch3d_march.cuh -- the row tables of the kernels that fuse the right-hand sides
// with the y Crank-Nicolson solves (ch3d_march.cu; filled by ch3d_substep.cu).
#pragma once
#include "ch3d_dev.cuh"

namespace ch3d {

// Row table (precision T, MT_W values per row j = 0..ny-1): the y metrics at
// jc = j + 1 and the Thomas factors a, 1/m, c/m of the two Helmholtz sets (set
// 0: ux and uz, set 1: uy; m_TSchemePIMP_inc.f90:392-430, 542-589, 702-740).
// cp of the last row is stored as 0 (it has no upper neighbour).
enum {
  MT_IY1, MT_IY3, MT_RDYP, MT_RDYC, MT_AP2C, MT_AC2C, MT_AM2C, MT_AP2P, MT_AC2P, MT_AM2P,
  MT_A0, MT_RM0, MT_CP0, MT_A1, MT_RM1, MT_CP1, MT_W
};
// Second table for the twisted march (lower half eliminated upwards, upper half
// downwards): the downward factors c, 1/m', a/m' of both sets, with
// m'_{ny-1} = b, m'_j = b_j - c_j aq_{j+1}; rows of MD_W values.
enum { MD_C0, MD_RQ0, MD_AQ0, MD_C1, MD_RQ1, MD_AQ1, MD_W = 8 };

// Layout of the table buffer (values of precision T at the start of a buffer
// sized for FP64): the row tables of the RK substeps ns = 1..3 (ny * MT_W values
// each), their downward tables (ny * MD_W each), then per substep the pmBeta its
// factors were computed for (FP64 bit patterns; all ones = not yet computed).
constexpr int kMarchTables = 3;
inline unsigned long long* march_beta_slots(void* mtab, int ny) {
  return (unsigned long long*)((char*)mtab + (size_t)kMarchTables * ny * (MT_W + MD_W) * sizeof(double));
}
template <class T> inline T* march_down_tables(void* mtab, int ny) { return (T*)mtab + (size_t)kMarchTables * ny * MT_W; }

}  // namespace ch3d
