// The quantised index of rtrnmc's exponential table (rrtmg_lw_rtrnmc.f90:385-388).
#pragma once

namespace gb {

constexpr float BPADE = 1.0f / 0.278f;

// od / (bpade + od) by PTX's approximate division: within 2 ulp for divisors
// up to 2^126; beyond, 0 for a finite od and not a number for an infinite one
// (index 0 both)
__device__ __forceinline__ float tbl_quotient(float od) {
  float r;
  asm("div.approx.ftz.f32 %0, %1, %2;" : "=f"(r) : "f"(od), "f"(BPADE + od));
  return r;
}
// rtrnmc's table index of an optical depth (rrtmg_lw_rtrnmc.f90:385-388):
// itr = int(tblint * od / (bpade + od) + 0.5), within 0 .. ntbl (od >= 0, and
// a quotient that is not a number converts to 0)
__device__ __forceinline__ int tbl_index(float od) {
  const float tblind = __fdividef(od, BPADE + od);
  const int itr = (int)fmaf(10000.0f, tblind, 0.5f);
  return itr < 0 ? 0 : (itr > 10000 ? 10000 : itr);
}
// tau_tbl at an index formed in registers, bpade * t / (1 - t) at t = itr /
// 10000 (1e10 at the last entry; rrtmg_lw_init.f90:120-142), instead of a
// table load that depends on the clear cell's lookup (fp32 arithmetic: within
// a few units in the last place of the fp64-built table's float)
__device__ __forceinline__ float tbl_tau(int itr) {
  const float t = (float)itr * 1.0e-4f;
  return itr >= 10000 ? 1.0e10f : BPADE * t / (1.0f - t);
}

}  // namespace gb
