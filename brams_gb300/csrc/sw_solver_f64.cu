// The fp64 instantiation of the RRTMG_SW column kernel (sw_kernel.cuh), with
// fused multiply-adds: GB300 issues two fp64 lanes a clock and SM, and the
// kernel is bound by that pipe.  Its table directory is this unit's own copy.
#include "sw_kernel.cuh"

cudaError_t gb_sw_set_tab_f64(const void* tab) { return gbsw::sw_set_tab(*static_cast<const gbsw::SwTab*>(tab)); }

size_t gb_sw_scratch_f64(int nlay, long long slots, long long ncol) {
  return gbsw::sw_scratch_bytes_t<double>(nlay, slots, ncol);
}

cudaError_t gb_sw_launch_f64(const SwArgs& a, const double* d_tables, void* scratch, size_t bytes, long long slots,
                             cudaStream_t stream) {
  return gbsw::sw_launch_t<double, SW_MINB_F64>(a, d_tables, scratch, bytes, slots, stream);
}
