// Launch interface of the RRTMG_LW column kernels (lw_solver.cu).
#pragma once
#include <cuda_fp16.h>
#include <cuda_runtime.h>
#include <stddef.h>

#include "lw_common.h"

// Where a grid's McICA sub-column clouds come from.
enum LwCloudMode {
  LW_CLOUD_SUBCOL = 0,  // caller-supplied (140, ld, nlay) arrays cldfmcl/ciwpmcl/clwpmcl/taucmcl
  LW_CLOUD_FUSED = 1,   // generated from layer clouds (icld 3, Mersenne twister,
                        // column c seeded with seed0 + c), as mcica_subcol_lw would for one column
  LW_CLOUD_BAND = 2,    // the non-McICA driver's band-level clouds (rrtmg_lw_rad.nomcica.f90):
                        // layer fractions cldfrac (ld, nlay), cldprop's optical depths tauc
                        // (16, ld, nlay) and its cloud-band count ncbands (ld); icld 1 random
                        // overlap (rtrn), 2 and 3 maximum/random overlap (rtrnmr)
};

// Device pointers in the reference's Fortran layout.  (ncol, .) arrays have
// leading dimension ld (>= ncol); McICA arrays are (140, ld, nlay); tauaer is
// (ld, nlay, 16); outputs (ldo, nlay+1) / (ldo, nlay).  In LW_CLOUD_FUSED mode
// cldfrac/ciwp/clwp are (ld, nlay), tauc is (16, ld, nlay) and reicmcl/relqmcl
// hold the layer radii rei/rel.
struct LwArgs {
  int ncol, nlay;
  long long ld, ldo;
  int icld, idrv, inflag, iceflag, liqflag;
  int cloud_mode;
  unsigned seed0;
  const double *play, *plev, *tlay, *tlev, *tsfc;
  const double *h2ovmr, *o3vmr, *co2vmr, *ch4vmr, *n2ovmr, *o2vmr;
  const double *cfc11vmr, *cfc12vmr, *cfc22vmr, *ccl4vmr, *emis;
  const double *cldfmcl, *taucmcl, *ciwpmcl, *clwpmcl, *reicmcl, *relqmcl, *tauaer;
  const double *cldfrac, *ciwp, *clwp, *tauc;
  double *uflx, *dflx, *hr, *uflxc, *dflxc, *hrc, *duflx_dt, *duflxc_dt;
  int* col_err;   // optional per-column status (ncol)
  int* err_flag;  // required: max status over the launch
  // optional learned gas optics: taug and Planck fractions per (column, layer, g)
  // in fp16 and a per-layer flag (1: use them, 0: taumol); NULL: taumol everywhere
  const __half *sur_tau, *sur_frac;
  const unsigned char* sur_flag;
  // fused cloud mode: the columns' 140 McICA draws [ncol][140] (gb_mcica_percol_mt);
  // required when cloud_mode is LW_CLOUD_FUSED and icld >= 1
  const double* draws;
  // band cloud mode: cldprop's cloud-band count per column (1, 5 or 16)
  const int* ncbands;
};

// Grids of one launch: grid i owns batch columns col0[i] .. col0[i+1]-1.  The
// kernels take this by value (kernel parameter space), so a launch carries
// no device-side descriptor and can be captured in a CUDA graph as is.
#define GB_LW_MAX_GRIDS 32
//
// Gas optics hand-over.  A batch is solved in units of cpb neighbouring
// columns of one grid; unit0[i] is grid i's first unit (a grid of an odd
// number of columns leaves a column of its last unit empty).  For the units
// [u0, u1) of one pass, taumol (gb_lw_launch_taumol) fills a plane per column
// slot, slot (u - u0) * cpb + c:
//   plane + (slot * nsmax + layer) * GB_LW_PROW   the layer's row: per pair of
//     neighbouring g-points of a band (tau, tau, fraction, fraction) as fp32
//     (taug without aerosol, Planck fractions), bands on 32-byte boundaries
//     (gb_pair0), so that the transfer reads a pair in one 16-byte load.
// coef and laytrop hold setcoef's words between taumol's two kernels.  A pass
// takes as many units as the planes have room for.
//
// Batches with learned gas optics (fall and nfall set) run in two launches:
// the transfer kernel solves every column whose layers are all on the network
// and hands the others (batch numbering) over in fall[0 .. *nfall), then the
// hand-over kernel runs taumol and the transfer for those in its blocks (block
// k in plane slot k), mixing per layer the network's values and taumol's.
// fall holds at least col0[ngrid] entries.
//
// gtau and gfrac ([slot][layer][140] planes, gstride floats per slot) are the
// outputs of the taumol-only launch (training samples, diagnostics).
constexpr int GB_LW_PROW = 304;        // floats per plane row: 76 pair positions
constexpr int GB_LW_CELL_WORDS = 10;   // cell bits of a layer (140 cloudy, 140 fractional, in groups of 32)
constexpr int GB_LW_COEF_WORDS = 26;   // setcoef words per column and layer
// first pair position of band b (1..16) in a plane row
__host__ __device__ constexpr int gb_pair0(int b) {
  constexpr int m[17] = {0, 0, 6, 12, 20, 28, 36, 40, 46, 50, 56, 60, 64, 68, 70, 72, 74};
  return m[b];
}
struct LwBatch {
  int ngrid;
  int nsmax;                              // largest nlay (stride of the shared-memory areas)
  long long col0[GB_LW_MAX_GRIDS + 1];
  int cpb = 1;                            // columns per unit (see above)
  long long unit0[GB_LW_MAX_GRIDS + 1];
  float* plane = nullptr;                 // gas-optics planes
  float* coef = nullptr;                  // setcoef's words
  int* laytrop = nullptr;                 // per slot
  long long pslots = 0;                   // plane slots available (a multiple of 32)
  float* gcld = nullptr;                  // caller sub-columns: each cloudy cell's optical depth (or
                                          // fractional cldfmcl), [nsmax][140] per slot (learned gas
                                          // optics: per resident column)
  unsigned* cellw = nullptr;              // and per slot and layer the cells' bits: GB_LW_CELL_WORDS words
  int* cellerr = nullptr;                 // and the columns' stop codes
  float* part = nullptr;                  // level sums per resident column
  long long rcols = 0;                    // resident columns there is room for
  float* gtau = nullptr;                  // taumol-only launch (see above)
  float* gfrac = nullptr;
  long long gstride = 0;                  // floats per slot (>= nsmax * 140)
  long long gslots = 0;                   // slots available
  long long* fall = nullptr;              // columns handed over off the network
  unsigned* nfall = nullptr;              // their count (device)
  LwArgs g[GB_LW_MAX_GRIDS];
};

// Compiled shapes of the transfer kernel: threads per column block (a unit of
// two columns, a pair of g-points per thread) and the most of them on an SM
// that the register allocation is sized for.
struct LwVariant {
  int threads, min_blocks;
};
// The learned-gas-optics transfer kernel (lean = true) has its own table of as many shapes.
int gb_lw_num_variants();
LwVariant gb_lw_variant(int v, bool lean = false);

// the variant sized for the units (column blocks) that fit on an SM at this nlay
int gb_lw_default_variant(int nlay);

// the most shared memory a block needs at this nlay at least (a unit of one
// column beside rtrnmc's table, or the hand-over kernel's taumol area); a
// launch is possible iff this fits in one block
size_t gb_lw_smem_bytes(int nlay);
// column blocks of `variant` resident on the device at once for this nlay
int gb_lw_slots(int nlay, int variant = 0, bool lean = false);
// bytes of the hand-over buffer a batch (its grids set) is solved with
// (learned: only the hand-over kernel's planes), and the least it runs with
size_t gb_lw_gas_bytes(const LwBatch& b, bool learned);
size_t gb_lw_gas_min_bytes(int nlay);
// points a descriptor at a hand-over buffer of `bytes`
void gb_lw_attach_gas(LwBatch& b, void* buf, size_t bytes);
// column blocks of the hand-over kernel of a learned batch
long long gb_lw_list_slots();
cudaError_t gb_lw_set_tables(const GbTables& T);
// All grids of `b` with `variant` at `nblocks` persistent blocks: taumol
// batches through taumol's kernels and the transfer kernel, pass by pass; with
// b.fall set the learned-gas-optics transfer kernel, then the hand-over
// kernel.  Batches of LW_CLOUD_BAND grids (all grids in that mode, taumol
// only) run the band-cloud flavour of the transfer kernel.
cudaError_t gb_lw_launch_batch(const LwBatch& b, const float* d_tables, int variant, int nblocks,
                               cudaStream_t stream);
// The taumol kernel alone over batch columns [c0, c1) into slots 0 .. c1-c0-1.
cudaError_t gb_lw_launch_gas(const LwBatch& b, const float* d_tables, long long c0, long long c1,
                             cudaStream_t stream);
// taumol of units [u0, u1) into plane slots 0 .. (lw_taumol.cu).
cudaError_t gb_lw_launch_taumol(const LwBatch& b, const float* d_tables, long long u0, long long u1,
                                cudaStream_t stream);
cudaError_t gb_lw_taumol_set_tables(const GbTables& T);
