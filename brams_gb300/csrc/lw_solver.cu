// RRTMG_LW column kernels for GB300 (sm_103a).
//
// The reference solves one column at a time (rrtmg_lw_rad.f90:486-593):
// inatm, cldprmc, setcoef, taumol, the aerosol add and rtrnmc.  Here a unit of
// 160 threads solves two neighbouring columns, 80 threads a column, each
// standing for a pair of g-points of one band (70 live); an SM holds up to four units, which
// walk the columns of a batch of grids.  Nothing per cell goes to global scratch
// but the planes between the kernels:
//
//   taumol -- of a batch, by kernels of its own (lw_taumol.cu), into a plane
//     per column that the transfer reads; the batch goes through in passes of
//     as many columns as the planes hold.  It was part of the column's block
//     before (setcoef by 45 of 160 threads, two barriers per band, a shared-
//     memory read and a 4-byte gather per multiply-add) and took 42% of its
//     time: 24.1 ms for 108,000 columns of 45 layers with caller sub-columns,
//     17.0 ms since, and 17.9 to 8.3 ms for 67,909 columns with in-kernel
//     clouds.  The in-block form (gas_column) is still the way where a block
//     finds its columns on the device only (lw_list_kernel), and for single
//     outputs per (layer, g-point) (lw_gas_kernel): setcoef
//     with one thread per layer, then band by band a prologue per layer builds
//     the layer's term list (lw_gasoptics.cuh) and one thread per (layer, g)
//     cell gathers taug = sum w * table[row + g].
//
//   transfer (rt_columns) -- inatm's column amounts, the laytrop and value
//     checks, Planck interpolation per (layer, band) and the surface source,
//     the McICA cloud bits and cldprmc's optical depths (caller sub-columns:
//     lw_cells_kernel), then rtrnmc: a
//     downward pass from the model top and an upward pass from the surface.
//     Each pass evaluates a cell's transmittance and sources in registers from
//     taug, the Planck fraction, the layer's Planck values and rtrnmc's
//     exp_tbl/tfn_tbl (rrtmg_lw_init.f90:120-142, built in double
//     precision at set-up, held in shared memory) at the reference's quantised index
//     (rtrnmc.f90:350-455 down, 486-529 up); the up pass recomputes what the
//     down pass computed instead of storing it.  The sums over the g-points
//     of a level go by transposed butterflies over a group of 32 g-points (two
//     streams down, four up); the five groups' fp32 partials
//     are added error-free (two-sum) into fp64, and the net fluxes and heating
//     rates heatfac*dF/dp are fp64 (rtrnmc.f90:566-592).
//
//     A thread had one g-point of one column before, with the table in L1:
//     66,000 warp instructions a column of 60 layers at 52% of the issue
//     slots, 28.8 ms for 262,144 columns.  Two g-points a thread share a layer's
//     records, loop and branches and half the sums (46,900 instructions); what
//     bounds it is those instructions, at 15 to 20 warps an SM, and the
//     latency of the set-up phases.  1.34 ms for 16,384 columns (1.80 before).
//
// Kernels: lw_rt_kernel (the transfer, on taumol's planes or on the network's
// fp16 taug and Planck fractions; there, columns with a layer off the network
// are handed over), lw_cells_kernel (caller sub-columns' cells), lw_list_kernel (taumol and the transfer of the columns
// handed over), lw_gas_kernel (taumol alone, for the network's training
// samples and the gas-optics diagnostics).
//
// Precision: gas optics and transfer in fp32, flux sums across warps
// error-free into fp64, net fluxes and the heating-rate step in fp64.
// Outputs follow the reference's layout: uflx(icol, k+1) for k = 0..nlay,
// hr(icol, k+1) for k = 0..nlay-1.  The unit is compiled without multiply-add
// contraction (every fused multiply-add is an explicit fmaf), so a column
// gives the same bits in every kernel flavour and launch shape.
#include <cuda_runtime.h>
#include <math.h>
#include <algorithm>
#include <cmath>
#include <stdint.h>
#include <climits>
#include <cstddef>

#include "lw_common.h"
#include "lw_solver.h"
#include "lw_gasoptics.cuh"
#include "lw_table.cuh"

namespace gb {

constexpr float REC_6 = 0.166667f;
constexpr int TGROUP = MAXT_ALL;  // term slots per layer of a band's term list
constexpr int RT_NT = 160;        // threads per block of two columns; virtual threads per column in the
                                  // phases whose order of operations goes by thread
constexpr int RT_CT = 80;         // threads per column in the passes: one per pair of g-points
constexpr int RT_NW = RT_NT / 32; // groups of 32 g-points of a column
constexpr int LIST_PER_SM = 2;    // hand-over kernel blocks per SM

__constant__ int c_icb[16] = {1, 2, 3, 3, 3, 4, 4, 4, 5, 5, 5, 5, 5, 5, 5, 5};  // cldprmc.f90:133
// diffusivity-angle coefficients (rtrnmc.f90:236-247)
__constant__ float c_a0[16] = {1.66f, 1.55f, 1.58f, 1.66f, 1.54f, 1.454f, 1.89f, 1.33f, 1.668f, 1.66f, 1.66f, 1.66f, 1.66f, 1.66f, 1.66f, 1.66f};
__constant__ float c_a1[16] = {0.f, 0.25f, 0.22f, 0.f, 0.13f, 0.446f, -0.10f, 0.40f, -0.006f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
__constant__ float c_a2[16] = {0.f, -12.0f, -11.7f, 0.f, -0.72f, -0.243f, 0.19f, -0.062f, 0.414f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};

__host__ __device__ inline size_t align16(size_t x) { return (x + 15) & ~size_t(15); }

// ------------------------------------------------------------------ helpers
// ---- two g-points per thread: packed fp32 arithmetic.  Each half rounds as the
// scalar operation does, but for a packed product whose one use is a packed sum:
// the assembler makes one multiply-add of these (probed: 13,616 of 65,536 sums
// differ), whatever -fmad says.  So no product goes into a sum directly here: the
// weighted radiances of sum4 and sum8 go through a select or a shuffle, sum2 adds
// the halves of one product (both probed: not fused), the surface's is scalar.
typedef unsigned long long u64;
__device__ __forceinline__ u64 pk(float2 v) {
  u64 r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(v.x), "f"(v.y));
  return r;
}
__device__ __forceinline__ float2 upk(u64 v) {
  float2 r;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(v));
  return r;
}
__device__ __forceinline__ float2 fma2(float2 a, float2 b, float2 c) {
  u64 r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(pk(a)), "l"(pk(b)), "l"(pk(c)));
  return upk(r);
}
__device__ __forceinline__ float2 mul2(float2 a, float2 b) {
  u64 r;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(pk(a)), "l"(pk(b)));
  return upk(r);
}
__device__ __forceinline__ float2 add2(float2 a, float2 b) {
  u64 r;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(pk(a)), "l"(pk(b)));
  return upk(r);
}
__device__ __forceinline__ float2 both(float v) { return make_float2(v, v); }
__device__ __forceinline__ float2 sel2(bool c, float2 a, float2 b) { return c ? a : b; }
__device__ __forceinline__ float2 shfl2(float2 v, int m) {
  return make_float2(__shfl_xor_sync(0xffffffffu, v.x, m), __shfl_xor_sync(0xffffffffu, v.y, m));
}

// Sums over the 32 g-points of a group: 16 lanes, lane l holding g-points 2l
// and 2l + 1 of the group in the halves of a value.  Transposed butterflies;
// the order of the additions (over bits of the g-point's number in the group)
// is part of the result: sum2 adds over bits 0, 1, 2, 3, 4; sum4 over 1, 0, 2,
// 3, 4; sum8 over 2, 1, 0, 3, 4 -- the orders of a butterfly with one g-point
// per lane, which is what the fluxes' last bits were before.
// sum2: lane l returns the sum of v[l & 1]
__device__ __forceinline__ float sum2(float2 v0, float2 v1, int l) {
  const float k0 = v0.x + v0.y, k1 = v1.x + v1.y;
  const bool h = l & 1;
  float k = h ? k1 : k0;
  k += __shfl_xor_sync(0xffffffffu, h ? k0 : k1, 1);
  k += __shfl_xor_sync(0xffffffffu, k, 2);
  k += __shfl_xor_sync(0xffffffffu, k, 4);
  k += __shfl_xor_sync(0xffffffffu, k, 8);
  return k;
}
// sum4: lane l returns the sum of v[sum4_at(l)]
__device__ __forceinline__ int sum4_at(int l) { return 2 * (l & 1) + ((l >> 1) & 1); }
__device__ __forceinline__ float sum4(float2 v0, float2 v1, float2 v2, float2 v3, int l) {
  const bool h = l & 1;
  const float2 a0 = add2(sel2(h, v2, v0), shfl2(sel2(h, v0, v2), 1));
  const float2 a1 = add2(sel2(h, v3, v1), shfl2(sel2(h, v1, v3), 1));
  const float k0 = a0.x + a0.y, k1 = a1.x + a1.y;
  const bool g = l & 2;
  float k = g ? k1 : k0;
  k += __shfl_xor_sync(0xffffffffu, g ? k0 : k1, 2);
  k += __shfl_xor_sync(0xffffffffu, k, 4);
  k += __shfl_xor_sync(0xffffffffu, k, 8);
  return k;
}
// sum8: lane l returns the sum of v[sum8_at(l)]
__device__ __forceinline__ int sum8_at(int l) { return 4 * ((l >> 1) & 1) + 2 * (l & 1) + ((l >> 2) & 1); }
__device__ __forceinline__ float sum8(float2 v0, float2 v1, float2 v2, float2 v3, float2 v4, float2 v5, float2 v6,
                                      float2 v7, int l) {
  const bool h = l & 2;
  const float2 a0 = add2(sel2(h, v4, v0), shfl2(sel2(h, v0, v4), 2));
  const float2 a1 = add2(sel2(h, v5, v1), shfl2(sel2(h, v1, v5), 2));
  const float2 a2 = add2(sel2(h, v6, v2), shfl2(sel2(h, v2, v6), 2));
  const float2 a3 = add2(sel2(h, v7, v3), shfl2(sel2(h, v3, v7), 2));
  const bool g = l & 1;
  const float2 c0 = add2(sel2(g, a2, a0), shfl2(sel2(g, a0, a2), 1));
  const float2 c1 = add2(sel2(g, a3, a1), shfl2(sel2(g, a1, a3), 1));
  const float k0 = c0.x + c0.y, k1 = c1.x + c1.y;
  const bool f = l & 4;
  float k = f ? k1 : k0;
  k += __shfl_xor_sync(0xffffffffu, f ? k0 : k1, 4);
  k += __shfl_xor_sync(0xffffffffu, k, 8);
  return k;
}

// cldprmc's optical depth ciwp*abscoice + clwp*abscoliq of one cell
// (cldprmc.f90:194-266; the radius bounds are checked beforehand), from
// w = (ciwp, clwp, radice, radliq) converted to float and flags bit 0: ciwp
// /= 0, bit 1: clwp /= 0
__device__ __forceinline__ float cloud_tau_layer(const LwArgs& a, int band, const float* __restrict__ T, float4 w,
                                                 int flags) {
  float abscoice = 0.0f, abscoliq = 0.0f;
  if (flags & 1) {
    const float radice = w.z;
    if (a.iceflag == 0) {
      abscoice = T[c_T.absice0] + T[c_T.absice0 + 1] / radice;
    } else if (a.iceflag == 1) {
      int ib = c_icb[band];
      abscoice = T[c_T.absice1 + 2 * (ib - 1)] + T[c_T.absice1 + 1 + 2 * (ib - 1)] / radice;
    } else {
      float factor = (radice - 2.0f) / 3.0f;
      int nrow = a.iceflag == 2 ? 43 : 46;
      int index = clampi((int)factor, 1, nrow - 1);
      float fint = factor - (float)index;
      const float* t = T + (a.iceflag == 2 ? c_T.absice2 : c_T.absice3) + nrow * band;
      abscoice = t[index - 1] + fint * (t[index] - t[index - 1]);
    }
  }
  if (flags & 2) {
    if (a.liqflag == 0) {
      abscoliq = c_T.absliq0;
    } else {
      const float radliq = w.w;
      int index = clampi((int)(radliq - 1.5f), 1, 57);
      float fint = radliq - 1.5f - (float)index;
      const float* t = T + c_T.absliq1 + 58 * band;
      abscoliq = t[index - 1] + fint * (t[index] - t[index - 1]);
    }
  }
  return w.x * abscoice + w.y * abscoliq;
}

// ================================================================== taumol
struct GasSmem {
  float* f;        // [NF][nl]   per-layer setcoef quantities
  int* iv;         // [NI][nl]
  float2* terms;   // [TGROUP][nl] gas-optics terms of the current band, term-major
  FracRec* frec;   // [nl] Planck-fraction records of the current band
  int* iscal;      // [4]: laytrop
};

__host__ __device__ inline size_t gas_smem_bytes(int nl) {
  return align16((size_t)(NF + NI) * nl * 4) + align16((size_t)nl * TGROUP * 8) + align16((size_t)nl * sizeof(FracRec)) + 16;
}

__device__ inline GasSmem gas_carve(char* p, int nl) {
  GasSmem s;
  s.f = (float*)p;
  s.iv = (int*)(p + (size_t)NF * nl * 4);
  p += align16((size_t)(NF + NI) * nl * 4);
  s.terms = (float2*)p;
  p += align16((size_t)nl * TGROUP * 8);
  s.frec = (FracRec*)p;
  p += align16((size_t)nl * sizeof(FracRec));
  s.iscal = (int*)p;
  return s;
}

// Prologue of band b for one layer: the band-specific per-layer code
// (lw_gasoptics.cuh) writing the layer's terms and Planck-fraction record.
template <int b>
__device__ __forceinline__ void band_prologue(const GasSmem& s, int nl, int lay, bool lower, const float* T,
                                              const LwArgs& a, long long icol) {
  Cell c{s.f, s.iv, nl, lay, T, &a, icol};
  Terms t{s.terms + lay, nl, 0};
  FracRec r = Band<b>::prologue(c, lower, t);
  t.pad(maxt(b), c_T.band[b - 1].sr);
  s.frec[lay] = r;
}

// taumol of band b for every layer of a column: the prologue of each layer,
// then one thread per (layer, g) cell gathering taug = sum w * table[row + g]
// (the band's term count and g-points are compile-time constants, so the
// gather loop is unrolled) and interpolating the Planck fraction.  Ends with
// a barrier.
template <int b, int NT, class Out>
__device__ __forceinline__ void gas_band(const LwArgs& a, long long icol, const GasSmem& s, int nl, int laytrop,
                                         const float* __restrict__ T, const Out& out) {
  constexpr int NG = ngb_const(b), M = maxt(b);
  for (int lay = threadIdx.x; lay < nl; lay += NT) band_prologue<b>(s, nl, lay, lay < laytrop, T, a, icol);
  __syncthreads();
  for (int cell = threadIdx.x; cell < nl * NG; cell += NT) {
    const int lay = cell / NG, gi = cell - lay * NG;
    const float2* tp = s.terms + lay;
    const float* Tg = T + gi;
    float acc = 0.0f;
#pragma unroll
    for (int k = 0; k < M; ++k) {
      const float2 w = tp[k * nl];
      acc = fmaf(w.x, __ldg(Tg + __float_as_int(w.y)), acc);
    }
    if ((b == 4 || b == 7) && lay >= laytrop) acc *= gscale(b, gi);
    const FracRec fr = s.frec[lay];
    const float* fp = T + fr.off + gi;
    const float f0 = __ldg(fp);
    out.put(b, lay, gi, acc, fmaf(fr.fpl, __ldg(fp + pitch_const(b)) - f0, f0));
  }
  __syncthreads();
}

// taumol of one column by the whole block: taug and Planck fraction of every
// (layer, g) cell through out.put.  Ends with a barrier.
template <int NT, class Out>
__device__ void gas_column(const LwArgs& a, long long icol, const GasSmem& s, const Out& out,
                           const float* __restrict__ T) {
  const int nl = a.nlay, tid = threadIdx.x;
  if (tid == 0) s.iscal[0] = 0;
  __syncthreads();
  for (int lay = tid; lay < nl; lay += NT) {
    LayerInts ix;
    const bool lower = setcoef_layer(a, icol, lay, T, ix, [&](int k, float v) { s.f[k * nl + lay] = v; });
    int* IV = s.iv;
    IV[I_JP * nl + lay] = ix.jp; IV[I_JT * nl + lay] = ix.jt; IV[I_JT1 * nl + lay] = ix.jt1;
    IV[I_INDSELF * nl + lay] = ix.indself; IV[I_INDFOR * nl + lay] = ix.indfor; IV[I_INDMINOR * nl + lay] = ix.indminor;
    if (lower) atomicAdd(&s.iscal[0], 1);  // laytrop (the transfer checks that these form a prefix)
  }
  __syncthreads();
  const int laytrop = s.iscal[0];
  gas_band<1, NT>(a, icol, s, nl, laytrop, T, out);
  gas_band<2, NT>(a, icol, s, nl, laytrop, T, out);
  gas_band<3, NT>(a, icol, s, nl, laytrop, T, out);
  gas_band<4, NT>(a, icol, s, nl, laytrop, T, out);
  gas_band<5, NT>(a, icol, s, nl, laytrop, T, out);
  gas_band<6, NT>(a, icol, s, nl, laytrop, T, out);
  gas_band<7, NT>(a, icol, s, nl, laytrop, T, out);
  gas_band<8, NT>(a, icol, s, nl, laytrop, T, out);
  gas_band<9, NT>(a, icol, s, nl, laytrop, T, out);
  gas_band<10, NT>(a, icol, s, nl, laytrop, T, out);
  gas_band<11, NT>(a, icol, s, nl, laytrop, T, out);
  gas_band<12, NT>(a, icol, s, nl, laytrop, T, out);
  gas_band<13, NT>(a, icol, s, nl, laytrop, T, out);
  gas_band<14, NT>(a, icol, s, nl, laytrop, T, out);
  gas_band<15, NT>(a, icol, s, nl, laytrop, T, out);
  gas_band<16, NT>(a, icol, s, nl, laytrop, T, out);
}

// ================================================================== transfer
// Shared memory of one column: a fixed header, one 320-byte record per
// layer (so that every per-layer access in the loops is base + layer * 320
// + a constant), then band clouds' fractions.  The level sums are in global
// scratch (LwBatch::part).
constexpr int CELL_WORDS = GB_LW_CELL_WORDS;
struct RtHead {
  float misc[64];         // secdiff[16], plankbnd[16], dplankbnd[16], semiss[16]
  float red[2 * RT_NW];   // column sums for pwvcm of 32 layers each
  int iscal[4];           // stop code, lower-layer count, cloud-band count or off the network, check bits
  int pad[2];
};
struct RtLayer {
  float4 rec[16];     // per band: Planck value of the layer, that of the level above it, aerosol optical
                      // depth, cloud optical depth (fused clouds; band clouds: secdiff(ib) * taucloud
                      // per cloud band ib, rtrn's odcld).  The record before layer 0 has the
                      // Planck value of the lowest level.  In the first phase the fourth words of
                      // the record before a layer hold the Planck-table row and fraction of the
                      // level below it (words 0 and 1) and of the layer (2 and 3).
  int cldlay;         // 1: a cell of the layer has cldfmc == 1 (rtrnmc's icldlyr), or band
                      // clouds: cldfrac >= 1e-6; in the first phase: 1 where the layer is in
                      // the lower atmosphere
  int lfl;            // cloud flags of the layer (bits 0-2) and cldprmc's stop code (bits
                      // 8..); band clouds: istcld (bit 0) and istcldd (bit 1) of rtrnmr
  // McICA clouds use the words below as named; band clouds overlay them with
  // 14 floats (RtSmem::ovl): cldfrac, rtrnmr's upward overlap factors at lev+1
  // (facclr1, facclr2, faccld1, faccld2, faccmb1, faccmb2) and the downward
  // ones at lev-1, in that order
  unsigned cbits[CELL_WORDS];  // the first five: per group of 32 g-points: bit l set where g-point 2l of the group is cloudy
                      // (cldfmc == 1; caller sub-columns: or a fraction, in a layer with a cell
                      // of 1), bit 16 + l where g-point 2l + 1 is
                      // caller sub-columns: the next five (RtSmem::fbits), as these: cldfmcl neither 0 nor 1
                      // fused clouds: the McICA threshold 1 - cldf as double bits in words 6 and 7 (RtSmem::cthr)
  float4 lcw;         // (ciwp, clwp, radice, radliq) as floats
};
static_assert(sizeof(RtHead) == 320 && sizeof(RtLayer) == 320, "transfer shared-memory records");
static_assert(offsetof(RtLayer, lcw) + sizeof(float4) - offsetof(RtLayer, cbits) == 14 * sizeof(float) && offsetof(RtLayer, cbits) % 8 == 0,
              "band-cloud overlay of the McICA words");

struct RtSmem {
  RtHead* h;
  RtLayer* L;   // [-1 .. nl-1]; in the last phase: fp64 net fluxes [nl+1][2]
  double* cf;   // [nl] band clouds' fractions
  float* part;  // [RT_NW][nl+1][6] level sums per group of 32 g-points: dn, dn clear, up, up clear, dup/dT,
                // dup clear/dT (global scratch)
  __device__ __forceinline__ unsigned* fbits(int lay) const { return L[lay].cbits + 5; }
  __device__ __forceinline__ long long& cthr(int lay) const { return *reinterpret_cast<long long*>(L[lay].cbits + 6); }
  __device__ __forceinline__ float* ovl(int lay) const { return reinterpret_cast<float*>(L[lay].cbits); }
};

__host__ __device__ inline size_t rt_layers_bytes(int nl) {
  return (size_t)(nl + 1) * sizeof(RtLayer);
}
__host__ __device__ inline size_t rt_smem_bytes(int nl) {
  return sizeof(RtHead) + rt_layers_bytes(nl) + align16((size_t)nl * sizeof(double));
}
// floats of a column's level sums
__host__ __device__ inline size_t rt_part_floats(int nl) { return (size_t)RT_NW * (nl + 1) * 6; }

__device__ inline RtSmem rt_carve(char* p, int nl, float* part) {
  RtSmem s;
  s.h = (RtHead*)p;
  p += sizeof(RtHead);
  s.L = (RtLayer*)p + 1;
  p += rt_layers_bytes(nl);
  s.cf = (double*)p;
  s.part = part;
  return s;
}

// Where taug and the Planck fractions of a column come from.
struct GasSrc {
  const float* plane;         // taumol's plane of the column (rows of GB_LW_PROW floats), or NULL
  float* gc;                  // caller sub-columns: the cells' cloud plane [nl][140]
  const unsigned* cw;         // ... and from lw_cells_kernel the unit's first column's cell bits
  int cerr;                   // and the column's stop code
  const __half* nt;           // fp16 rows [nl][140] (network), or NULL
  const __half* nf;
  const unsigned char* flag;  // per layer: 1 -> network, 0 -> fp32 planes
};
// taumol's planes; the network's rows, on 4-byte boundaries or on any; per
// layer one or the other
enum RtMode { RT_GAS = 0, RT_NET = 1, RT_NETODD = 2, RT_MIX = 3 };

// g-point gi of band b (1..16) in a plane row: its taug, and its Planck fraction two floats on
__host__ __device__ constexpr int plane_pos(int b, int gi) { return 4 * (gb_pair0(b) + gi / 2) + gi % 2; }

// taug (x, y) and Planck fractions (z, w) of the pair of g-points g, g + 1 of
// a layer; po: the pair's position in a plane row
template <int MODE>
__device__ __forceinline__ float4 gas_at(const GasSrc& src, int lay, int g, int po) {
  if (MODE == RT_NET) {
    const int o = lay * GB_NGPT + g;
    const float2 t = __half22float2(__ldg(reinterpret_cast<const __half2*>(src.nt + o)));
    const float2 f = __half22float2(__ldg(reinterpret_cast<const __half2*>(src.nf + o)));
    return make_float4(t.x, t.y, f.x, f.y);
  }
  if (MODE == RT_NETODD || (MODE == RT_MIX && src.flag[lay] != 0)) {
    const int o = lay * GB_NGPT + g;
    return make_float4(__half2float(__ldg(src.nt + o)), __half2float(__ldg(src.nt + o + 1)),
                       __half2float(__ldg(src.nf + o)), __half2float(__ldg(src.nf + o + 1)));
  }
  // plain loads: the hand-over kernel's taumol wrote its planes in the same launch
  return *reinterpret_cast<const float4*>(src.plane + lay * GB_LW_PROW + po);
}

// Total (gas + cloud) absorptance and source factor of a cloudy cell
// (rtrnmc.f90:356-379): the expansion below 0.06, else the table at the
// clear cell's optical depth (odepth itself below 0.06, else tau_tbl at its
// index) plus the cloud's.
__device__ __forceinline__ void cloud_total(const float2* tt, int itr, float od, float odcld, float& atot,
                                            float& x) {
  const float odtot = od + odcld;
  if (odtot < 0.06f) {
    atot = fmaf(-0.5f * odtot, odtot, odtot);
    x = REC_6 * odtot;
  } else {
    const float tauq = od <= 0.06f ? od : tbl_tau(itr);
    const float2 et = tt[tbl_index(tauq + odcld)];
    atot = 1.0f - et.x;
    x = et.y;
  }
}

// ciwp + clwp >= 1e-20: on the bit patterns where neither is negative or NaN
// (the sum is no less than either, and no rounding takes it below 1e-20), in fp64 where that leaves it open
__device__ __forceinline__ bool has_paths(double ciwp, double clwp) {
  const long long i = __double_as_longlong(ciwp), l = __double_as_longlong(clwp);
  const long long kMin = __double_as_longlong(1.0e-20), kInf = 0x7FF0000000000000LL;
  if (i >= 0 && l >= 0 && i <= kInf && l <= kInf) {
    if (i >= kMin || l >= kMin) return true;
    if ((i | l) == 0) return false;
  }
  return ciwp + clwp >= 1.e-20;
}

// a caller sub-column cell's cloud value for the transfer: its cloud optical
// depth (cldprmc.f90:178-266, rtrnmc.f90:300-312) where cldfmcl = 1,
// the fraction itself where it is neither 0 nor 1
__device__ __forceinline__ float cell_value(const LwArgs& a, const RtSmem& S, int lay, int band, bool one,
                                            double cf, double ciwp, double clwp, bool paths, double tin,
                                            const float* __restrict__ T) {
  if (!one) return (float)cf;
  float tauc = 0.0f;
  bool from_paths = a.inflag == 2 && paths;
  if (!from_paths) {
    const long long tb = __double_as_longlong(tin);
    from_paths = a.inflag == 2 && tb >= __double_as_longlong(1.0e-20) && tb <= 0x7FF0000000000000LL;
    tauc = (float)tin;
  }
  if (from_paths) {
    const int fl = ((__double_as_longlong(ciwp) << 1) != 0LL ? 1 : 0) | ((__double_as_longlong(clwp) << 1) != 0LL ? 2 : 0);
    const float4 r = S.L[lay].lcw;
    tauc = cloud_tau_layer(a, band, T, make_float4((float)ciwp, (float)clwp, r.z, r.w), fl);
  }
  return tauc;
}

// the transfer's cloud of a caller sub-column cell from its hand-over value; a
// fractional cldfmc enters with zero cloud optical depth
__device__ __forceinline__ float cell_from_value(bool one, float v, float secdiff, float& odcld, float& efcl) {
  if (!one) {
    odcld = 0.0f;
    efcl = 0.0f;
    return v;
  }
  odcld = secdiff * v;
  efcl = 1.0f - __expf(-odcld);
  return 1.0f;
}

// radius checks of cldprmc (cldprmc.f90:217-266): the code it stops with for
// ice radius `rice` (iceflag) and liquid radius `rliq` (liqflag)
__device__ __forceinline__ int ice_code(int iceflag, double rice) {
  if (iceflag == 0 && rice < 10.0) return GB_COL_ICE_SMALL;
  if (iceflag == 1 && (rice < 13.0 || rice > 130.0)) return GB_COL_ICE_BOUNDS;
  if (iceflag == 2 && (rice < 5.0 || rice > 131.0)) return GB_COL_ICE_BOUNDS;
  if (iceflag == 3 && (rice < 5.0 || rice > 140.0)) return GB_COL_DGE_BOUNDS;
  return 0;
}
__device__ __forceinline__ int liq_code(int liqflag, double rliq) {
  return liqflag == 1 && (rliq < 2.5 || rliq > 60.0) ? GB_COL_LIQ_BOUNDS : 0;
}

// a unit of a block: the threads that solve a unit's columns, with a barrier of their own
struct Unit {
  int tid, nt, bar;
  const float2* tt;  // rtrnmc's (exp_tbl, tfn_tbl), in shared memory (hand-over kernel: in global)
  __device__ __forceinline__ void sync() const { asm volatile("bar.sync %0, %1;" ::"r"(bar), "r"(nt) : "memory"); }
};
// the columns of a unit: n (1 or 2) neighbouring columns of one grid from
// col0 on, `last` the grid's last column (the second column of a grid's last
// unit may be missing: it reads the last column's inputs and writes nothing)
struct Cols {
  char* smem;
  size_t stride;  // shared memory per column
  float* part;    // level sums of the first column
  int n, nlmax;
  long long col0, last;
  // item i of a loop over the unit's columns and something else: its column and the rest
  __device__ __forceinline__ int c(int i) const { return i & (n - 1); }
  __device__ __forceinline__ int rest(int i) const { return i >> (n - 1); }
  __device__ __forceinline__ RtSmem S(int c) const {
    return rt_carve(smem + c * stride, nlmax, part + c * rt_part_floats(nlmax));
  }
  __device__ __forceinline__ long long icol(int c) const { return col0 + c < last ? col0 + c : last; }
};

// rtrnmr's maximum/random overlap factors (rrtmg_lw_rtrnmr.f90:345-514), by
// one thread in fp64 from the layer fractions cf[0 .. nl-1]; lev is the
// reference's 1-based layer.  The fractions beyond the column (lev 0 and
// nl+1) are 0: the driver's cloud array is zeroed above the column
// (nomcica.f90 inatm), and below it the reference reads outside its array,
// where the surface (no cloud) is taken.  faccmb, which the reference leaves
// undefined where istcld = 1, is 0 there.  Layer lev keeps its istcld
// (istcldd) in bit 0 (1) of lfl, the upward factors at lev+1 in ovl[1..6]
// and the downward ones at lev-1 in ovl[7..12].
__device__ __noinline__ void band_overlap(const RtSmem& S, const double* __restrict__ cf, int nl) {
  auto CF = [&](int lev) -> double { return lev >= 1 && lev <= nl ? cf[lev - 1] : 0.0; };
  auto cloudy = [&](int lev) { return S.L[lev - 1].cldlay != 0; };
  enum { CLR1 = 0, CLR2, CLD1, CLD2, CMB1, CMB2 };
  double rat1 = 0.0, rat2 = 0.0;
  int st = 1;  // istcld(lev)
  for (int lev = 1; lev <= nl; ++lev) {
    if (st) S.L[lev - 1].lfl |= 1;
    float* u = S.ovl(lev - 1) + 1;  // factors at lev+1
    if (!cloudy(lev)) {
      st = 1;
      continue;
    }
    double f[6] = {0.0, 0.0, 0.0, 0.0, 0.0, 0.0};
    const double c0 = CF(lev), cp = CF(lev + 1), cm = CF(lev - 1);
    if (lev == nl) {
      // all six 0
    } else if (cp >= c0) {
      if (st) {
        if (c0 < 1.0) f[CLR2] = (cp - c0) / (1.0 - c0);
        if (lev >= 2) S.ovl(lev - 2)[1 + CLR2] = S.ovl(lev - 2)[1 + CLD2] = 0.0f;  // facclr2(lev), faccld2(lev)
      } else {
        const double fmax = c0 > cm ? c0 : cm;
        if (cp > fmax) {
          f[CLR1] = rat2;
          f[CLR2] = (cp - fmax) / (1.0 - fmax);
        } else if (cp < fmax) {
          f[CLR1] = (cp - c0) / (cm - c0);
        } else {
          f[CLR1] = rat2;
        }
      }
      if (f[CLR1] > 0.0 || f[CLR2] > 0.0) {
        rat1 = 1.0;
        rat2 = 0.0;
      } else {
        rat1 = rat2 = 0.0;
      }
    } else {
      if (st) {
        f[CLD2] = (c0 - cp) / c0;
        if (lev >= 2) S.ovl(lev - 2)[1 + CLR2] = S.ovl(lev - 2)[1 + CLD2] = 0.0f;
      } else {
        const double fmin = c0 < cm ? c0 : cm;
        if (cp <= fmin) {
          f[CLD1] = rat1;
          f[CLD2] = (fmin - cp) / fmin;
        } else {
          f[CLD1] = (c0 - cp) / (c0 - fmin);
        }
      }
      if (f[CLD1] > 0.0 || f[CLD2] > 0.0) {
        rat1 = 0.0;
        rat2 = 1.0;
      } else {
        rat1 = rat2 = 0.0;
      }
    }
    if (!st) {
      f[CMB1] = fmax(0.0, fmin(cp - c0, cm - c0));
      f[CMB2] = fmax(0.0, fmin(c0 - cp, c0 - cm));
    }
    for (int k = 0; k < 6; ++k) u[k] = (float)f[k];
    st = 0;
  }
  int sd = 1;  // istcldd(lev); rat1 and rat2 carry over from the loop above
  for (int lev = nl; lev >= 1; --lev) {
    if (sd) S.L[lev - 1].lfl |= 2;
    float* d = S.ovl(lev - 1) + 7;  // factors at lev-1
    if (!cloudy(lev)) {
      sd = 1;
      continue;
    }
    double f[6] = {0.0, 0.0, 0.0, 0.0, 0.0, 0.0};
    const double c0 = CF(lev), cp = CF(lev + 1), cm = CF(lev - 1);
    if (lev == 1) {
      // all six 0
    } else if (cm >= c0) {
      if (sd) {
        if (c0 < 1.0) f[CLR2] = (cm - c0) / (1.0 - c0);
        if (lev < nl) S.ovl(lev)[7 + CLR2] = S.ovl(lev)[7 + CLD2] = 0.0f;  // facclr2d(lev), faccld2d(lev)
      } else {
        const double fmax = c0 > cp ? c0 : cp;
        if (cm > fmax) {
          f[CLR1] = rat2;
          f[CLR2] = (cm - fmax) / (1.0 - fmax);
        } else if (cm < fmax) {
          f[CLR1] = (cm - c0) / (cp - c0);
        } else {
          f[CLR1] = rat2;
        }
      }
      if (f[CLR1] > 0.0 || f[CLR2] > 0.0) {
        rat1 = 1.0;
        rat2 = 0.0;
      } else {
        rat1 = rat2 = 0.0;
      }
    } else {
      if (sd) {
        f[CLD2] = (c0 - cm) / c0;
        if (lev < nl) S.ovl(lev)[7 + CLR2] = S.ovl(lev)[7 + CLD2] = 0.0f;
      } else {
        const double fmin = c0 < cp ? c0 : cp;
        if (cm <= fmin) {
          f[CLD1] = rat1;
          f[CLD2] = (fmin - cm) / fmin;
        } else {
          f[CLD1] = (c0 - cm) / (c0 - fmin);
        }
      }
      if (f[CLD1] > 0.0 || f[CLD2] > 0.0) {
        rat1 = 0.0;
        rat2 = 1.0;
      } else {
        rat1 = rat2 = 0.0;
      }
    }
    if (!sd) {
      f[CMB1] = fmax(0.0, fmin(cp - c0, cm - c0));
      f[CMB2] = fmax(0.0, fmin(c0 - cp, c0 - cm));
    }
    for (int k = 0; k < 6; ++k) d[k] = (float)f[k];
    sd = 0;
  }
}

// The band clouds of the non-McICA driver (nomcica.f90:886-920, rtrn.f90:319-336,
// rtrnmr.f90:334-343), for each of the block's columns: per layer the fraction, icldlyr (cldfrac >= 1e-6) and
// odcld = secdiff(ib) * taucloud(ib) for the cloud bands ib < ncbands, then
// for maximum/random overlap the overlap factors.  Ends with a barrier when
// it computes them.
__device__ __forceinline__ void band_clouds(const LwArgs& a, const Unit& U, const Cols& C, int nl, bool clouds) {
  const int tid = U.tid, nt = U.nt;
  if (!clouds) {
    for (int it = tid; it < C.n * nl; it += nt) C.S(C.c(it)).L[C.rest(it)].cldlay = 0;
    return;
  }
  for (int it = tid; it < C.n * nl; it += nt) {
    const int c = C.c(it), lay = C.rest(it);
    const RtSmem S = C.S(c);
    const double cf = in2(a.cldfrac, a.ld, C.icol(c), lay);
    S.L[lay].cldlay = cf >= 1.e-6;
    S.L[lay].lfl = 0;
    float* ov = S.ovl(lay);
    ov[0] = (float)cf;
#pragma unroll
    for (int k = 1; k < 14; ++k) ov[k] = 0.0f;
    S.cf[lay] = cf;
    if (lay == 0) S.h->iscal[2] = __ldg(a.ncbands + C.icol(c));
  }
  U.sync();  // the records' fourth words are the Planck-table rows until here
  for (int it = tid; it < C.n * nl * 16; it += nt) {
    const int c = C.c(it), lay = C.rest(it) >> 4, ib = C.rest(it) & 15;
    const RtSmem S = C.S(c);
    const long long icol = C.icol(c);
    S.L[lay].rec[ib].w = ib < __ldg(a.ncbands + icol)
                           ? S.h->misc[ib] * (float)__ldg(a.tauc + ib + 16 * (icol + a.ld * lay)) : 0.0f;
  }
  if (a.icld >= 2) {
    U.sync();
    if (tid % RT_CT == 0 && tid / RT_CT < C.n) {
      const RtSmem S = C.S(tid / RT_CT);
      band_overlap(S, S.cf, nl);
    }
  }
}

// cloud band of spectral band `band` for cldprop's band count (rtrn.f90:253-255, 345-351)
__device__ __forceinline__ int cloud_band(int ncb, int band) {
  if (ncb == 1) return 0;
  if (ncb == 5) return band < 1 ? 0 : band < 2 ? 1 : band < 5 ? 2 : band < 8 ? 3 : 4;
  return band;
}

// ---------------------------------------------------------------- the passes
// Clouds of the passes: in-kernel sub-columns (or none), caller sub-columns,
// band clouds with random or with maximum/random overlap.
enum PassKind { PK_FUSED = 0, PK_SUBCOL = 1, PK_RANDOM = 2, PK_MAXRAN = 3 };

// The downward and the upward pass of one column by the threads of its pairs of
// g-points (rtrnmc.f90:347-529), level sums per group of 32 g-points into part.
// What a thread reads of a layer is one 16-byte word of shared memory (its
// band's record), one word of cloud bits and one 16-byte load of gas optics.
// The layers go two by two.  Software pipelined: the gas optics are loaded two
// pairs of layers ahead, the exponential table is looked up one pair ahead; the
// level sums of a pair share one transposed butterfly.  A pair of layers in
// which no lane of the warp has a cloud is one run of code without a branch,
// so that its four cells' chains, the next pair's lookups and the sums
// overlap in one warp's instruction stream: an SM holds 20 of these warps,
// and a chain of a layer's cells is some 900 cycles long.
template <int MODE, int KIND>
struct Passes {
  static constexpr bool BAND = KIND >= PK_RANDOM;
  struct Stage {
    float od0, od1;  // optical depths
    float2 e0, e1;   // (exp_tbl, tfn_tbl) at their indices (used above 0.06; index 0 below, so that such
                     // lanes share a load's line)
    float2 pf;       // Planck fractions
  };
  const GasSrc& src;
  const RtLayer* L0;
  const float2* tt;  // (exp_tbl, tfn_tbl)
  const float* gc;
  float* part;
  float sd;
  float2 wgt;
  int nl, band, cband, g, po, grp, l16, lw;
  float2 cr, kr, radm;  // rtrnmr's cloudy and clear radiances and overlap term

  __device__ __forceinline__ static int index(float od) {
    return min((int)fmaf(10000.0f, tbl_quotient(od), 0.5f), 10000);
  }
  __device__ __forceinline__ float4 gas(int lay) const { return gas_at<MODE>(src, lay, g, po); }
  // stages layer lay, whose gas optics are p
  __device__ __forceinline__ Stage stage(int lay, const float4& p) const {
    Stage s;
    const float taua = L0[lay].rec[band].z;
    s.pf = make_float2(p.z, p.w);
    s.od0 = fmaxf(sd * (p.x + taua), 0.0f);
    s.od1 = fmaxf(sd * (p.y + taua), 0.0f);
    s.e0 = tt[s.od0 <= 0.06f ? 0 : index(s.od0)];
    s.e1 = tt[s.od1 <= 0.06f ? 0 : index(s.od1)];
    return s;
  }
  __device__ __forceinline__ unsigned bits(int lay) const {
    return BAND ? (unsigned)L0[lay].cldlay : (L0[lay].cbits[grp] >> l16) & 0x10001u;
  }
  // caller sub-columns: the cloud values of the layer's cells (where one has a cloud)
  __device__ __forceinline__ float2 cell_values(int lay, unsigned cl) const {
    return KIND == PK_SUBCOL && cl ? *reinterpret_cast<const float2*>(gc + lay * GB_NGPT) : make_float2(0.0f, 0.0f);
  }
  // a layer's clear-sky transmittance and source: rtrnmc's odepth <= 0.06
  // expansion or its table (rtrnmc.f90:380-413); x is odepth/6 or tfn, the
  // source plfrac * (blay + x * dplank)
  struct Clear {
    float2 at, tr, gs;
    float blay, dpl;  // layer Planck value, that of the level the pass comes to minus it
  };
  template <bool UP>
  __device__ __forceinline__ Clear clear(const Stage& s, int lay) const {
    Clear c;
    const float2 q = *reinterpret_cast<const float2*>(&L0[lay].rec[band]);
    c.blay = q.x;
    c.dpl = (UP ? q.y : L0[lay - 1].rec[band].y) - q.x;
    const bool t0 = s.od0 <= 0.06f, t1 = s.od1 <= 0.06f;
    c.at = make_float2(t0 ? fmaf(-0.5f * s.od0, s.od0, s.od0) : 1.0f - s.e0.x,
                       t1 ? fmaf(-0.5f * s.od1, s.od1, s.od1) : 1.0f - s.e1.x);
    const float x0 = t0 ? REC_6 * s.od0 : s.e0.y, x1 = t1 ? REC_6 * s.od1 : s.e1.y;
    c.gs = mul2(mul2(s.pf, make_float2(fmaf(x0, c.dpl, c.blay), fmaf(x1, c.dpl, c.blay))), c.at);
    c.tr = make_float2(1.0f - c.at.x, 1.0f - c.at.y);
    return c;
  }
  // the clouds of a layer: A and B of the total radiance's step r' = r A + B,
  // and D, by which its temperature derivative goes down
  template <bool UP>
  __device__ __forceinline__ void cloud(const Stage& s, const Clear& c, int lay, unsigned cl, const float2& cv,
                                        const float2& r, float2& A, float2& B, float2& D) {
    const RtLayer& L = L0[lay];
    float odl = 0.0f, efl = 0.0f;  // cloud optical depth and absorptance of the (layer, band)
    if (KIND == PK_FUSED) odl = sd * L.rec[band].w;
    if (BAND) odl = L.rec[cband].w;
    if (KIND == PK_FUSED || KIND == PK_RANDOM) efl = 1.0f - __expf(-odl);
    const unsigned frac = KIND == PK_SUBCOL ? L.cbits[5 + grp] >> l16 : 0u;
    auto cell = [&](bool cloudy, bool one, float od, float pf, float at, float gs, float tr, float v, float r1, float& A1,
                    float& B1, float& D1, float& cr1, float& kr1, float& rm1) {
      if constexpr (BAND) {
        const float* ov = reinterpret_cast<const float*>(L.cbits);
        const float cf = ov[0];
        float atot, x;
        cloud_total(tt, index(od), od, odl, atot, x);
        const float bbd = pf * fmaf(x, c.dpl, c.blay);
        if (UP) D1 = fmaf(cf, 1.0f - atot, (1.0f - cf) * (1.0f - at));
        if (KIND == PK_RANDOM) {  // rtrn.f90:370-432, 495-507
          const float efcl = efl * cf;
          A1 = 1.0f - fmaf(efcl, 1.0f - at, at);
          B1 = fmaf(cf, fmaf(bbd, atot, -gs), gs);
        } else {  // rtrnmr.f90:590-609, 688-713
          constexpr int o = UP ? 1 : 7;
          if (L.lfl & (UP ? 1 : 2)) {
            cr1 = cf * r1;
            kr1 = r1 - cr1;
            rm1 = 0.0f;
          }
          const float ttot = 1.0f - atot, cldsrc = bbd * atot;
          cr1 = fmaf(cr1, ttot, cf * cldsrc);
          kr1 = fmaf(kr1, tr, (1.0f - cf) * gs);
          A1 = 0.0f;
          B1 = cr1 + kr1;
          const float radmod = fmaf(rm1, fmaf(ov[o], tr, ov[o + 2] * ttot), fmaf(ov[o + 5], cldsrc, -ov[o + 4] * gs));
          const float oc = cr1 - radmod, ok = kr1 + radmod;
          rm1 = fmaf(ov[o + 1], ok, fmaf(-ov[o + 3], oc, -radmod));
          cr1 += rm1;
          kr1 -= rm1;
        }
      } else {
        if (!cloudy) return;
        float odcld = odl, efcl = efl, cldf = 1.0f, atot, x;
        if (KIND == PK_SUBCOL) cldf = cell_from_value(one, v, sd, odcld, efcl);
        cloud_total(tt, index(od), od, odcld, atot, x);
        A1 = 1.0f - fmaf(efcl, 1.0f - at, at);
        B1 = fmaf(cldf, fmaf(pf * fmaf(x, c.dpl, c.blay), atot, -gs), gs);
        if (UP) D1 = fmaf(cldf, 1.0f - atot, (1.0f - cldf) * (1.0f - at));
      }
    };
    cell(cl & 1u, !(frac & 1u), s.od0, s.pf.x, c.at.x, c.gs.x, c.tr.x, cv.x, r.x, A.x, B.x, D.x, cr.x, kr.x, radm.x);
    cell(cl >> 16, !(frac >> 16 & 1u), s.od1, s.pf.y, c.at.y, c.gs.y, c.tr.y, cv.y, r.y, A.y, B.y, D.y, cr.y, kr.y, radm.y);
  }

  // one layer of the downward pass: total and clear-sky radiance
  __device__ __forceinline__ void fall(const Stage& s, int lay, unsigned cl, const float2& cv, float2& rd,
                                       float2& rc) {
    const Clear c = clear<false>(s, lay);
    rc = fma2(rc, c.tr, c.gs);
    float2 A = c.tr, B = c.gs, D;
    if (cl) cloud<false>(s, c, lay, cl, cv, rd, A, B, D);
    rd = fma2(rd, A, B);
  }
  // one layer of the upward pass: total and clear-sky radiance and their temperature derivatives
  __device__ __forceinline__ void rise(const Stage& s, int lay, unsigned cl, const float2& cv, float2& ru,
                                       float2& rc, float2& du, float2& dc) {
    const Clear c = clear<true>(s, lay);
    rc = fma2(rc, c.tr, c.gs);
    dc = mul2(dc, c.tr);
    float2 A = c.tr, B = c.gs, D = c.tr;
    if (cl) cloud<true>(s, c, lay, cl, cv, ru, A, B, D);
    ru = fma2(ru, A, B);
    du = mul2(du, D);
  }

  // whether a lane of the warp has a cloud in either of two layers
  __device__ __forceinline__ bool cloudy(int l0, int l1) const {
    const unsigned w = BAND ? (unsigned)(L0[l0].cldlay | L0[l1].cldlay) : L0[l0].cbits[grp] | L0[l1].cbits[grp];
    return __any_sync(0xffffffffu, w != 0u);
  }

  // ---------------- downward pass (rtrnmc.f90:347-455): total and clear-sky streams; f1: layer 0's fractions
  __device__ __forceinline__ void down(float2& rd, float2& rc, float2& f1) {
    const int s4 = sum4_at(l16);
    float4 pa = gas(nl - 1), pb = gas(max(nl - 2, 0));
    Stage sa = stage(nl - 1, pa), sb = stage(max(nl - 2, 0), pb);
    pa = gas(max(nl - 3, 0)), pb = gas(max(nl - 4, 0));
    int lay = nl - 1;
#pragma unroll 1
    for (; lay >= 1; lay -= 2) {
      f1 = sb.pf;
      float2 p0, p1;
      if (cloudy(lay, lay - 1)) {
        const unsigned c0 = bits(lay), c1 = bits(lay - 1);
        const float2 v0 = cell_values(lay, c0), v1 = cell_values(lay - 1, c1);
        fall(sa, lay, c0, v0, rd, rc);
        p0 = mul2(rd, wgt), p1 = mul2(rc, wgt);
        fall(sb, lay - 1, c1, v1, rd, rc);
        sa = stage(max(lay - 2, 0), pa), sb = stage(max(lay - 3, 0), pb);
        pa = gas(max(lay - 4, 0)), pb = gas(max(lay - 5, 0));
        const float s = sum4(p0, p1, mul2(rd, wgt), mul2(rc, wgt), l16);
        if (lw < 4) part[(lay - (s4 >> 1)) * 6 + (s4 & 1)] = s;
      } else {
        const Clear c0 = clear<false>(sa, lay), c1 = clear<false>(sb, lay - 1);
        sa = stage(max(lay - 2, 0), pa), sb = stage(max(lay - 3, 0), pb);
        pa = gas(max(lay - 4, 0)), pb = gas(max(lay - 5, 0));
        rd = fma2(rd, c0.tr, c0.gs), rc = fma2(rc, c0.tr, c0.gs);
        p0 = mul2(rd, wgt), p1 = mul2(rc, wgt);
        rd = fma2(rd, c1.tr, c1.gs), rc = fma2(rc, c1.tr, c1.gs);
        const float s = sum4(p0, p1, mul2(rd, wgt), mul2(rc, wgt), l16);
        if (lw < 4) part[(lay - (s4 >> 1)) * 6 + (s4 & 1)] = s;
      }
    }
    if (lay == 0) {  // layer 0 on its own
      f1 = sa.pf;
      fall(sa, 0, bits(0), cell_values(0, bits(0)), rd, rc);
      const float s = sum2(mul2(rd, wgt), mul2(rc, wgt), l16);
      if (lw < 2) part[l16] = s;
    }
  }

  // ---------------- upward pass (rtrnmc.f90:486-529): level lay+1 above layer lay
  template <bool IDRV>
  __device__ __forceinline__ void up(float2& ru, float2& rc, float2& du, float2& dc) {
    const int s4 = sum4_at(l16), s8 = sum8_at(l16), top = nl - 1;
    auto put1 = [&](float* p) {
      if (IDRV) {
        const float s = sum4(mul2(ru, wgt), mul2(rc, wgt), mul2(du, wgt), mul2(dc, wgt), l16);
        if (lw < 4) p[s4] = s;
      } else {
        const float s = sum2(mul2(ru, wgt), mul2(rc, wgt), l16);
        if (lw < 2) p[l16] = s;
      }
    };
    float2 q0, q1, q2, q3;
    auto put2 = [&](int lay) {
      float* p = part + (lay + 1) * 6 + 2;  // levels lay+1 and lay+2
      if (IDRV) {
        const float s = sum8(q0, q1, q2, q3, mul2(ru, wgt), mul2(rc, wgt), mul2(du, wgt), mul2(dc, wgt), l16);
        if (lw < 8) p[(s8 >> 2) * 6 + (s8 & 3)] = s;
      } else {
        const float s = sum4(q0, q1, mul2(ru, wgt), mul2(rc, wgt), l16);
        if (lw < 4) p[(s4 >> 1) * 6 + (s4 & 1)] = s;
      }
    };
    put1(part + 2);
    float4 pa = gas(0), pb = gas(min(1, top));
    Stage sa = stage(0, pa), sb = stage(min(1, top), pb);
    pa = gas(min(2, top)), pb = gas(min(3, top));
    int lay = 0;
#pragma unroll 1
    for (; lay + 1 < nl; lay += 2) {
      if (cloudy(lay, lay + 1)) {
        const unsigned c0 = bits(lay), c1 = bits(lay + 1);
        const float2 v0 = cell_values(lay, c0), v1 = cell_values(lay + 1, c1);
        rise(sa, lay, c0, v0, ru, rc, du, dc);
        q0 = mul2(ru, wgt), q1 = mul2(rc, wgt), q2 = mul2(du, wgt), q3 = mul2(dc, wgt);
        rise(sb, lay + 1, c1, v1, ru, rc, du, dc);
        sa = stage(min(lay + 2, top), pa), sb = stage(min(lay + 3, top), pb);
        pa = gas(min(lay + 4, top)), pb = gas(min(lay + 5, top));
        put2(lay);
      } else {
        const Clear c0 = clear<true>(sa, lay), c1 = clear<true>(sb, lay + 1);
        sa = stage(min(lay + 2, top), pa), sb = stage(min(lay + 3, top), pb);
        pa = gas(min(lay + 4, top)), pb = gas(min(lay + 5, top));
        ru = fma2(ru, c0.tr, c0.gs), rc = fma2(rc, c0.tr, c0.gs), du = mul2(du, c0.tr), dc = mul2(dc, c0.tr);
        q0 = mul2(ru, wgt), q1 = mul2(rc, wgt), q2 = mul2(du, wgt), q3 = mul2(dc, wgt);
        ru = fma2(ru, c1.tr, c1.gs), rc = fma2(rc, c1.tr, c1.gs), du = mul2(du, c1.tr), dc = mul2(dc, c1.tr);
        put2(lay);
      }
    }
    if (lay < nl) {  // level nl on its own
      rise(sa, lay, bits(lay), cell_values(lay, bits(lay)), ru, rc, du, dc);
      put1(part + nl * 6 + 2);
    }
  }
};

template <int MODE, int KIND>
__device__ __forceinline__ void rt_passes(const LwArgs& a, const RtSmem& S, const GasSrc& src,
                                          const float2* tt, int band, int g, int po, int grp, int l16, bool inblk,
                                          float wgt) {
  const float2 zero = make_float2(0.0f, 0.0f);
  const int nl = a.nlay;
  Passes<MODE, KIND> P{src, S.L, tt,
                       KIND == PK_SUBCOL ? src.gc + g : nullptr, S.part + grp * (nl + 1) * 6, S.h->misc[band],
                       make_float2(wgt, wgt), nl, band, KIND >= PK_RANDOM ? cloud_band(S.h->iscal[2], band) : band, g, po,
                       grp, l16, inblk ? l16 : 16, zero, zero, zero};
  float2 rd = zero, rc = zero, f1 = zero;
  P.down(rd, rc, f1);
  // surface emission and reflection (rtrnmc.f90:465-485)
  const float2 rad0 = make_float2(f1.x * S.h->misc[16 + band], f1.y * S.h->misc[16 + band]);
  const float reflect = 1.0f - S.h->misc[48 + band];  // scalar: see mul2
  float2 ru = make_float2(rad0.x + reflect * rd.x, rad0.y + reflect * rd.y);
  float2 rcu = make_float2(rad0.x + reflect * rc.x, rad0.y + reflect * rc.y);
  float2 du = make_float2(f1.x * S.h->misc[32 + band], f1.y * S.h->misc[32 + band]);
  float2 dcu = du;
  if (a.idrv == 1)
    P.template up<true>(ru, rcu, du, dcu);
  else
    P.template up<false>(ru, rcu, du, dcu);
}

// a layer's radii as floats and the codes cldprmc's radius checks stop with: bits 0-7 ice, 8-15 liquid
__device__ __forceinline__ void layer_radii(const LwArgs& a, const RtSmem& S, long long icol, int lay) {
  const double rice = in2(a.reicmcl, a.ld, icol, lay), rliq = in2(a.relqmcl, a.ld, icol, lay);
  S.L[lay].lfl = ice_code(a.iceflag, rice) | (liq_code(a.liqflag, rliq) << 8);
  S.L[lay].lcw = make_float4(0.0f, 0.0f, (float)rice, (float)rliq);
}
// the layer's cloudy cells: none where no cell has cldfmcl == 1, else the fractions too
__device__ __forceinline__ void cloudy_words(const RtSmem& S, int lay) {
  unsigned* c = S.L[lay].cbits;
  const unsigned* f = S.fbits(lay);
  const bool any = (c[0] | c[1] | c[2] | c[3] | c[4]) != 0u;
  for (int w = 0; w < RT_NW; ++w) c[w] = any ? c[w] | f[w] : 0u;
}
// The cells of one of the caller's sub-columns' columns, a pair of g-points per
// thread (16 lanes of a group of 32 g-points): the layers' cloud bits into their
// records (RtLayer::cbits, RtSmem::fbits), the cloudy cells' values into the plane
// gc; returns the largest of the pair's codes that cldprmc stops with (of several
// going up the column the last).  The layers' radii and their codes (lcw, lfl) are there.
__device__ __forceinline__ int subcol_cells(const LwArgs& a, const RtSmem& S, long long icol, int nl, bool live, int g,
                                            int band, int lane, int grp, bool inblk, float* gc,
                                            const float* __restrict__ T) {
  const unsigned FULL = 0xffffffffu;
  const int l16 = lane & 15;
  // a group's word of a layer from the ballots over the low and the high g-points of its pairs
  auto word = [&](unsigned lo, unsigned hi) {
    return lane < 16 ? (lo & 0xffffu) | (hi << 16) : (lo >> 16) | (hi & 0xffff0000u);
  };
  // per layer, each group: its 32 cldfmcl values tested on their bit
  // patterns: == 1, /= 0, >= 1e-20.  A pair is one 16-byte load where the
  // caller's arrays start on such a boundary (rows are 1,120 bytes).
  const long long kOne = 0x3FF0000000000000LL, kInf = 0x7FF0000000000000LL;
  const long long kMin = __double_as_longlong(1.0e-20);
  const bool wide = (((uintptr_t)a.cldfmcl | (uintptr_t)a.ciwpmcl | (uintptr_t)a.clwpmcl | (uintptr_t)a.taucmcl) & 15) == 0;
  auto pair = [&](const double* p, long long o) {
    return wide ? __ldg(reinterpret_cast<const double2*>(p + o)) : make_double2(__ldg(p + o), __ldg(p + o + 1));
  };
#pragma unroll 8
  for (int lay = 0; lay < nl; ++lay) {
    const double2 cf = pair(a.cldfmcl, g + GB_NGPT * (icol + a.ld * lay));
    const long long b0 = live ? __double_as_longlong(cf.x) : 0LL, b1 = live ? __double_as_longlong(cf.y) : 0LL;
    const bool one0 = b0 == kOne, one1 = b1 == kOne;
    const bool fr0 = !one0 && (b0 << 1) != 0LL, fr1 = !one1 && (b1 << 1) != 0LL;  // neither +-0 nor 1 (NaN included, as /= 0 is)
    const unsigned m0 = __ballot_sync(FULL, one0), m1 = __ballot_sync(FULL, one1);
    const unsigned f0 = __ballot_sync(FULL, fr0), f1 = __ballot_sync(FULL, fr1);
    if (l16 == 0 && inblk) {
      S.L[lay].cbits[grp] = word(m0, m1);
      S.fbits(lay)[grp] = word(f0, f1);
    }
  }
  __syncwarp();
  // then, per pair with a cloud: the water paths for cldprmc's checks and the
  // cells' optical depths, formed once instead of in both passes.  Two layers'
  // loads are in flight, and the two cells share one copy of the optics: with
  // four layers and eight copies the warps waited for instructions
  int err0 = 0, err1 = 0;
#pragma unroll 2
  for (int lay = 0; lay < nl; ++lay) {
    const unsigned ob = S.L[lay].cbits[grp] >> l16, fb = S.fbits(lay)[grp] >> l16;
    if (!live || !((ob | fb) & 0x10001u)) continue;
    const long long o = g + GB_NGPT * (icol + a.ld * lay);
    const double2 cf = fb & 0x10001u ? pair(a.cldfmcl, o) : make_double2(ob & 1u, ob >> 16 & 1u);
    const double2 ci = pair(a.ciwpmcl, o), cl = pair(a.clwpmcl, o), ti = pair(a.taucmcl, o);
    auto cell = [&](bool one, bool cloudy, double cfv, double ciwp, double clwp, double tin, int& err) {
      if (!cloudy) return 0.0f;
      const long long cb = __double_as_longlong(cfv);
      if (!(cb >= kMin && cb <= kInf)) return (float)cfv;  // a fraction below cldmin: cldfmcl itself, no cloud optics
      const bool paths = has_paths(ciwp, clwp);
      const float v = cell_value(a, S, lay, band, one, cfv, ciwp, clwp, paths, tin, T);  // cldfmc >= cldmin (cldprmc.f90:178)
      const long long tb = __double_as_longlong(tin);
      if (paths || (tb >= kMin && tb <= kInf)) {
        const int e = S.L[lay].lfl;
        if (a.inflag == 1) err = GB_COL_INFLAG1;
        if (a.inflag == 2) {
          if ((__double_as_longlong(ciwp) << 1) != 0LL && (e & 0xff)) err = e & 0xff;  // ciwp /= 0
          if ((__double_as_longlong(clwp) << 1) != 0LL && (e >> 8)) err = e >> 8;      // clwp /= 0
        }
      }
      return v;
    };
    float v0 = 0.0f, v1 = 0.0f;
#pragma unroll 1
    for (int k = 0; k < 2; ++k) {
      const float v = cell(ob >> 16 * k & 1u, (ob | fb) >> 16 * k & 1u, k ? cf.y : cf.x, k ? ci.y : ci.x, k ? cl.y : cl.x,
                           k ? ti.y : ti.x, k ? err1 : err0);
      (k ? v1 : v0) = v;
    }
    *reinterpret_cast<float2*>(gc + lay * GB_NGPT + g) = make_float2(v0, v1);
  }
  return max(err0, err1);
}

// The transfer of a unit's columns (see the file header); src is that of this
// thread's column.  RT_NET: a column with any layer off the network is not
// solved; returns whether this thread's column was solved.  BAND: the non-McICA
// driver's band clouds (random overlap for icld 1, maximum/random otherwise).
// Ends with a barrier.
// CELLS: caller sub-columns' cells come from lw_cells_kernel (src.cw).
template <int MODE, bool BAND = false, bool CELLS = false>
__device__ __forceinline__ bool rt_columns(const LwArgs& a, const Unit& U, const Cols& C, const GasSrc& src,
                           const float* __restrict__ T) {
  constexpr bool NET = MODE == RT_NET || MODE == RT_NETODD;
  const unsigned FULL = 0xffffffffu;
  const int tid = U.tid, lane = tid & 31, warp = tid >> 5, nt = U.nt;
  const int nl = a.nlay;
  const bool fused = a.cloud_mode == LW_CLOUD_FUSED;
  const bool clouds = a.icld >= 1;
  // this thread's column (threads past the unit's columns go along with the last one and write nothing),
  // group of 32 g-points, lane in the group's 16, and pair of g-points (the last group has 6 live pairs)
  const int half = tid / RT_CT;
  const bool inblk = half < C.n;
  const int col = inblk ? half : C.n - 1;
  const int t = tid - half * RT_CT, grp = t >> 4, l16 = t & 15;
  const RtSmem S = C.S(col);
  const long long icol = C.icol(col);
  bool act = inblk && C.col0 + col <= C.last;
  if (tid < 4 * C.n) C.S(tid >> 2).h->iscal[tid & 3] = 0;
  if (NET) {
    U.sync();
    int off = 0;
    for (int l = t; l < nl && inblk; l += RT_CT) off |= src.flag[l] == 0;
    if (off) S.h->iscal[2] = 1;
    U.sync();
    act = act && S.h->iscal[2] == 0;
    if (C.S(0).h->iscal[2] != 0 && (C.n == 1 || C.col0 + 1 > C.last || C.S(1).h->iscal[2] != 0)) return false;
  }
  // this thread's g-points and their band (read from the table blob: a
  // constant-bank lookup indexed by the thread would be re-issued in the loops
  // wherever the compiler does not keep the value in a register)
  const bool live = inblk && t < GB_NGPT / 2;
  const int g = live ? 2 * t : GB_NGPT - 2;
  const int band = __float_as_int(__ldg(T + c_T.gpt_band + g));
  const int po = plane_pos(band + 1, g - c_T.band[band].g0);
  U.sync();

  // ---------------- per layer: inatm's column amounts (pwvcm), value checks, laytrop, Planck rows
  const float amd = 28.9660f, amw = 18.0160f;
  const int nvw = min(RT_NW, (nl + 31) >> 5);  // sums of 32 layers each (layers 160 apart in one lane)
  for (int i = warp; i < C.n * nvw; i += nt >> 5) {
    const int c = C.c(i), vw = C.rest(i);
    const RtSmem Sc = C.S(c);
    const long long ic = C.icol(c);
    float amttl = 0.0f, wvttl = 0.0f;
    int bad = 0;
    for (int lay = vw * 32 + lane; lay < nl; lay += RT_NT) {
      const double pd = in2(a.play, a.ld, ic, lay);
      const float pavel = (float)pd;
      const float tavel = (float)in2(a.tlay, a.ld, ic, lay);
      const double dpz = in2(a.plev, a.ld, ic, lay) - in2(a.plev, a.ld, ic, lay + 1);
      const float w1 = (float)in2(a.h2ovmr, a.ld, ic, lay);
      const float tz = (float)in2(a.tlev, a.ld, ic, lay);
      const float amm = (1.0f - w1) * amd + w1 * amw;
      const float coldry = (float)dpz * 1.e3f * (float)c_T.avogad / (1.e2f * (float)c_T.grav * amm * (1.0f + w1));
      const float wk1 = coldry * w1;
      amttl += coldry + wk1;
      wvttl += wk1;
      if (!(pavel > 0.0f) || !(tavel > 0.0f) || !isfinite(pavel) || !isfinite(tavel)) bad = 1;
      const bool lower = lower_atmosphere(pd, __logf(pavel));
      Sc.L[lay].cldlay = lower;
      if (lower) atomicAdd(&Sc.h->iscal[1], 1);
      // Planck-table rows of the level below and of the layer (setcoef.f90:173-269)
      const int ind = clampi((int)(tz - 159.0f), 1, 180);
      const int il = clampi((int)(tavel - 159.0f), 1, 180);
      float4* r = Sc.L[lay - 1].rec;
      r[0].w = __int_as_float(ind), r[1].w = tz - 159.0f - (float)ind;
      r[2].w = __int_as_float(il), r[3].w = tavel - 159.0f - (float)il;
      if (lay == nl - 1) {
        const float tt = (float)in2(a.tlev, a.ld, ic, nl);
        const int it = clampi((int)(tt - 159.0f), 1, 180);
        float4* t = Sc.L[lay].rec;
        t[0].w = __int_as_float(it), t[1].w = tt - 159.0f - (float)it;
      }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {  // fixed-order sums: 32 layers, then these in order
      amttl += __shfl_xor_sync(FULL, amttl, o);
      wvttl += __shfl_xor_sync(FULL, wvttl, o);
    }
    if (lane == 0) {
      Sc.h->red[2 * vw] = amttl;
      Sc.h->red[2 * vw + 1] = wvttl;
    }
    if (bad) atomicOr(&Sc.h->iscal[3], 1);
  }
  U.sync();
  // lower-atmosphere layers must form the prefix 0 .. laytrop-1
  for (int i = tid; i < C.n * nl; i += nt) {
    const RtSmem Sc = C.S(C.c(i));
    const int lay = C.rest(i);
    if (Sc.L[lay].cldlay != (lay < Sc.h->iscal[1] ? 1 : 0)) atomicOr(&Sc.h->iscal[3], 2);
  }
  if (tid < 16 * C.n) {
    // pwvcm (inatm :869-870) and secdiff (rtrnmc.f90:258-266), one band per thread
    const int ib = C.rest(tid);
    const RtSmem Sc = C.S(C.c(tid));
    const long long ic = C.icol(C.c(tid));
    float at = Sc.h->red[0], wt = Sc.h->red[1];
    for (int w = 1; w < nvw; ++w) {
      at += Sc.h->red[2 * w];
      wt += Sc.h->red[2 * w + 1];
    }
    const float wvsh = (amw * wt) / (amd * at);
    const float pz0 = (float)in2(a.plev, a.ld, ic, 0);
    const float pwvcm = wvsh * (1.e3f * pz0) / (1.e2f * (float)c_T.grav);
    float sd = 1.66f;
    if (!(ib == 0 || ib == 3 || ib >= 9)) {
      sd = c_a0[ib] + c_a1[ib] * __expf(c_a2[ib] * pwvcm);
      sd = fminf(fmaxf(sd, 1.50f), 1.80f);
    }
    Sc.h->misc[ib] = sd;
    // surface source and its temperature derivative (setcoef.f90:270-282)
    const float tb = (float)__ldg(a.tsfc + ic);
    const int ind = clampi((int)(tb - 159.0f), 1, 180);
    const float fr = tb - 159.0f - (float)ind;
    const float se = (float)__ldg(a.emis + ic + a.ld * ib);
    const float* tp = T + c_T.totplnk + ib * 181;
    const float* td = T + c_T.totplnkderiv + ib * 181;
    Sc.h->misc[16 + ib] = se * (tp[ind - 1] + fr * (tp[ind] - tp[ind - 1]));
    Sc.h->misc[32 + ib] = se * (td[ind - 1] + fr * (td[ind] - td[ind - 1]));
    Sc.h->misc[48 + ib] = se;
  }
  U.sync();
  // ---------------- per (layer, band): Planck values and the aerosol optical depth (rrtmg_lw_rad.f90:548-553)
#pragma unroll 2
  for (int i = tid; i < C.n * nl * 16; i += nt) {
    const int lay = C.rest(i) >> 4, ib = C.rest(i) & 15;
    const RtSmem Sc = C.S(C.c(i));
    const float* tp = T + c_T.totplnk + ib * 181;
    const float4 *r0 = Sc.L[lay - 1].rec, *r1 = Sc.L[lay].rec;  // their fourth words (see the phase above)
    const int i0 = __float_as_int(r0[0].w), il = __float_as_int(r0[2].w), i1 = __float_as_int(r1[0].w);
    const float pdn = tp[i0 - 1] + r0[1].w * (tp[i0] - tp[i0 - 1]);
    const float pup = tp[i1 - 1] + r1[1].w * (tp[i1] - tp[i1 - 1]);
    const float blay = tp[il - 1] + r0[3].w * (tp[il] - tp[il - 1]);
    const float taua = (float)__ldg(a.tauaer + C.icol(C.c(i)) + a.ld * (lay + (long long)nl * ib));
    float4& r = Sc.L[lay].rec[ib];  // its w is the clouds'
    *reinterpret_cast<float2*>(&r) = make_float2(blay, pup);
    r.z = taua;
    if (lay == 0) Sc.L[-1].rec[ib].y = pdn;
  }
  // ---------------- clouds: the cells' McICA bits, cldprmc's optical depths and stop conditions
  if constexpr (BAND) {
    band_clouds(a, U, C, nl, clouds);
  } else {
  for (int i = tid; i < C.n * nl * 5 && !(CELLS && clouds && !fused); i += nt) {
    const int r = C.rest(i), l = r / 5, w = r - 5 * l;
    const RtSmem Sc = C.S(C.c(i));
    Sc.L[l].cbits[w] = 0u;
  }
  // a group's word of a layer from the ballots over the low and the high g-points of its pairs
  auto word = [&](unsigned lo, unsigned hi) {
    return lane < 16 ? (lo & 0xffffu) | (hi << 16) : (lo >> 16) | (hi & 0xffff0000u);
  };
  if (clouds && fused) {
    // per layer, once: the McICA threshold and the layer's cloud quantities
    for (int i = tid; i < C.n * nl; i += nt) {
      const int lay = C.rest(i);
      const RtSmem Sc = C.S(C.c(i));
      const long long ic = C.icol(C.c(i));
      double cf = in2(a.cldfrac, a.ld, ic, lay);
      if (cf < 1.0e-20) cf = 0.0;
      // draws are in [0, 1], so cdf >= 1 - cldf compares the bit patterns (and
      // for a threshold >= 0 the integer order is the floating-point order);
      // a negative threshold takes every cell, a NaN none
      const double thr = 1.0 - cf;
      Sc.cthr(lay) = thr < 0.0 ? LLONG_MIN : (thr == thr ? __double_as_longlong(thr) : LLONG_MAX);
      const double ciwp = in2(a.ciwp, a.ld, ic, lay), clwp = in2(a.clwp, a.ld, ic, lay);
      const double rice = in2(a.reicmcl, a.ld, ic, lay), rliq = in2(a.relqmcl, a.ld, ic, lay);
      const int fl = (ciwp != 0.0 ? 1 : 0) | (clwp != 0.0 ? 2 : 0) | (ciwp + clwp >= 1.e-20 ? 4 : 0);
      int e = 0;
      if (ciwp != 0.0) e = ice_code(a.iceflag, rice);
      if (clwp != 0.0 && liq_code(a.liqflag, rliq)) e = GB_COL_LIQ_BOUNDS;
      Sc.L[lay].lfl = fl | (e << 8);
      Sc.L[lay].lcw = make_float4((float)ciwp, (float)clwp, (float)rice, (float)rliq);
    }
    // these g-points' draws (mcica_subcol_gen_lw.f90:484-512, icld 3) as bit
    // patterns, and the warp's largest
    const double2 dr = __ldg(reinterpret_cast<const double2*>(a.draws + icol * GB_NGPT + g));
    const long long d0 = __double_as_longlong(dr.x), d1 = __double_as_longlong(dr.y);
    long long mx = live ? (d0 > d1 ? d0 : d1) : LLONG_MIN;
#pragma unroll
    for (int o = 8; o > 0; o >>= 1) {
      const long long v = __shfl_xor_sync(FULL, mx, o);
      mx = v > mx ? v : mx;
    }
    U.sync();
    // cloudy cells: cdf(g) >= 1 - cldf(lay) (mcica_subcol_gen_lw.f90:650); a
    // layer whose threshold is above every draw of the warp has none there
    for (int lay = 0; lay < nl; ++lay) {
      const long long tb = S.cthr(lay);
      if (__all_sync(FULL, tb > mx)) continue;
      const unsigned m0 = __ballot_sync(FULL, live && d0 >= tb), m1 = __ballot_sync(FULL, live && d1 >= tb);
      if (l16 == 0 && inblk) S.L[lay].cbits[grp] = word(m0, m1);
    }
    U.sync();
    for (int i = tid; i < C.n * nl; i += nt) {
      const RtSmem Sc = C.S(C.c(i));
      const unsigned* c = Sc.L[C.rest(i)].cbits;
      Sc.L[C.rest(i)].cldlay = (c[0] | c[1] | c[2] | c[3] | c[4]) != 0u;
    }
    U.sync();
    // cloud optical depth per (layer, band) where the band has a cloudy
    // sub-column (the values cldprmc computes for every such cell), and
    // cldprmc's stop conditions (of several in a column the one that 160
    // threads, each going up the column, would be left with)
    const long long kMin = __double_as_longlong(1.0e-20), kInf = 0x7FF0000000000000LL;
    for (int v = tid; v < C.n * RT_NT; v += nt) {
      const RtSmem Sc = C.S(C.c(v));
      const long long ic = C.icol(C.c(v));
      int err = 0;
      for (int it = C.rest(v); it < nl * 16; it += RT_NT) {
        const int lay = it >> 4, ib = it & 15;
        if (!Sc.L[lay].cldlay) continue;
        const int p0 = c_T.band[ib].g0 >> 1, np = c_T.band[ib].ng >> 1;
        bool any = false;
        for (int k = p0; k < p0 + np; ++k) {
          const unsigned w = Sc.L[lay].cbits[k >> 4];
          any |= ((w | w >> 16) >> (k & 15)) & 1u;
        }
        if (!any) continue;
        const double tin = __ldg(a.tauc + ib + 16 * (ic + a.ld * lay));
        const long long tinb = __double_as_longlong(tin);
        const bool tin_ok = tinb >= kMin && tinb <= kInf;  // tin >= 1e-20
        const int fl = Sc.L[lay].lfl;
        const bool cond = (fl & 4) || tin_ok;
        Sc.L[lay].rec[ib].w = a.inflag == 2 && cond ? cloud_tau_layer(a, ib, T, Sc.L[lay].lcw, fl) : (float)tin;
        if (cond) {
          if (a.inflag == 1) err = GB_COL_INFLAG1;
          if (a.inflag == 2 && (fl >> 8)) err = fl >> 8;
        }
      }
      if (err) atomicMax(&Sc.h->iscal[0], err);
    }
  } else if (clouds) {
    // caller sub-columns
    if constexpr (CELLS) {
      for (int i = tid; i < C.n * nl * CELL_WORDS; i += nt) {
        const int c = C.c(i), r = C.rest(i), lay = r / CELL_WORDS, w = r - CELL_WORDS * lay;
        C.S(c).L[lay].cbits[w] = src.cw[(size_t)c * C.nlmax * CELL_WORDS + r];
      }
      if (t == 0 && inblk) S.h->iscal[0] = src.cerr;
    } else {
    for (int i = tid; i < C.n * nl; i += nt) layer_radii(a, C.S(C.c(i)), C.icol(C.c(i)), C.rest(i));
    U.sync();
    const int err = subcol_cells(a, S, icol, nl, live, g, band, lane, grp, inblk, src.gc, T);
    if (err) atomicMax(&S.h->iscal[0], err);
    U.sync();
    for (int i = tid; i < C.n * nl; i += nt) cloudy_words(C.S(C.c(i)), C.rest(i));
    }
  } else {
    for (int i = tid; i < C.n * nl; i += nt) C.S(C.c(i)).L[C.rest(i)].cldlay = 0;
  }
  }
  U.sync();
  if (t == 0 && act) {
    int err = S.h->iscal[0];
    if (S.h->iscal[3] & 2) err = GB_COL_LAYTROP;
    if (S.h->iscal[3] & 1) err = GB_COL_BADVAL;
    if (BAND) {  // the column status already holds cldprop's code
      if (err) {
        if (a.col_err) atomicMax(a.col_err + icol, err);
        atomicMax(a.err_flag, err);
      }
    } else if (err) {
      if (a.col_err) a.col_err[icol] = err;
      atomicMax(a.err_flag, err);
    } else if (a.col_err) {
      a.col_err[icol] = 0;
    }
  }

  if (warp * 32 < C.n * RT_CT) {  // a warp with threads of the unit's columns
    const float wgt = live ? __ldg(T + c_T.gpt_wgt + g) : 0.0f;
    if (BAND && a.icld >= 2)
      rt_passes<MODE, BAND ? PK_MAXRAN : PK_FUSED>(a, S, src, U.tt, band, g, po, grp, l16, inblk, wgt);
    else if (BAND)
      rt_passes<MODE, BAND ? PK_RANDOM : PK_FUSED>(a, S, src, U.tt, band, g, po, grp, l16, inblk, wgt);
    else if (clouds && !fused)
      rt_passes<MODE, BAND ? PK_FUSED : PK_SUBCOL>(a, S, src, U.tt, band, g, po, grp, l16, inblk, wgt);
    else
      rt_passes<MODE, PK_FUSED>(a, S, src, U.tt, band, g, po, grp, l16, inblk, wgt);
  }
  U.sync();

  // ---------------- fp64 outputs: fluxes, net fluxes, heating rates (rtrnmc.f90:566-592)
  const long long ldo = a.ldo;
  const bool idrv = a.idrv == 1;
  auto solved = [&](int c) {  // a column of the grid, and on the network where that was asked
    return C.col0 + c <= C.last && (!NET || C.S(c).h->iscal[2] == 0);
  };
  for (int i = tid; i < C.n * (nl + 1); i += nt) {
    const int c = C.c(i), lev = C.rest(i);
    const RtSmem Sc = C.S(c);
    double* fnet = reinterpret_cast<double*>(Sc.L);  // [nl+1][2]
    // the five groups' fp32 partials summed without rounding error: Knuth's
    // two-sum keeps each addition's rounding error, and the sum and the
    // accumulated errors go to fp64 together
    double acc[6];
#pragma unroll
    for (int k = 0; k < 6; ++k) {
      float hi = Sc.part[lev * 6 + k], lo = 0.0f;
#pragma unroll
      for (int w = 1; w < RT_NW; ++w) {
        const float b = Sc.part[(w * (nl + 1) + lev) * 6 + k];
        const float sum = hi + b, bv = sum - hi;
        lo += (hi - (sum - bv)) + (b - bv);
        hi = sum;
      }
      acc[k] = (double)hi + (double)lo;
    }
    if (lev == nl) acc[0] = acc[1] = 0.0;  // no downward radiation at the model top
    fnet[lev * 2 + 0] = acc[2] - acc[0];
    fnet[lev * 2 + 1] = acc[3] - acc[1];
    if (!solved(c)) continue;
    const long long o = C.col0 + c + ldo * lev;
    a.uflx[o] = acc[2];
    a.dflx[o] = acc[0];
    a.uflxc[o] = acc[3];
    a.dflxc[o] = acc[1];
    if (idrv) {
      a.duflx_dt[o] = acc[4];
      a.duflxc_dt[o] = acc[5];
    }
  }
  U.sync();
  for (int i = tid; i < C.n * nl; i += nt) {
    const int c = C.c(i), l = C.rest(i);
    if (!solved(c)) continue;
    const double* fnet = reinterpret_cast<const double*>(C.S(c).L);
    const double dp = in2(a.plev, a.ld, C.col0 + c, l) - in2(a.plev, a.ld, C.col0 + c, l + 1);
    const double f = c_T.heatfac / dp;  // one division for both heating rates
    const long long o = C.col0 + c + ldo * l;
    a.hr[o] = f * (fnet[l * 2] - fnet[(l + 1) * 2]);
    a.hrc[o] = f * (fnet[l * 2 + 1] - fnet[(l + 1) * 2 + 1]);
  }
  U.sync();
  return act;
}

// ------------------------------------------------------------------ kernels
__device__ __forceinline__ int grid_of(const LwBatch& B, long long gc, int gi) {
  while (gc >= B.col0[gi + 1]) ++gi;
  return gi;
}

// The column's grid arguments are copied into shared memory (the first
// ARGS_BYTES of every kernel's dynamic shared memory): the loops then read
// them as shared-memory broadcasts instead of constant-bank loads indexed by
// the grid number, which the compiler re-issues wherever it does not keep a
// field in a register.
constexpr size_t ARGS_BYTES = (sizeof(LwArgs) + 15) & ~size_t(15);
static_assert(sizeof(LwArgs) % 4 == 0, "LwArgs copied as 32-bit words");
__device__ __forceinline__ const LwArgs& stage_args(const LwArgs& a, char* smem, const Unit& U) {
  U.sync();  // every thread is done with the previous column's copy
  int* dst = reinterpret_cast<int*>(smem);
  const int* src = reinterpret_cast<const int*>(&a);
  for (int k = U.tid; k < (int)(sizeof(LwArgs) / 4); k += U.nt) dst[k] = src[k];
  U.sync();
  return *reinterpret_cast<const LwArgs*>(smem);
}

// rtrnmc's (exp_tbl, tfn_tbl) copied to shared memory by the whole block; ends with a barrier
constexpr size_t TABLE_BYTES = (size_t(10001) * 8 + 15) & ~size_t(15);
__device__ __forceinline__ const float2* stage_table(const float* __restrict__ T, char* smem) {
  const float4* src = reinterpret_cast<const float4*>(T + c_T.tbl_tt);  // tables start on 16-byte boundaries
  float4* dst = reinterpret_cast<float4*>(smem);
  for (int k = threadIdx.x; k < (int)(TABLE_BYTES / 16); k += blockDim.x) dst[k] = __ldg(src + k);
  __syncthreads();
  return reinterpret_cast<const float2*>(smem);
}

// taumol's outputs as [layer][140] planes
struct SampleOut {
  float *gt, *gf;
  __device__ __forceinline__ void put(int b, int lay, int gi, float tau, float frac) const {
    const int o = lay * GB_NGPT + g0_const(b) + gi;
    gt[o] = tau;
    gf[o] = frac;
  }
};
// taumol's outputs as the transfer's plane of a column
struct PlaneOut {
  float* plane;
  __device__ __forceinline__ void put(int b, int lay, int gi, float tau, float frac) const {
    float* p = plane + lay * GB_LW_PROW + plane_pos(b, gi);
    p[0] = tau;
    p[2] = frac;
  }
};

// taumol alone over batch columns [c0, c1): column c0 + k into slot k of gtau and gfrac.
template <int NT>
__global__ void __launch_bounds__(NT) lw_gas_kernel(const __grid_constant__ LwBatch B, const float* __restrict__ T,
                                                    long long c0, long long c1) {
  extern __shared__ __align__(16) char smem_raw[];
  const GasSmem s = gas_carve(smem_raw + ARGS_BYTES, B.nsmax);
  int gi = 0;
  for (long long i = c0 + blockIdx.x; i < c1; i += gridDim.x) {
    gi = grid_of(B, i, gi);
    const LwArgs& a = stage_args(B.g[gi], smem_raw, Unit{(int)threadIdx.x, NT, 1, nullptr});
    const long long slot = i - c0;
    gas_column<NT>(a, i - B.col0[gi], s, SampleOut{B.gtau + slot * B.gstride, B.gfrac + slot * B.gstride}, T);
  }
}

// what a thread's column reads its gas optics from
__device__ __forceinline__ GasSrc net_source(const LwArgs& a, long long icol) {
  GasSrc src{};
  const long long row = icol * a.nlay * GB_NGPT;
  src.nt = a.sur_tau + row;
  src.nf = a.sur_frac + row;
  src.flag = a.sur_flag + icol * a.nlay;
  return src;
}

// The transfer over units [u0, u1).  A block is the SM's only one: MAXU units
// at most, of RT_NT threads (two columns) or of half as many (one), that go
// through the batch side by side, each with its own barrier; they share one copy of
// rtrnmc's table (80 KB) in shared memory.  In L1 the table's lookups, spread
// over 32 lines a warp, missed to L2 in every second case.
// RT_GAS: on taumol's planes, unit u in plane slots (u - u0) * cpb .. (BAND: the
// non-McICA driver's band clouds).  RT_NET: on the network's gas optics; a
// column with a layer off the network is appended to B.fall instead.
template <int MAXU, int MODE, bool BAND>
__global__ void __launch_bounds__(RT_NT * MAXU, 1) lw_rt_kernel(const __grid_constant__ LwBatch B,
                                                                const float* __restrict__ T, long long u0,
                                                                long long u1, int nunit) {
  extern __shared__ __align__(16) char smem_raw[];
  const float2* tt = stage_table(T, smem_raw);
  const int nt = blockDim.x / nunit, unit = threadIdx.x / nt;
  const Unit U{(int)threadIdx.x - unit * nt, nt, 1 + unit, tt};
  const int slot = blockIdx.x * nunit + unit;  // of the resident units
  char* smem = smem_raw + TABLE_BYTES + unit * (ARGS_BYTES + B.cpb * rt_smem_bytes(B.nsmax));
  const int half = U.tid / RT_CT, col = half < B.cpb ? half : B.cpb - 1;
  int gi = 0;
  for (long long u = u0 + slot; u < u1; u += (long long)gridDim.x * nunit) {
    while (u >= B.unit0[gi + 1]) ++gi;
    const LwArgs& a = stage_args(B.g[gi], smem, U);
    const Cols C{smem + ARGS_BYTES, rt_smem_bytes(B.nsmax), B.part + (size_t)slot * B.cpb * rt_part_floats(B.nsmax),
                 B.cpb, B.nsmax, (u - B.unit0[gi]) * B.cpb, a.ncol - 1};
    GasSrc src{};
    if (MODE == RT_GAS)
      src.plane = B.plane + ((u - u0) * B.cpb + col) * B.nsmax * GB_LW_PROW;
    else if (a.sur_flag)
      src = net_source(a, C.icol(col));
    constexpr bool CELLS = MODE == RT_GAS && !BAND;
    if constexpr (CELLS) {
      if (B.cellw) {
        const long long ps = (u - u0) * B.cpb;
        src.gc = B.gcld + (ps + col) * B.nsmax * GB_NGPT;
        src.cw = B.cellw + ps * B.nsmax * CELL_WORDS;
        src.cerr = __ldg(B.cellerr + ps + col);
      }
    } else if (!BAND) {
      src.gc = B.gcld + ((long long)slot * B.cpb + col) * B.nsmax * GB_NGPT;
    }
    const bool done = (MODE == RT_GAS || a.sur_flag) && rt_columns<MODE, BAND, CELLS>(a, U, C, src, T);
    if (MODE != RT_GAS && !done && U.tid == half * RT_CT && half < B.cpb && C.col0 + col <= C.last)
      B.fall[atomicAdd(B.nfall, 1u)] = B.col0[gi] + C.col0 + col;
  }
}

// The cells of caller sub-columns for the column slots of units [u0, ..): each
// column's cloud bits, the cloudy cells' values and its stop code, a block per
// column.  The arrays are read once, so what bounds it is latency: it has 39 warps
// of an SM in flight, the transfer kernel 20, where this took as long as the
// passes (32,768 columns of 45 layers, all kernels: 4.45 ms there, 3.78 ms as
// a kernel of its own, 3.45 ms with two layers unrolled in place of four and without a
// sum in fp64 per cell).
constexpr int CELL_NT = 96;
__global__ void __launch_bounds__(CELL_NT, 13) lw_cells_kernel(const __grid_constant__ LwBatch B,
                                                           const float* __restrict__ T, long long u0) {
  extern __shared__ __align__(16) char smem_raw[];
  const long long slot = blockIdx.x;
  long long icol;
  const LwArgs& a = B.g[slot_column(B, u0, slot, icol)];
  const bool none = icol >= a.ncol || a.cloud_mode != LW_CLOUD_SUBCOL || a.icld < 1;
  if (none) {
    if (threadIdx.x == 0) B.cellerr[slot] = 0;
    return;
  }
  const int t = threadIdx.x, lane = t & 31, nl = a.nlay;
  const RtSmem S = rt_carve(smem_raw, nl, nullptr);
  const bool inblk = t < RT_CT, live = t < GB_NGPT / 2;
  const int g = live ? 2 * t : GB_NGPT - 2;
  const int band = __float_as_int(__ldg(T + c_T.gpt_band + g));
  if (t == 0) S.h->iscal[0] = 0;
  for (int lay = t; lay < nl; lay += CELL_NT) layer_radii(a, S, icol, lay);
  __syncthreads();
  const int err = subcol_cells(a, S, icol, nl, live, g, band, lane, t >> 4, inblk, B.gcld + slot * B.nsmax * GB_NGPT, T);
  if (err) atomicMax(&S.h->iscal[0], err);
  __syncthreads();
  for (int lay = t; lay < nl; lay += CELL_NT) cloudy_words(S, lay);
  if (t == 0) B.cellerr[slot] = S.h->iscal[0];
  __syncthreads();
  unsigned* out = B.cellw + slot * B.nsmax * CELL_WORDS;
  for (int i = t; i < nl * CELL_WORDS; i += CELL_NT) out[i] = S.L[i / CELL_WORDS].cbits[i % CELL_WORDS];
}

// The columns handed over by the network's transfer kernel (B.fall), one per
// block: taumol into the block's plane slot, then the transfer with each
// layer's gas optics from the network or from taumol.  rtrnmc's table is read
// through L1: with a copy of it in shared memory a second block fitted up to 96
// layers only (3,000 columns handed over: of 128 layers 3.74 ms, 2.45 ms with the
// table in L1; 8,192 columns of 45 and of 60 layers 3.23 and 3.86 ms, 3.23 and 3.57 ms).
__global__ void __launch_bounds__(RT_NT, LIST_PER_SM) lw_list_kernel(const __grid_constant__ LwBatch B,
                                                                     const float* __restrict__ T) {
  extern __shared__ __align__(16) char smem_raw[];
  const long long n = (long long)*B.nfall;
  if (blockIdx.x >= n) return;
  const Unit U{(int)threadIdx.x, RT_NT, 1, reinterpret_cast<const float2*>(T + c_T.tbl_tt)};
  char* smem = smem_raw;
  const GasSmem gs = gas_carve(smem + ARGS_BYTES, B.nsmax);  // the transfer uses the same memory afterwards
  float* plane = B.plane + (long long)blockIdx.x * B.nsmax * GB_LW_PROW;
  for (long long i = blockIdx.x; i < n; i += gridDim.x) {
    const long long gc = B.fall[i];
    const int gi = grid_of(B, gc, 0);  // the list is in no particular order
    const LwArgs& a = stage_args(B.g[gi], smem, U);
    const long long icol = gc - B.col0[gi];
    gas_column<RT_NT>(a, icol, gs, PlaneOut{plane}, T);
    const Cols C{smem + ARGS_BYTES, rt_smem_bytes(B.nsmax), B.part + blockIdx.x * rt_part_floats(B.nsmax), 1, B.nsmax,
                 icol, icol};
    GasSrc src = a.sur_flag ? net_source(a, icol) : GasSrc{};
    src.plane = plane;
    src.gc = B.gcld + (long long)blockIdx.x * B.nsmax * GB_NGPT;
    if (a.sur_flag)
      rt_columns<RT_MIX>(a, U, C, src, T);
    else
      rt_columns<RT_GAS>(a, U, C, src, T);
  }
}

constexpr int GAS_NT = 128;      // threads of the taumol kernel
constexpr int BAND_MAXU = 4;

// compiled shapes: the most units (column blocks) of an SM that the register
// allocation is sized for; variant 0 is the default
#define GB_LW_VARIANTS(X) X(0, 4) X(1, 3) X(2, 5) X(3, 2)

}  // namespace gb

// ------------------------------------------------------------------ host side
namespace {

struct VariantInfo {
  int max_units;
  const void* fn;  // the kernel this shape launches
  cudaError_t (*launch)(const LwBatch&, const float*, long long, long long, int, int, int, size_t, cudaStream_t);
};

template <int MAXU, int MODE, bool BAND>
cudaError_t launch_rt(const LwBatch& b, const float* T, long long u0, long long u1, int nblocks, int threads, int nunit,
                      size_t smem, cudaStream_t st) {
  gb::lw_rt_kernel<MAXU, MODE, BAND><<<nblocks, threads, smem, st>>>(b, T, u0, u1, nunit);
  return cudaGetLastError();
}
template <int MAXU, int MODE, bool BAND>
constexpr VariantInfo variant_of() {
  return {MAXU, (const void*)gb::lw_rt_kernel<MAXU, MODE, BAND>, launch_rt<MAXU, MODE, BAND>};
}

// the transfer kernel on taumol's planes, on the network's outputs (also where
// these do not start on 4-byte boundaries), and for band clouds
#define GB_LW_GAS_ENTRY(i, mu) variant_of<mu, gb::RT_GAS, false>(),
#define GB_LW_NET_ENTRY(i, mu) variant_of<mu, gb::RT_NET, false>(),
const VariantInfo kVariants[] = {GB_LW_VARIANTS(GB_LW_GAS_ENTRY)};
const VariantInfo kLean[] = {GB_LW_VARIANTS(GB_LW_NET_ENTRY)};
const VariantInfo kOdd = variant_of<4, gb::RT_NETODD, false>();
const VariantInfo kBand = variant_of<gb::BAND_MAXU, gb::RT_GAS, true>();
constexpr int kNumVariants = sizeof(kVariants) / sizeof(kVariants[0]);
constexpr int kMaxPerSm = 5;  // most units of an SM any shape launches

const VariantInfo& info(int variant, bool lean) { return lean ? kLean[variant] : kVariants[variant]; }

size_t device_smem() {
  int dev = 0, n = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&n, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
  return (size_t)n;
}

int device_sms() {
  int dev = 0, nsm = 1;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
  return nsm;
}

// shared memory of a block of the transfer kernel, and of the hand-over kernel (taumol or transfer area)
size_t block_smem(int nlay, int cpb, int units) {
  return gb::TABLE_BYTES + units * (gb::ARGS_BYTES + cpb * gb::rt_smem_bytes(nlay));
}
size_t list_smem(int nlay) {
  return gb::ARGS_BYTES + std::max(gb::rt_smem_bytes(nlay), gb::gas_smem_bytes(nlay));
}

// Shared-memory carve-out for `per` resident blocks of `smem` bytes: just what
// they need, so that the rest of the SM's memory stays L1 for the table
// gathers and input loads.
cudaError_t set_carveout(const void* fn, size_t smem, int per) {
  int dev = 0, max_sm = 0, reserved = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&max_sm, cudaDevAttrMaxSharedMemoryPerMultiprocessor, dev);
  cudaDeviceGetAttribute(&reserved, cudaDevAttrReservedSharedMemoryPerBlock, dev);
  if (max_sm <= 0) return cudaSuccess;
  int pct = (int)std::ceil(100.0 * (double)per * (double)(smem + reserved) / (double)max_sm);
  pct = pct < 1 ? 1 : (pct > 100 ? 100 : pct);
  return cudaFuncSetAttribute(fn, cudaFuncAttributePreferredSharedMemoryCarveout, pct);
}

// resident blocks per SM of `fn` with `threads` and `smem`
cudaError_t occupancy(const void* fn, int threads, size_t smem, int* per) {
  cudaError_t e = gb_allow_smem(fn);
  if (e == cudaSuccess) e = cudaFuncSetAttribute(fn, cudaFuncAttributePreferredSharedMemoryCarveout, cudaSharedmemCarveoutMaxShared);
  if (e != cudaSuccess) return e;
  return cudaOccupancyMaxActiveBlocksPerMultiprocessor(per, fn, threads, smem);
}

// One launch of a kernel with `nblocks` blocks and the carve-out for those resident.
template <class F>
cudaError_t launch_resident(const void* fn, int threads, size_t smem, int nblocks, F&& go) {
  int per = 0;
  cudaError_t e = occupancy(fn, threads, smem, &per);
  if (e != cudaSuccess) return e;
  if (per < 1) return cudaErrorInvalidConfiguration;
  const int nsm = device_sms();
  const int resident = (nblocks + nsm - 1) / nsm;
  e = set_carveout(fn, smem, resident < per ? resident : per);
  if (e != cudaSuccess) return e;
  return go(nblocks);
}

cudaError_t launch_gas_range(const LwBatch& b, const float* T, long long c0, long long c1, cudaStream_t st) {
  const void* fn = (const void*)gb::lw_gas_kernel<gb::GAS_NT>;
  const size_t smem = gb::ARGS_BYTES + gb::gas_smem_bytes(b.nsmax);
  int per = 0;
  cudaError_t e = occupancy(fn, gb::GAS_NT, smem, &per);
  if (e != cudaSuccess) return e;
  long long nb = (long long)device_sms() * (per < 1 ? 1 : per);
  if (nb > c1 - c0) nb = c1 - c0;
  if (nb < 1) return cudaSuccess;
  return launch_resident(fn, gb::GAS_NT, smem, (int)nb, [&](int n) {
    gb::lw_gas_kernel<gb::GAS_NT><<<n, gb::GAS_NT, smem, st>>>(b, T, c0, c1);
    return cudaGetLastError();
  });
}

}  // namespace

int gb_lw_num_variants() { return kNumVariants; }

LwVariant gb_lw_variant(int v, bool lean) {
  if (v < 0 || v >= kNumVariants) return LwVariant{0, 0};
  return LwVariant{gb::RT_NT, info(v, lean).max_units};
}

size_t gb_lw_smem_bytes(int nlay) { return std::max(block_smem(nlay, 1, 1), list_smem(nlay)); }

cudaError_t gb_lw_set_tables(const GbTables& T) {
  const cudaError_t e = cudaMemcpyToSymbol(gb::c_T, &T, sizeof(GbTables));
  return e == cudaSuccess ? gb_lw_taumol_set_tables(T) : e;
}

namespace {
// Columns per unit: two, a thread per pair of g-points (80 a column), where
// two columns fit in a block's shared memory (up to 229 layers; 3,000 columns of 227
// layers with maximum/random overlap take 3.00 ms so, 4.69 ms one by one), and where the batch has more
// columns than the device has SMs: of fewer, each gets an SM to itself.
int cols_per_unit(int nlay, long long ncols) {
  return ncols > device_sms() && block_smem(nlay, 2, 1) <= device_smem() ? 2 : 1;
}
int unit_threads(int cpb) { return cpb == 2 ? gb::RT_NT : (gb::RT_CT + 31) / 32 * 32; }
int units_per_sm(int nlay, int cpb, const VariantInfo& v) {
  int n = v.max_units;
  while (n > 1 && block_smem(nlay, cpb, n) > device_smem()) --n;
  return n;
}
}  // namespace

// Four units where their shared memory fits (96 registers a thread), else
// three with 128: at 60 layers three fit, and 32,768 columns of the learned
// path take 3.65 ms with 128 registers, 3.76 with 96 (in-kernel clouds with
// taumol 4.37 and 4.51); at 45 layers four with 96 take 4.90 ms, three with
// 128 5.12 (caller sub-columns).  Five with 72 registers spill (5.8 ms).
int gb_lw_default_variant(int nlay) {
  const int cpb = cols_per_unit(nlay, LLONG_MAX);
  for (int v : {0, 1, 3})
    if (units_per_sm(nlay, cpb, kVariants[v]) == kVariants[v].max_units) return v;
  return 3;
}

int gb_lw_slots(int nlay, int variant, bool lean) {
  if (variant < 0 || variant >= kNumVariants) variant = 0;
  return device_sms() * units_per_sm(nlay, cols_per_unit(nlay, LLONG_MAX), info(variant, lean));
}

namespace {
// plane bytes of one column slot: its rows, setcoef's words, laytrop
size_t slot_bytes(int nlay) { return (size_t)nlay * (GB_LW_PROW + GB_LW_COEF_WORDS) * 4 + sizeof(int); }
// ... and of a batch with caller sub-columns: the cells' values and bits, the stop code
size_t cell_bytes(int nlay) { return (size_t)nlay * (GB_NGPT + GB_LW_CELL_WORDS) * 4 + sizeof(int); }
bool has_cells(const LwBatch& b) {
  bool any = false;
  for (int i = 0; i < b.ngrid; ++i) {
    if (b.g[i].sur_flag) return false;  // learned gas optics take their cells in the transfer kernel
    any |= b.g[i].cloud_mode == LW_CLOUD_SUBCOL && b.g[i].icld >= 1;
  }
  return any;
}
// per resident column: the cloud plane of caller sub-columns, the level sums
size_t resident_cols() { return (size_t)device_sms() * kMaxPerSm * 2; }
size_t resident_bytes(int nlay) {
  return resident_cols() * ((size_t)nlay * GB_NGPT + gb::rt_part_floats(nlay)) * sizeof(float);
}
size_t round_slots(size_t n) { return (n + 31) & ~size_t(31); }
// a pass's planes: enough columns that the tail of a pass is small beside it
// (a wave of the transfer is about 1,200 columns), few enough that the buffer
// stays small beside the batch's own arrays
constexpr size_t kPlaneBytes = size_t(1536) << 20;
}  // namespace

size_t gb_lw_gas_min_bytes(int nlay) {
  return resident_bytes(nlay) + round_slots((size_t)gb_lw_list_slots()) * slot_bytes(nlay);
}

size_t gb_lw_gas_bytes(const LwBatch& b, bool learned) {
  const size_t per = slot_bytes(b.nsmax) + (has_cells(b) ? cell_bytes(b.nsmax) : 0);
  const size_t room = std::max<size_t>(kPlaneBytes / per & ~size_t(31), 32);
  const size_t want = learned ? 0 : round_slots((size_t)b.col0[b.ngrid] + GB_LW_MAX_GRIDS);  // a column may be missing per grid
  return std::max(resident_bytes(b.nsmax) + std::min(want, room) * per, gb_lw_gas_min_bytes(b.nsmax));
}

void gb_lw_attach_gas(LwBatch& b, void* buf, size_t bytes) {
  const size_t res = resident_bytes(b.nsmax);
  const bool cells = has_cells(b);
  const size_t per = slot_bytes(b.nsmax) + (cells ? cell_bytes(b.nsmax) : 0);
  b.rcols = (long long)resident_cols();
  b.pslots = bytes > res ? (long long)((bytes - res) / per & ~size_t(31)) : 0;
  const size_t rows = (size_t)b.pslots * b.nsmax;
  b.plane = static_cast<float*>(buf);  // the rows first: each on a 32-byte boundary
  b.coef = b.plane + rows * GB_LW_PROW;
  b.gcld = b.coef + rows * GB_LW_COEF_WORDS;
  b.part = b.gcld + std::max(cells ? rows : 0, (size_t)b.rcols * b.nsmax) * GB_NGPT;
  b.laytrop = reinterpret_cast<int*>(b.part + (size_t)b.rcols * gb::rt_part_floats(b.nsmax));
  b.cellerr = cells ? b.laytrop + b.pslots : nullptr;
  b.cellw = cells ? reinterpret_cast<unsigned*>(b.cellerr + b.pslots) : nullptr;
}

long long gb_lw_list_slots() { return (long long)device_sms() * gb::LIST_PER_SM; }

cudaError_t gb_lw_launch_gas(const LwBatch& b, const float* d_tables, long long c0, long long c1,
                             cudaStream_t stream) {
  if (c1 <= c0) return cudaSuccess;
  if (c1 - c0 > b.gslots || !b.gtau || !b.gfrac) return cudaErrorInvalidValue;
  return launch_gas_range(b, d_tables, c0, c1, stream);
}

cudaError_t gb_lw_launch_batch(const LwBatch& bin, const float* d_tables, int variant, int nblocks,
                               cudaStream_t stream) {
  LwBatch b = bin;
  if (variant < 0 || variant >= kNumVariants || b.ngrid < 1 || b.ngrid > GB_LW_MAX_GRIDS) return cudaErrorInvalidValue;
  const long long n = b.col0[b.ngrid];
  if (n <= 0 || nblocks <= 0) return cudaSuccess;
  if (!b.plane || b.pslots < 32) return cudaErrorInvalidValue;
  b.cpb = cols_per_unit(b.nsmax, n);
  b.unit0[0] = 0;
  for (int i = 0; i < b.ngrid; ++i) b.unit0[i + 1] = b.unit0[i] + (b.col0[i + 1] - b.col0[i] + b.cpb - 1) / b.cpb;
  const long long units = b.unit0[b.ngrid];
  for (int i = 0; i < b.ngrid; ++i)  // fused-cloud grids come with their McICA draws
    if (b.g[i].cloud_mode == LW_CLOUD_FUSED && b.g[i].icld >= 1 && b.g[i].ncol > 0 && !b.g[i].draws)
      return cudaErrorInvalidValue;
  int nband = 0;
  for (int i = 0; i < b.ngrid; ++i) {
    const LwArgs& g = b.g[i];
    if (g.cloud_mode != LW_CLOUD_BAND) continue;
    ++nband;
    if (g.icld >= 1 && g.ncol > 0 && (!g.ncbands || !g.cldfrac || !g.tauc)) return cudaErrorInvalidValue;
  }
  // nblocks units, over the SMs: nunit of them in a block, a block per SM
  const int nsm = device_sms();
  auto transfer = [&](const VariantInfo& v, long long u0, long long u1) -> cudaError_t {
    const long long want = std::min<long long>(nblocks, std::min(u1 - u0, b.rcols / b.cpb));
    const int nunit = (int)std::min<long long>((want + nsm - 1) / nsm, units_per_sm(b.nsmax, b.cpb, v));
    const int blocks = (int)std::min<long long>((want + nunit - 1) / nunit, nsm);
    const size_t smem = block_smem(b.nsmax, b.cpb, nunit);
    const cudaError_t e = gb_allow_smem(v.fn);
    if (e != cudaSuccess) return e;
    return v.launch(b, d_tables, u0, u1, blocks, nunit * unit_threads(b.cpb), nunit, smem, stream);
  };
  if (!b.fall || !b.nfall) {
    // pass by pass: taumol into the planes, caller sub-columns' cells, then the transfer
    for (int i = 0; i < b.ngrid; ++i)
      if (b.g[i].cloud_mode == LW_CLOUD_SUBCOL && b.g[i].icld >= 1 && !b.cellw) return cudaErrorInvalidValue;
    if (nband && nband != b.ngrid) return cudaErrorInvalidValue;  // band clouds: every grid in that mode
    const long long room = b.pslots / b.cpb, passes = (units + room - 1) / room, step = (units + passes - 1) / passes;
    for (long long u0 = 0; u0 < units; u0 += step) {
      const long long u1 = std::min(u0 + step, units);
      cudaError_t e = gb_lw_launch_taumol(b, d_tables, u0, u1, stream);
      if (e == cudaSuccess && b.cellw) {
        const size_t smem = gb::rt_smem_bytes(b.nsmax);
        e = gb_allow_smem((const void*)gb::lw_cells_kernel);
        if (e != cudaSuccess) return e;
        gb::lw_cells_kernel<<<(unsigned)((u1 - u0) * b.cpb), gb::CELL_NT, smem, stream>>>(b, d_tables, u0);
        e = cudaGetLastError();
      }
      if (e == cudaSuccess) e = transfer(nband ? kBand : info(variant, false), u0, u1);
      if (e != cudaSuccess) return e;
    }
    return cudaSuccess;
  }
  // learned gas optics: the transfer kernel on the network's outputs, then the
  // hand-over kernel over the columns it passed on (its blocks find an empty
  // list and return when every column was on the network)
  if (nband || b.pslots < gb_lw_list_slots() || b.rcols < gb_lw_list_slots()) return cudaErrorInvalidValue;
  cudaError_t e = cudaMemsetAsync(b.nfall, 0, sizeof(unsigned), stream);
  if (e != cudaSuccess) return e;
  bool odd = false;  // network rows (280 bytes) that do not start on 4-byte boundaries
  for (int i = 0; i < b.ngrid; ++i) odd |= (((uintptr_t)b.g[i].sur_tau | (uintptr_t)b.g[i].sur_frac) & 3) != 0;
  e = transfer(odd ? kOdd : info(variant, true), 0, units);
  if (e != cudaSuccess) return e;
  const void* fn = (const void*)gb::lw_list_kernel;
  const size_t lsmem = list_smem(b.nsmax);
  return launch_resident(fn, gb::RT_NT, lsmem, (int)gb_lw_list_slots(), [&](int nb) {
    gb::lw_list_kernel<<<nb, gb::RT_NT, lsmem, stream>>>(b, d_tables);
    return cudaGetLastError();
  });
}
