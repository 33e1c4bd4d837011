// taumol for many columns at once (rrtmg_lw_setcoef.f90, rrtmg_lw_taumol.f90):
// two kernels that fill the gas-optics planes the transfer kernel reads.
//
//   lw_setcoef_kernel -- one warp per (32 columns, layer): inatm's column
//     amounts and setcoef's interpolation factors and indices, and each
//     column's laytrop.  A (32 columns, layer) tile is one contiguous run of
//     CW words per lane, so that the taumol kernel's reads are coalesced and
//     at constant offsets.
//   lw_taumol_kernel -- one thread per (column, layer) of one band, the 32
//     lanes of a warp being neighbouring columns of one layer: the band's
//     term list (lw_gasoptics.cuh) stays in registers, and the band's
//     g-points are swept four at a time, every term one 16-byte load of a
//     table row.  Neighbouring columns share most of their rows (pressures
//     alike, temperatures within a table step), so a warp's load touches a few
//     rows, where a warp spread over one layer's g-points loads four bytes a
//     lane and reads each term's weight and row from shared memory first.
//     A block works on one band, and the bands of a run of columns follow one
//     another, so that a band's code and tables stay in the SM's caches and
//     the run's setcoef words in L2.
//
// What bounds the taumol kernel is the latency and the width of its table loads
// (a warp's 16-byte load fills registers for four cycles, 2,220 multiply-adds per column
// and layer, and the L1 pipe is three quarters busy): with 64 registers a thread and 8
// blocks per SM 16,384 columns of 60 layers take 0.2 ms less than with 128 and 4
// (transfer included 2.14 ms, now 1.94 ms; 9 or 10 blocks spill more than they
// hide), of it 0.04 ms from runs of 304 blocks (two per SM) in place of 1,216;
// with runs of 152 the last wave of each band shows (1.99 ms).
// Compiled without multiply-add contraction: the prologues and the order of
// every sum are those of the in-block taumol of lw_solver.cu, bit for bit.
#include <cuda_runtime.h>
#include <math.h>
#include <stdint.h>

#include "lw_common.h"
#include "lw_solver.h"
#include "lw_gasoptics.cuh"

namespace gb {

constexpr int CW = NF + 1;       // words per (column, layer): the LayerFields, the packed indices
constexpr int TILE = 32;         // columns per tile: one per lane
constexpr int SET_NT = 256;      // setcoef kernel: eight warps, one tile, layers dealt to the warps
constexpr int TAU_NT = 128;      // taumol kernel: four (tile, layer) units per block
constexpr int TAU_RUN = 304;     // blocks of one band before the next band of the same columns

static_assert(GB_LW_COEF_WORDS == CW, "setcoef words per column and layer");

// setcoef's words of one (column, layer), in global memory
struct CoefCell {
  const float* w;  // word k of this lane at w[k * TILE]
  int lay;
  const float* T;
  const LwArgs* a;
  long long icol;
  int ints;
  __device__ __forceinline__ float F(int k) const { return __ldg(w + k * TILE); }
  __device__ __forceinline__ int I(int k) const {
    return k == I_JP ? ints & 63 : k == I_JT ? (ints >> 6) & 7 : k == I_JT1 ? (ints >> 9) & 7
         : k == I_INDSELF ? (ints >> 12) & 15 : k == I_INDFOR ? (ints >> 16) & 3 : (ints >> 18) & 31;
  }
  __device__ __forceinline__ double D(int k) const { return amount64(*a, icol, lay, k); }
  __device__ __forceinline__ Amt A(int field) const { return Amt{F(field), amount_of(field)}; }
};
__device__ __forceinline__ int pack_ints(const LayerInts& x) {
  return x.jp | (x.jt << 6) | (x.jt1 << 9) | (x.indself << 12) | (x.indfor << 16) | (x.indminor << 18);
}

// a term list in registers (every index a compile-time constant once inlined)
struct RegTerms {
  float w[MAXT_ALL];
  int off[MAXT_ALL];
  int n = 0;
  __device__ __forceinline__ void add(float wt, int o) {
    w[n] = wt;
    off[n] = o;
    ++n;
  }
  __device__ __forceinline__ void scale(float s) {
#pragma unroll
    for (int k = 0; k < MAXT_ALL; ++k)
      if (k < n) w[k] *= s;
  }
};

__global__ void __launch_bounds__(SET_NT) lw_setcoef_kernel(const __grid_constant__ LwBatch B,
                                                            const float* __restrict__ T, long long u0, long long nslot) {
  __shared__ int lt[TILE];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const long long slot = (long long)blockIdx.x * TILE + lane;
  if (threadIdx.x < TILE) lt[threadIdx.x] = 0;
  __syncthreads();
  if (slot < nslot) {
    long long icol;
    const LwArgs& a = B.g[slot_column(B, u0, slot, icol)];
    if (icol < a.ncol) {
      for (int lay = warp; lay < a.nlay; lay += SET_NT / 32) {
        float* w = B.coef + ((long long)blockIdx.x * B.nsmax + lay) * (CW * TILE) + lane;
        LayerInts ix;
        const bool lower = setcoef_layer(a, icol, lay, T, ix, [&](int k, float v) { w[k * TILE] = v; });
        w[NF * TILE] = __int_as_float(pack_ints(ix));
        if (lower) atomicAdd(&lt[lane], 1);  // laytrop (the transfer checks that these form a prefix)
      }
    }
  }
  __syncthreads();
  if (threadIdx.x < TILE && slot < nslot) B.laytrop[slot] = lt[threadIdx.x];
}

__device__ __forceinline__ float4 ldg4(const float* p) { return __ldg(reinterpret_cast<const float4*>(p)); }
// 32 bytes in one store (both on a 32-byte boundary)
__device__ __forceinline__ void store8(float* p, float4 a, float4 b) {
  asm volatile("st.global.v8.f32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"l"(p), "f"(a.x), "f"(a.y), "f"(a.z),
               "f"(a.w), "f"(b.x), "f"(b.y), "f"(b.z), "f"(b.w)
               : "memory");
}

// band b of one (column, layer): row is the layer's row of the plane
template <int b, bool LOWER>
__device__ __forceinline__ void taumol_cell(const CoefCell& c, float* row) {
  constexpr int NG = ngb_const(b), P = pitch_const(b);
  RegTerms t;
  const FracRec fr = Band<b>::prologue(c, LOWER, t);
  const float* __restrict__ T = c.T;
  float* out = row + 4 * gb_pair0(b);
  if constexpr (NG == 2) {
    float2 acc = make_float2(0.0f, 0.0f);
#pragma unroll
    for (int k = 0; k < MAXT_ALL; ++k)
      if (k < t.n) {
        const float2 v = __ldg(reinterpret_cast<const float2*>(T + t.off[k]));
        acc.x = fmaf(t.w[k], v.x, acc.x);
        acc.y = fmaf(t.w[k], v.y, acc.y);
      }
    const float2 f0 = __ldg(reinterpret_cast<const float2*>(T + fr.off));
    const float2 f1 = __ldg(reinterpret_cast<const float2*>(T + fr.off + P));
    *reinterpret_cast<float4*>(out) =
        make_float4(acc.x, acc.y, fmaf(fr.fpl, f1.x - f0.x, f0.x), fmaf(fr.fpl, f1.y - f0.y, f0.y));
  } else {
#pragma unroll 1
    for (int q = 0; q < P / 4; ++q) {
      float4 acc = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
      const float* Tq = T + 4 * q;
#pragma unroll
      for (int k = 0; k < MAXT_ALL; ++k)
        if (k < t.n) {
          const float4 v = ldg4(Tq + t.off[k]);
          acc.x = fmaf(t.w[k], v.x, acc.x);
          acc.y = fmaf(t.w[k], v.y, acc.y);
          acc.z = fmaf(t.w[k], v.z, acc.z);
          acc.w = fmaf(t.w[k], v.w, acc.w);
        }
      if ((b == 4 || b == 7) && !LOWER) {
        acc.x *= gscale(b, 4 * q);
        acc.y *= gscale(b, 4 * q + 1);
        acc.z *= gscale(b, 4 * q + 2);
        acc.w *= gscale(b, 4 * q + 3);
      }
      const float4 f0 = ldg4(Tq + fr.off), f1 = ldg4(Tq + fr.off + P);
      // the pairs past the band's g-points (rows are padded) land in the plane's padding
      store8(out + 8 * q,
             make_float4(acc.x, acc.y, fmaf(fr.fpl, f1.x - f0.x, f0.x), fmaf(fr.fpl, f1.y - f0.y, f0.y)),
             make_float4(acc.z, acc.w, fmaf(fr.fpl, f1.z - f0.z, f0.z), fmaf(fr.fpl, f1.w - f0.w, f0.w)));
    }
  }
}

__constant__ unsigned char c_order[16] = {5, 3, 13, 9, 7, 4, 8, 12, 15, 16, 6, 1, 11, 2, 10, 14};  // longest first

// PER_SM: blocks an SM the register allocation is sized for
template <int PER_SM>
__global__ void __launch_bounds__(TAU_NT, PER_SM) lw_taumol_kernel(const __grid_constant__ LwBatch B,
                                                              const float* __restrict__ T, long long u0,
                                                              long long nslot, int nblk) {
  // block -> (run of column blocks, band, block within the run)
  const int run = blockIdx.x / (TAU_RUN * 16);
  const int left = nblk - run * TAU_RUN, cnt = left < TAU_RUN ? left : TAU_RUN;
  const int rem = blockIdx.x - run * (TAU_RUN * 16);
  const int band = c_order[rem / cnt];
  const long long unit = (long long)(run * TAU_RUN + rem % cnt) * (TAU_NT / 32) + (threadIdx.x >> 5);
  const int lane = threadIdx.x & 31;
  const long long tile = unit / B.nsmax;
  const int lay = (int)(unit - tile * B.nsmax);
  const long long slot = tile * TILE + lane;
  if (slot >= nslot) return;
  long long icol;
  const LwArgs& a = B.g[slot_column(B, u0, slot, icol)];
  if (icol >= a.ncol || lay >= a.nlay) return;
  const float* w = B.coef + unit * (CW * TILE) + lane;
  const CoefCell c{w, lay, T, &a, icol, __float_as_int(__ldg(w + NF * TILE))};
  const bool lower = lay < __ldg(B.laytrop + slot);
  float* row = B.plane + (slot * B.nsmax + lay) * GB_LW_PROW;
#define GB_BAND(b)                   \
  case b:                            \
    if (lower)                       \
      taumol_cell<b, true>(c, row);  \
    else                             \
      taumol_cell<b, false>(c, row); \
    break;
  switch (band) {
    GB_BAND(1) GB_BAND(2) GB_BAND(3) GB_BAND(4) GB_BAND(5) GB_BAND(6) GB_BAND(7) GB_BAND(8)
    GB_BAND(9) GB_BAND(10) GB_BAND(11) GB_BAND(12) GB_BAND(13) GB_BAND(14) GB_BAND(15) GB_BAND(16)
  }
#undef GB_BAND
}

}  // namespace gb

cudaError_t gb_lw_taumol_set_tables(const GbTables& T) { return cudaMemcpyToSymbol(gb::c_T, &T, sizeof(GbTables)); }

cudaError_t gb_lw_launch_taumol(const LwBatch& b, const float* d_tables, long long u0, long long u1,
                                cudaStream_t stream) {
  const long long nslot = (u1 - u0) * b.cpb;
  if (nslot <= 0) return cudaSuccess;
  if (!b.plane || !b.coef || !b.laytrop || nslot > b.pslots) return cudaErrorInvalidValue;
  const long long tiles = (nslot + gb::TILE - 1) / gb::TILE;
  gb::lw_setcoef_kernel<<<(unsigned)tiles, gb::SET_NT, 0, stream>>>(b, d_tables, u0, nslot);
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return e;
  const int per = gb::TAU_NT / 32;
  const int nblk = (int)((tiles * b.nsmax + per - 1) / per);
  int dev = 0, nsm = 1;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
  // where every block is resident at four an SM, the more loads a warp has in
  // flight at 128 registers count, not the warps (calls of 1x38, 32x60, 64x38, 96x45
  // and 128x38 columns and layers: 72.0, 97.6, 84.0, 92.3 and 84.2 us at 64 registers,
  // 69.8, 94.6, 80.1, 90.3 and 82.1 at 128; 16x45 83.2 either way)
  if (nblk * 16LL <= 4LL * nsm)
    gb::lw_taumol_kernel<4><<<(unsigned)nblk * 16u, gb::TAU_NT, 0, stream>>>(b, d_tables, u0, nslot, nblk);
  else
    gb::lw_taumol_kernel<8><<<(unsigned)nblk * 16u, gb::TAU_NT, 0, stream>>>(b, d_tables, u0, nslot, nblk);
  return cudaGetLastError();
}
