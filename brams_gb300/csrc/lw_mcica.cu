// McICA sub-column generator on the GPU (mcica_subcol_gen_lw.f90:183-703,
// mcica_random_numbers.f90:77-306).
//
// The reference draws every random number from one Mersenne-twister (irng=1)
// or KISS (irng=0) sequence in a fixed loop order and marks sub-column isub
// of layer ilev cloudy when CDF >= 1 - cldf (:650).  The GPU reproduces the
// draws bit for bit:
//   * draw generation -- per column for per-column seeds (the reference called
//     with ncol = 1 and seed = base + column), or one block stepping the single
//     sequence 624 words at a time for the reference's all-columns call (draw
//     order isub, column, layer);
//   * CDF construction and the cloudy test in double precision, a thread per
//     column and pair of sub-columns, layers in order (max-random and
//     exponential overlap carry CDF from one layer to the next).
// Draws are kept as doubles exactly as getRandomReal/kissvec return them.
#include <cuda_runtime.h>
#include <limits.h>
#include <stdint.h>

#include <mutex>

#include "../../include/gb_rrtmg_lw.h"
#include "lw_common.h"
#include "lw_mcica.h"
#include "lw_mt.cuh"

namespace gbm {

// ---------------------------------------------------------------- Mersenne twister
using gbmt::temper;
using gbmt::real;
__device__ __forceinline__ uint32_t mt_temper(uint32_t y) { return gbmt::temper(y); }
__device__ __forceinline__ uint32_t mt_twist(uint32_t u, uint32_t v) { return gbmt::twist(u, v); }
__device__ __forceinline__ double mt_real(uint32_t u) { return gbmt::real(u); }

// The first n outputs of per-column seeds (column c: seed0 + c), draws[c * n + k].
// They need the initial state's words 0..n and 397..396+n only (nextState's
// first loop; n <= 227).  A block has 32 columns: a lane of its first warp walks a
// column's initialisation, a chain of 536 dependent steps, and leaves those
// words in shared memory; all threads then temper them and write the rows.
// The chain bounds it (some 4 us).  One thread per column for both parts took 54 us
// for 8,192 columns, most of it in fp64 divisions, which also issue one by one
// (a solver call of 64 columns, draws included: 122 us, now 80 us).
constexpr int MT_NT = 256;
constexpr int MT_MAX = 181;  // (2 n + 1) words of 33 columns in 48 KB
__global__ void __launch_bounds__(MT_NT) mt_percol_kernel(int ncol, uint32_t seed0, int n, double* __restrict__ draws) {
  extern __shared__ uint32_t word[];  // [2 n + 1][33]
  const long long c0 = blockIdx.x * 32LL;
  if (threadIdx.x < 32) {
    uint32_t s = seed0 + (uint32_t)c0 + threadIdx.x;
    uint32_t* w = word + threadIdx.x;
    w[0] = s;
    auto next = [&](int i) { s = 1812433253u * (s ^ (s >> 30)) + (uint32_t)i; };
#pragma unroll 8
    for (int i = 1; i <= n; ++i) {
      next(i);
      w[33 * i] = s;
    }
#pragma unroll 8
    for (int i = n + 1; i < 397; ++i) next(i);
    w += 33 * (n + 1);
#pragma unroll 8
    for (int k = 0; k < n; ++k) {
      next(397 + k);
      w[33 * k] = s;
    }
  }
  __syncthreads();
  const int nc = (int)min(32LL, ncol - c0);
  double* out = draws + c0 * n;
  for (int i = threadIdx.x; i < nc * n; i += MT_NT) {
    const int c = i / n, k = i - c * n;
    const uint32_t* w = word + c + 33 * k;
    out[i] = mt_real(mt_temper(w[33 * (n + 1)] ^ mt_twist(w[0], w[33])));
  }
}

// One sequence per block, seeded with seed0 + block: a block keeps the 624-word
// state in shared memory and produces it one twist (624 draws) at a time.  One
// block for the reference's own call, else a block per column.
__global__ void __launch_bounds__(256) mt_stream_kernel(uint32_t seed0, long long ndraw, double* __restrict__ draws) {
  __shared__ uint32_t st[624];
  __shared__ uint32_t nw[624];
  if (threadIdx.x == 0) {
    uint32_t s = seed0 + blockIdx.x;
    st[0] = s;
#pragma unroll 7
    for (int i = 1; i < 624; ++i) {
      s = 1812433253u * (s ^ (s >> 30)) + (uint32_t)i;
      st[i] = s;
    }
  }
  __syncthreads();
  draws += blockIdx.x * ndraw;
  for (long long base = 0; base < ndraw; base += 624) {
    // nextState (:127-139): words 0..226 from old words, 227..622 from new 0..395, 623 from new 396 and new 0
    for (int k = threadIdx.x; k < 227; k += blockDim.x) nw[k] = st[k + 397] ^ mt_twist(st[k], st[k + 1]);
    __syncthreads();
    for (int k = 227 + threadIdx.x; k < 454; k += blockDim.x) nw[k] = nw[k - 227] ^ mt_twist(st[k], st[k + 1]);
    __syncthreads();
    for (int k = 454 + threadIdx.x; k < 623; k += blockDim.x) nw[k] = nw[k - 227] ^ mt_twist(st[k], st[k + 1]);
    __syncthreads();
    if (threadIdx.x == 0) nw[623] = nw[396] ^ mt_twist(st[623], nw[0]);
    __syncthreads();
    for (int k = threadIdx.x; k < 624; k += blockDim.x) {
      st[k] = nw[k];
      long long d = base + k;
      if (d < ndraw) draws[d] = mt_real(mt_temper(nw[k]));
    }
    __syncthreads();
  }
}

// ---------------------------------------------------------------- KISS (irng = 0)
struct Kiss {
  uint32_t s1, s2, s3, s4;
  __device__ double next() {
    s1 = 69069u * s1 + 1327217885u;
    uint32_t k = s2;
    k ^= k << 13;
    k ^= k >> 17;
    k ^= k << 5;
    s2 = k;
    s3 = 18000u * (s3 & 65535u) + (s3 >> 16);
    s4 = 30903u * (s4 & 65535u) + (s4 >> 16);
    int32_t kiss = (int32_t)(s1 + s2 + (s3 << 16) + s4);
    return (double)kiss * 2.328306e-10 + 0.5;
  }
};

// kissvec seeds from the fractional part of the bottom four layer pressures
// (:460-474), warmed up changeSeed times; then the column's own sequence.
// skip_per_draw > 0 reproduces icld 4/5, where every kissvec call of the
// reference advances all columns although only column c's value is kept.
__global__ void kiss_percol_kernel(int ncol, long long ld, const double* __restrict__ play, int change_seed,
                                   int seed_step, int ndraw, int ncol_call, int nsub, int* __restrict__ err,
                                   double* __restrict__ draws) {
  int c = blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= ncol) return;
  double p[4];
  for (int l = 0; l < 4; ++l) p[l] = play[c + ld * l] * 1.e2;
  if (p[0] < p[1]) {
    // the reference stops here (status 8); the column's draws are set to 0 so
    // that its sub-columns are the same on every call, not the previous
    // contents of the draw buffer
    atomicMax(err, 8);
    for (int d = 0; d < ndraw; ++d) draws[(long long)c * ndraw + d] = 0.0;
    return;
  }
  Kiss k;
  auto sd = [](double x) { return (uint32_t)(int32_t)((x - (double)(long long)x) * 1000000000.0); };
  k.s1 = sd(p[0]); k.s2 = sd(p[1]); k.s3 = sd(p[2]); k.s4 = sd(p[3]);
  const int warm = change_seed + seed_step * c;
  for (int i = 0; i < warm; ++i) k.next();
  double* out = draws + (long long)c * ndraw;
  if (ncol_call <= 1) {
    for (int d = 0; d < ndraw; ++d) out[d] = k.next();
  } else {
    // icld 4/5 in one call over ncol_call columns: pairs of draws per
    // (isub, column, layer), each advancing every column; keep column c's
    int nlay_pairs = ndraw / 2 / nsub;  // = nlay
    int col_in_call = c % ncol_call;
    int d = 0;
    for (int isub = 0; isub < nsub; ++isub)
      for (int i = 0; i < ncol_call; ++i)
        for (int l = 0; l < nlay_pairs; ++l) {
          double a = k.next(), b = k.next();
          if (i == col_in_call) {
            out[d++] = a;
            out[d++] = b;
          }
        }
  }
}

// ---------------------------------------------------------------- CDF + outputs
// A block has FILL_C neighbouring columns, whose rows lie side by side in the
// outputs, and a thread one of their pairs of sub-columns; the layers come in
// chunks of FILL_L, whose thresholds, water paths and optical properties are
// staged in shared memory.  `D(ilev, which)` locates the draw the reference would
// use for a cell.  What bounds it is the write of the sub-column arrays.  The
// random draws are in [0, 1], so cdf >= 1 - cldf is a comparison of the bit
// patterns as integers, a negative threshold takes every cell and a NaN none: a
// double comparison, difference and maximum at 1/64 of the integer rate per cell kept
// the fp64 pipe half busy (36,000 columns of 45 layers, draws included: 2.54 ms,
// now 1.22 ms; the writes are 7.3 GB).
constexpr int FILL_C = 4, FILL_L = 16;
struct FillCell {
  long long key;  // 1 - cldf for the integer comparison
  double omc;     // 1 - cldf
  double clwp, ciwp;
};

template <bool RANDOM_MAX>  // icld 3: the same draw in all layers
__global__ void __launch_bounds__(FILL_C * 70) mcica_fill_kernel(McicaArgs a, const double* __restrict__ draws, bool wide) {
  __shared__ FillCell cells[FILL_L][FILL_C];
  extern __shared__ double optics[];  // [1 or 4: tauc, ssac, asmc, fsfc][FILL_L][FILL_C][nbnd]
  const int np = a.nsub / 2, nt = FILL_C * np, tid = threadIdx.x;
  const int cc = tid / np, isub = 2 * (tid - cc * np);
  const long long c0 = (long long)blockIdx.x * FILL_C;
  const int nc = (int)min((long long)FILL_C, a.ncol - c0);
  const bool on = cc < nc;
  const long long c = c0 + (on ? cc : 0);
  const int nlay = a.nlay, nbnd = a.nbnd;
  const long long ld = a.ld;
  const bool sw = a.ssacmcl != nullptr;
  auto D = [&](int is, int ilev, int which) -> double {
    long long idx;
    if (a.mode == MCICA_STREAM_MT) {
      // one sequence over the call: loop order isub, column, layer (:476-645)
      long long ncol = a.ncol;
      if (RANDOM_MAX) idx = (long long)is * ncol + c;
      else if (a.icld <= 2) idx = ((long long)is * ncol + c) * nlay + ilev;
      else idx = 2 * (((long long)is * ncol + c) * nlay + ilev) + which;
      return draws[idx];
    }
    // per-column sequences (MT with per-column seeds, or KISS)
    long long base = c * a.ndraw_per_col;
    if (RANDOM_MAX) idx = is;
    else if (a.icld <= 2) idx = (long long)is * nlay + ilev;
    else idx = 2 * ((long long)is * nlay + ilev) + which;
    return draws[base + idx];
  };
  // the band of the sub-column's optical properties (mcica_subcol_gen_sw.f90:
  // n = ngb(isubcol) - ngbm; the longwave one uses ngb itself)
  const int b0 = a.ngb[isub] - a.band0 - 1, b1 = a.ngb[isub + 1] - a.band0 - 1;
  double cdf[2] = {0.0, 0.0}, omp = 0.0;  // the CDF and 1 - cldf of the layer below
  if (RANDOM_MAX) cdf[0] = D(isub, 0, 0), cdf[1] = D(isub + 1, 0, 0);
  const long long row = a.nsub * ld;  // of a layer
  long long o = isub + a.nsub * c;
  const int nopt = FILL_L * FILL_C * nbnd;
  for (int l0 = 0; l0 < nlay; l0 += FILL_L) {
    const int n = min(FILL_L, nlay - l0);
    __syncthreads();
    for (int i = tid; i < n * FILL_C; i += nt) {
      const int l = i / FILL_C, k = i % FILL_C;
      if (k >= nc) continue;
      const long long oc = c0 + k + ld * (l0 + l);
      const double v = a.cldfrac[oc], omc = 1.0 - (v < 1.0e-20 ? 0.0 : v);
      FillCell& f = cells[l][k];
      f.key = omc < 0.0 ? LLONG_MIN : (omc == omc ? __double_as_longlong(omc) : LLONG_MAX);
      f.omc = omc;
      f.clwp = a.clwp[oc];
      f.ciwp = a.ciwp[oc];
      a.reicmcl[oc] = a.rei[oc];  // reicmcl / relqmcl copies (:264-265)
      a.relqmcl[oc] = a.rel[oc];
    }
    for (int i = tid; i < n * nc * nbnd; i += nt) {
      const int l = i / (nc * nbnd), r = i - l * (nc * nbnd);  // r: column and band
      const long long ob = r + nbnd * (c0 + ld * (l0 + l));
      double* d = optics + l * (FILL_C * nbnd) + r;
      d[0] = a.tauc[ob];
      if (sw) d[nopt] = a.ssac[ob], d[2 * nopt] = a.asmc[ob], d[3 * nopt] = a.fsfc[ob];
    }
    __syncthreads();
    if (!on) continue;
#pragma unroll 4
    for (int l = 0; l < n; ++l, o += row) {
      const FillCell& f = cells[l][cc];
      bool y[2];
      if (RANDOM_MAX) {
        y[0] = __double_as_longlong(cdf[0]) >= f.key, y[1] = __double_as_longlong(cdf[1]) >= f.key;
      } else {
        const int ilev = l0 + l;
#pragma unroll
        for (int q = 0; q < 2; ++q) {
          double v = D(isub + q, ilev, 0);
          if (a.icld <= 2) {
            if (a.icld == 2 && ilev > 0) v = (cdf[q] > omp) ? cdf[q] : v * omp;  // :528-537
          } else {
            const double v2 = D(isub + q, ilev, 1);
            if (ilev > 0 && v2 < a.alpha[c + ld * ilev]) v = cdf[q];  // :626-630, 639-643
          }
          cdf[q] = v;
          y[q] = v >= f.omc;
        }
        omp = f.omc;
      }
      auto put = [&](double* p, double v0, double v1) {
        if (wide) {
          *reinterpret_cast<double2*>(p + o) = make_double2(v0, v1);
        } else {
          p[o] = v0;
          p[o + 1] = v1;
        }
      };
      auto sel = [&](double* p, double v0, double v1, double off) { put(p, y[0] ? v0 : off, y[1] ? v1 : off); };
      const double *t0 = optics + (l * FILL_C + cc) * nbnd + b0, *t1 = t0 + (b1 - b0);
      sel(a.cldfmcl, 1.0, 1.0, 0.0);
      sel(a.clwpmcl, f.clwp, f.clwp, 0.0);
      sel(a.ciwpmcl, f.ciwp, f.ciwp, 0.0);
      sel(a.taucmcl, t0[0], t1[0], 0.0);
      if (sw) {
        sel(a.ssacmcl, t0[nopt], t1[nopt], 1.0);
        sel(a.asmcmcl, t0[2 * nopt], t1[2 * nopt], 0.0);
        sel(a.fsfcmcl, t0[3 * nopt], t1[3 * nopt], 0.0);
      }
    }
  }
}

// the Mersenne-twister draws of per-column seeds
static void percol_mt(int ncol, uint32_t seed0, int ndraw, double* draws, cudaStream_t stream) {
  if (ndraw <= MT_MAX)
    mt_percol_kernel<<<(ncol + 31) / 32, MT_NT, (2 * ndraw + 1) * 33 * sizeof(uint32_t), stream>>>(ncol, seed0, ndraw, draws);
  else
    mt_stream_kernel<<<ncol, 256, 0, stream>>>(seed0, ndraw, draws);
}

}  // namespace gbm

cudaError_t gb_mcica_launch(const McicaArgs& a, double* d_draws, int* d_err, cudaStream_t stream,
                            bool seed_per_column) {
  if (a.ncol <= 0) return cudaSuccess;
  const int per = a.icld == 3 ? 1 : (a.icld <= 2 ? a.nlay : 2 * a.nlay);
  const int ndraw = a.nsub * per;
  if (a.mode == MCICA_PERCOL_MT) {
    gbm::percol_mt(a.ncol, (uint32_t)a.seed, ndraw, d_draws, stream);
  } else if (a.mode == MCICA_STREAM_MT) {
    gbm::mt_stream_kernel<<<1, 256, 0, stream>>>((uint32_t)a.seed, (long long)ndraw * a.ncol, d_draws);
  } else {
    gbm::kiss_percol_kernel<<<(a.ncol + 127) / 128, 128, 0, stream>>>(
        a.ncol, a.ld, a.play, a.seed, seed_per_column ? 1 : 0, ndraw, a.icld >= 4 ? a.ncol_call : 1, a.nsub, d_err,
        d_draws);
  }
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return e;
  McicaArgs b = a;
  b.ndraw_per_col = ndraw;
  // 16-byte stores where the arrays start on such a boundary (rows are 1,120 or 896 bytes)
  uintptr_t at = 0;
  for (const double* p : {b.cldfmcl, b.clwpmcl, b.ciwpmcl, b.taucmcl, b.ssacmcl, b.asmcmcl, b.fsfcmcl}) at |= (uintptr_t)p;
  const unsigned blocks = (unsigned)((b.ncol + gbm::FILL_C - 1) / gbm::FILL_C), nt = gbm::FILL_C * (b.nsub / 2);
  const size_t smem = (size_t)(b.ssacmcl ? 4 : 1) * gbm::FILL_L * gbm::FILL_C * b.nbnd * sizeof(double);
  if (b.icld == 3)
    gbm::mcica_fill_kernel<true><<<blocks, nt, smem, stream>>>(b, d_draws, (at & 15) == 0);
  else
    gbm::mcica_fill_kernel<false><<<blocks, nt, smem, stream>>>(b, d_draws, (at & 15) == 0);
  return cudaGetLastError();
}

cudaError_t gb_mcica_percol_mt(int ncol, unsigned seed0, int ndraw, double* d_draws, cudaStream_t stream) {
  if (ncol <= 0) return cudaSuccess;
  gbm::percol_mt(ncol, seed0, ndraw, d_draws, stream);
  return cudaGetLastError();
}

size_t gb_mcica_draw_count(int ncol, int nlay, int icld, int nsub) {
  const int per = icld == 3 ? 1 : (icld <= 2 ? nlay : 2 * nlay);
  return (size_t)nsub * per * (size_t)ncol;
}

// ----------------------------------------------------------------------------
// Allocation-free McICA entry point.
//
// Some callers must not allocate device memory while a model runs: a host
// model whose device memory is owned by another runtime (an OpenACC or
// OpenMP-offload data region, or a pooled allocator that forbids allocations
// outside its pool), and time-stepping codes that cannot afford the implicit
// device-wide synchronisation of cudaMalloc/cudaFree in the middle of a step.
// gb_mcica_subcol_lw_noalloc serves them: its draw buffer is this fixed
// file-scope array, so a call allocates nothing.  Every GPU that loads the
// library holds the array until the process exits.
//
// Layout: the first 256 bytes hold the status word, the rest holds draws.
// All calls share the array and it keeps the previous call's contents: the
// status word is cleared at the start of every call, and every draw slot a
// call reads is written by that call first (a column whose KISS seeding
// fails gets zero draws and status 8).  Calls whose kernels overlap on
// the GPU (different streams without ordering, or several host threads)
// race on the array and must be serialised by the caller.
static __device__ __align__(256) double g_mcica_scratch[GB_MCICA_NOALLOC_STATUS_DOUBLES + GB_MCICA_NOALLOC_MAX_DRAWS];

namespace {
constexpr int kMaxDevices = 64;
std::mutex g_scratch_mutex;
double* g_scratch_ptr[kMaxDevices] = {nullptr};

// Device address of g_mcica_scratch on the current device.  In host code the
// array's name stands for a host-side shadow, not a device address, so the
// address is queried once per device (with that device current) and cached.
cudaError_t scratch_on_current_device(double** out) {
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  if (dev < 0 || dev >= kMaxDevices) return cudaErrorInvalidDevice;
  std::lock_guard<std::mutex> lock(g_scratch_mutex);
  if (!g_scratch_ptr[dev]) {
    void* p = nullptr;
    e = cudaGetSymbolAddress(&p, g_mcica_scratch);
    if (e != cudaSuccess) return e;
    g_scratch_ptr[dev] = static_cast<double*>(p);
  }
  *out = g_scratch_ptr[dev];
  return cudaSuccess;
}
}  // namespace

extern "C" int gb_mcica_subcol_lw_noalloc(void* stream, int ncol, int nlay, int icld, int permuteseed, int* irng,
                                          const double* play, const double* cldfrac, const double* ciwp,
                                          const double* clwp, const double* rei, const double* rel,
                                          const double* tauc, const double* alpha, double* cldfmcl,
                                          double* ciwpmcl, double* clwpmcl, double* reicmcl, double* relqmcl,
                                          double* taucmcl, int64_t ld, int seed_per_column, int* d_status) {
  if (!irng) return GB_LW_E_ARGS;
  if (icld == 0) return GB_LW_OK;
  if (icld < 0 || icld > 5) return GB_LW_E_ICLD;
  if (ncol < 0 || nlay < 1 || ld < ncol) return GB_LW_E_ARGS;
  if (*irng != 0) *irng = 1;
  if (icld >= 4 && !alpha) return GB_LW_E_ARGS;
  if (*irng == 0 && nlay < 4) return GB_LW_E_ARGS;
  if (!play || !cldfrac || !ciwp || !clwp || !rei || !rel || !tauc || !cldfmcl || !ciwpmcl || !clwpmcl ||
      !reicmcl || !relqmcl || !taucmcl)
    return GB_LW_E_ARGS;
  if (ncol == 0) return GB_LW_OK;
  if (gb_mcica_draw_count(ncol, nlay, icld) > (size_t)GB_MCICA_NOALLOC_MAX_DRAWS) return GB_LW_E_SCRATCH;
  double* scratch = nullptr;
  if (scratch_on_current_device(&scratch) != cudaSuccess) return GB_LW_E_CUDA;
  cudaStream_t s = (cudaStream_t)stream;
  int* status = reinterpret_cast<int*>(scratch);
  if (cudaMemsetAsync(status, 0, sizeof(int), s) != cudaSuccess) return GB_LW_E_CUDA;
  McicaArgs a{};
  a.mode = *irng == 0 ? MCICA_PERCOL_KISS : (seed_per_column ? MCICA_PERCOL_MT : MCICA_STREAM_MT);
  a.ncol = ncol;
  a.nlay = nlay;
  a.icld = icld;
  a.seed = permuteseed;
  a.ncol_call = seed_per_column ? 1 : ncol;
  a.ld = ld;
  a.play = play; a.cldfrac = cldfrac; a.ciwp = ciwp; a.clwp = clwp; a.rei = rei; a.rel = rel;
  a.tauc = tauc; a.alpha = alpha;
  a.cldfmcl = cldfmcl; a.ciwpmcl = ciwpmcl; a.clwpmcl = clwpmcl; a.taucmcl = taucmcl;
  a.reicmcl = reicmcl; a.relqmcl = relqmcl;
  // g-point -> band map (rrtmg_lw_init.f90:359-374): band b owns ng(b) consecutive g-points
  static const int ng_list[16] = GB_NG_LIST;
  for (int b = 0, g = 0; b < 16; ++b)
    for (int k = 0; k < ng_list[b]; ++k) a.ngb[g++] = b + 1;
  if (gb_mcica_launch(a, scratch + GB_MCICA_NOALLOC_STATUS_DOUBLES, status, s, seed_per_column != 0) != cudaSuccess)
    return GB_LW_E_CUDA;
  if (d_status && cudaMemcpyAsync(d_status, status, sizeof(int), cudaMemcpyDeviceToDevice, s) != cudaSuccess)
    return GB_LW_E_CUDA;
  return GB_LW_OK;
}
