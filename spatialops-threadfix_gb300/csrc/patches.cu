// Batched patches: many independent periodic heat-equation patches of uneven sizes advanced by
// ONE persistent launch per step over a device patch table, with the steps captured in a CUDA
// graph and the tile shape of each patch picked by a small autotuner.
//
// The reference advances patches one `<<=` at a time from the caller's patch loop (Uintah/
// Wasatch-style; spatialops/NeboLhs.h:29-41 launches a 16x16 grid per expression), paying a
// launch and a tail per patch and expression.  Here:
//   * all patches live in one arena per buffer, each a ghosted window, x fastest: FP64 states,
//     or FP32 states (half the bytes), or two-float states (FP32 arithmetic, ~48-bit state);
//   * a work list enumerates (patch, x-tile, y-tile, z-chunk) items; a fixed grid of blocks
//     (a multiple of the SM count) strides through it, so small and large patches share SMs;
//   * FP64 tiles hold up to 256 cells of a plane, fitted to the patch's extents (tile_shape) under a
//     width limit of 16, 32 or 64 per patch (the autotuner times each on the patches of each
//     x-extent class and keeps the fastest); FP32 items are strips of full rows;
//   * each item is the fused heat step of nebo_heat_step: face fluxes computed once, high
//     faces shared through shared memory, z-face carried in a register, and the new values
//     written to the interior and to their periodic ghost images in the same pass.
// Lambda is a scalar per patch, so each face costs (2 lambda) * (Tb - Ta): exactly twice the flux
// the reference computes for a constant lambda field, (lam*1/2 + lam*1/2) * (Ta*(-1) + Tb*1),
// and with the update scaled by dt/2 the FP64 results are bit-identical to the reference's
// serial walk with such a field.
#include <algorithm>
#include <map>
#include <vector>

#include "common.cuh"
#include "bulk.cuh"
#include "fp64_int.cuh"
#include "softflux.cuh"

struct nebo_patchset;  // opaque handle of the C ABI

namespace nebo {
namespace {

constexpr int PT_THREADS = 256;
constexpr int PF = 4;  // z planes prefetched ahead per thread
constexpr int PT_MAX_TY = 16;   // TX = 16
constexpr int PT_MAX_TX = 64;   // TY = 4

struct PatchDev {
  long long offset;  // element offset of the patch window in the arena
  long long off32;   // FP32 slab layout: element offset of the patch's interior (0,0,0)
  int nx, ny, nz;
  int log2tx;        // tile x extent = 1 << log2tx
  int pitch32;       // FP32 slab layout: row pitch in floats (nx rounded up to a multiple of 4)
  double lam2;       // 2*lambda
  double hdt;        // dt/2
};

struct WorkItem {
  int patch;
  int x0, y0;
  int z0, z1;
};

// Storage and arithmetic of the three precision modes.
//   PMODE_F64   value = double, fluxes double, round-to-nearest FP64 ops (bit-exact form)
//   PMODE_F32   value = float: FP32 storage and arithmetic (half the bytes of FP64); served by
//               patches_f32_strip_kernel below
//   PMODE_F32X2 value = float2 (hi, lo): the state as an unevaluated sum of two floats (~48-bit
//               significand); differences (hb-ha)+(lb-la), fluxes and the update in float, the
//               update added with an error-free two-sum.  No FP64 operation on the sweep.
enum { PMODE_F64 = 0, PMODE_F32 = 1, PMODE_F32X2 = 2 };

template <int M> struct PM;
template <> struct PM<PMODE_F64> {
  typedef double S;
  typedef double F;
  static __device__ __forceinline__ F diff(S a, S b) { return __dsub_rn(b, a); }
  static __device__ __forceinline__ F add(F a, F b) { return __dadd_rn(a, b); }
  static __device__ __forceinline__ F sub(F a, F b) { return __dsub_rn(a, b); }
  static __device__ __forceinline__ F mul(F a, F b) { return __dmul_rn(a, b); }
};
template <> struct PM<PMODE_F32X2> {
  typedef float2 S;
  typedef float F;
  static __device__ __forceinline__ F diff(S a, S b) { return (b.x - a.x) + (b.y - a.y); }
  static __device__ __forceinline__ F add(F a, F b) { return a + b; }
  static __device__ __forceinline__ F sub(F a, F b) { return a - b; }
  static __device__ __forceinline__ F mul(F a, F b) { return a * b; }
};

// (hi, lo) + inc with Knuth's two-sum, renormalised (Dekker's fast two-sum)
__device__ __forceinline__ float2 ff_add(float2 v, float inc) {
  const float s = __fadd_rn(v.x, inc);
  const float bb = __fsub_rn(s, v.x);
  const float e = __fadd_rn(__fsub_rn(v.x, __fsub_rn(s, bb)), __fsub_rn(inc, bb));
  const float lo = __fadd_rn(v.y, e);
  const float hi = __fadd_rn(s, lo);
  return make_float2(hi, __fsub_rn(lo, __fsub_rn(hi, s)));
}

template <typename T>
__device__ __forceinline__ void store_images(T* base, int sy, long sz, int x, int y, int z, int nx, int ny, int nz,
                                             T v) {
  base[(long)x + (long)sy * y + sz * z] = v;
  if (x != 0 && x != nx - 1 && y != 0 && y != ny - 1 && z != 0 && z != nz - 1) return;
  // a boundary cell: also write its periodic ghost images (up to 7 more cells; n >= 2 per axis)
  const int ax = x == 0 ? nx : -1, ay = y == 0 ? ny : -1, az = z == 0 ? nz : -1;
  const int m = (x == 0 || x == nx - 1) | ((y == 0 || y == ny - 1) << 1) | ((z == 0 || z == nz - 1) << 2);
  for (int b = 1; b < 8; ++b) {
    if (b & ~m) continue;
    const int xx = (b & 1) ? ax : x, yy = (b & 2) ? ay : y, zz = (b & 4) ? az : z;
    base[(long)xx + (long)sy * yy + sz * zz] = v;
  }
}

template <typename S>
__device__ __forceinline__ S ldg_s(const S* p) { return __ldg(p); }

// One persistent launch = one time step of every patch (mode M, see PM above).
template <int M>
__global__ void __launch_bounds__(PT_THREADS) patches_step_kernel(const PatchDev* __restrict__ patches,
                                                                  const WorkItem* __restrict__ items, int nitems,
                                                                  const typename PM<M>::S* __restrict__ src,
                                                                  typename PM<M>::S* __restrict__ dst) {
  typedef typename PM<M>::S S;
  typedef typename PM<M>::F F;
  __shared__ F sfx[2][PT_MAX_TY * (PT_MAX_TX + 1) / 4 + 64];  // TY*(TX+1) <= 16*17, 8*33, 4*65
  __shared__ F sfy[2][(PT_MAX_TY + 1) * 16 + 64];            // (TY+1)*TX <= 17*16, 9*32, 5*64
  const int tid = threadIdx.x;
  for (int w = blockIdx.x; w < nitems; w += gridDim.x) {
    const WorkItem it = items[w];
    const PatchDev P = patches[it.patch];
    const int lx = P.log2tx, TX = 1 << lx, TY = PT_THREADS >> lx;
    const int tx = tid & (TX - 1), ty = tid >> lx;
    const int nx = P.nx, ny = P.ny, nz = P.nz;
    const int sy = nx + 2;
    const long sz = (long)(nx + 2) * (ny + 2);
    const long interior = (long)1 + sy + sz;  // flat offset of interior (0,0,0)
    const S* tin = src + P.offset + interior;
    S* tout = dst + P.offset + interior;
    const F l2 = (F)P.lam2, hdt = (F)P.hdt;
    const int x = it.x0 + tx, y = it.y0 + ty;
    const bool active = x < nx && y < ny;
    const int xc = min(x, nx), yc = min(y, ny);
    auto at = [&](int i, int j, int k) { return (long)i + (long)sy * j + sz * k; };
    auto flux = [&](S ta, S tb) { return PM<M>::mul(l2, PM<M>::diff(ta, tb)); };
    S tc = ldg_s(tin + at(xc, yc, it.z0));
    F fzlo = flux(ldg_s(tin + at(xc, yc, it.z0 - 1)), tc);
    // register queue of the next PF planes (loads issued PF planes ahead of use; clamped to
    // the +z ghost plane, which exists)
    S q[PF];
#pragma unroll
    for (int i = 0; i < PF; ++i) q[i] = ldg_s(tin + at(xc, yc, min(it.z0 + 1 + i, nz)));
    for (int z = it.z0; z < it.z1; ++z) {
      const int buf = z & 1;
      const S tn = q[0];
#pragma unroll
      for (int i = 0; i < PF - 1; ++i) q[i] = q[i + 1];
      q[PF - 1] = ldg_s(tin + at(xc, yc, min(z + 1 + PF, nz)));
      const F fzhi = flux(tc, tn);
      const F fx = flux(ldg_s(tin + at(xc - 1, yc, z)), tc);
      const F fy = flux(ldg_s(tin + at(xc, yc - 1, z)), tc);
      sfx[buf][ty * (TX + 1) + tx] = fx;
      sfy[buf][ty * TX + tx] = fy;
      if (ty == 0) {  // +y halo faces of the tile
        const int yh = it.y0 + TY;
        if (yh <= ny && x <= nx) sfy[buf][TY * TX + tx] = flux(ldg_s(tin + at(xc, yh - 1, z)), ldg_s(tin + at(xc, yh, z)));
      } else if (ty == 1 && tx < TY) {  // +x halo faces of the tile
        const int xh = it.x0 + TX, yr = it.y0 + tx;
        if (xh <= nx && yr < ny) sfx[buf][tx * (TX + 1) + TX] = flux(ldg_s(tin + at(xh - 1, yr, z)), ldg_s(tin + at(xh, yr, z)));
      }
      __syncthreads();
      if (active) {
        const F fxhi = sfx[buf][ty * (TX + 1) + tx + 1];
        const F fyhi = sfy[buf][(ty + 1) * TX + tx];
        const F s = PM<M>::add(PM<M>::add(PM<M>::sub(fxhi, fx), PM<M>::sub(fyhi, fy)), PM<M>::sub(fzhi, fzlo));
        if constexpr (M == PMODE_F64) {
          store_images(tout, sy, sz, x, y, z, nx, ny, nz, __dadd_rn(tc, __dmul_rn(hdt, s)));
        } else {
          store_images(tout, sy, sz, x, y, z, nx, ny, nz, ff_add(tc, hdt * s));
        }
      }
      tc = tn;
      fzlo = fzhi;
    }
    __syncthreads();  // shared faces are reused by the next item
  }
}

// One persistent launch = one FP64 time step of every patch, the x and y face fluxes on the integer
// pipe (soft_flux, softflux.cuh; lambda is one s = 2 lambda per patch) beside the FP64 z flux and
// update, arranged as in heat_soft.cuh: values are unpacked once and staged with their halo two
// planes ahead, the update of plane z runs beside the integer fluxes of plane z + 1.  The same bits
// as FP64 fluxes: 9 FP64 operations per cell instead of 13, which is what bounds the step (with the
// lanes that a tile's ragged edge leaves idle).  128 patches of 16..96 cells an edge: 816 -> 560 us
// per step (612 with tiles of 16, 32 or 64 columns and z chunks of 16 planes).
//
// Tile shape: at most 2^log2tx columns (the autotuner's choice) and 256 cells, the patch's columns
// and then its rows split evenly, so that few lanes idle whatever the patch's extents (the FP64
// pipe's time goes by warps).  At most 64 rows: the tile's halo cells and faces have a thread each.
__host__ __device__ __forceinline__ void tile_shape(int nx, int ny, int log2tx, int& TX, int& TY) {
  const int lim = 1 << log2tx, kx = (nx + lim - 1) / lim;
  TX = (nx + kx - 1) / kx;
  const int most = PT_THREADS / TX < 64 ? PT_THREADS / TX : 64, ky = (ny + most - 1) / most;
  TY = (ny + ky - 1) / ky;
}
constexpr int PSOFT_CELLS = 400;  // max (TX + 2)(TY + 2): 66 x 6
struct PatchSoftShared {
  long long m[2][PSOFT_CELLS];
  int e[2][PSOFT_CELLS];
  double fx[2][PT_THREADS + 64];  // TY (TX + 1)
  double fy[2][PT_THREADS + 64];  // (TY + 1) TX
  int2 halo[PT_THREADS - 64];     // a halo cell's offset in a plane and staged index
  PatchDev P;                     // the item at hand (its 64 registers are taken)
  WorkItem it;
};

__device__ __forceinline__ void patch_soft_item(PatchSoftShared& sm, const double* __restrict__ src,
                                                double* __restrict__ dst) {
  using softfp::SoftVal;
  const PatchDev& P = sm.P;
  const WorkItem& it = sm.it;
  int TX, TY;
  tile_shape(P.nx, P.ny, P.log2tx, TX, TY);
  const int W = TX + 2, tid = threadIdx.x;
  // threads beyond the tile repeat its first cell and store nothing
  const bool in_tile = tid < TX * TY;
  const int ty = in_tile ? tid / TX : 0, tx = in_tile ? tid - ty * TX : 0;
  const int nx = P.nx, ny = P.ny, nz = P.nz, sy = nx + 2, sz = (nx + 2) * (ny + 2);
  const double s = P.lam2, hdt = P.hdt;
  const double* tin = src + P.offset + 1 + sy + sz;  // interior (0, 0, 0)
  double* tout = dst + P.offset + 1 + sy + sz;
  const int x0 = it.x0, y0 = it.y0, z0 = it.z0, z1 = it.z1;
  const int ic = min(x0 + tx, nx) + sy * min(y0 + ty, ny);
  const int si = (ty + 1) * W + tx + 1, fi = ty * (TX + 1) + tx, gi = ty * TX + tx;
  auto hard = [&](SoftVal a, SoftVal b) { return __dmul_rn(s, __dsub_rn(softfp::pack(b), softfp::pack(a))); };
  auto stage = [&](int buf, int i, double t) {
    const SoftVal v = softfp::unpack(t);
    sm.m[buf][i] = v.m;
    sm.e[buf][i] = v.e;
    return v;
  };
  auto staged = [&](int buf, int i) {
    SoftVal v;
    v.m = sm.m[buf][i];
    v.e = sm.e[buf][i];
    return v;
  };
  // halo cells, from thread 64 on (2 (TX + TY) <= 192 of them): columns x0 + TX and x0 - 1, rows
  // y0 - 1 and y0 + TY (clamped into the window; a clamped cell feeds no active face)
  const int h = tid - 64;
  const bool halo = h >= 0 && h < 2 * TY + 2 * TX;
  if (halo) {
    int2 c;
    if (h < 2 * TY) {
      const bool right = h < TY;
      const int r = right ? h : h - TY;
      c.x = (right ? min(x0 + TX, nx) : x0 - 1) + sy * min(y0 + r, ny);
      c.y = (r + 1) * W + (right ? TX + 1 : 0);
    } else {
      const bool above = h >= 2 * TY + TX;
      const int q = h - 2 * TY - (above ? TX : 0);
      c.x = min(x0 + q, nx) + sy * (above ? min(y0 + TY, ny) : y0 - 1);
      c.y = (above ? (TY + 1) * W : 0) + q + 1;
    }
    sm.halo[h] = c;  // (read by this thread only)
  }
  // the extra faces: the first TX threads those above the tile, the next TY those right of it
  const bool up = tid < TX;
  const bool xface = up ? (y0 + TY <= ny && x0 + tid <= nx)
                        : (tid < TX + TY && x0 + TX <= nx && y0 + (tid - TX) < ny);
  auto extra = [&](int buf) {
    if (xface) {
      const int i = up ? TY * W + tid + 1 : (tid - TX + 1) * W + TX;
      const SoftVal a = staged(buf, i), b = staged(buf, i + (up ? W : 1));
      bool ok;
      double f = softfp::soft_flux(s, a, b, ok);
      if (!ok) f = hard(a, b);
      *(up ? &sm.fy[buf][TY * TX + tid] : &sm.fx[buf][(tid - TX) * (TX + 1) + TX]) = f;
    }
  };
  double tc, tn, tn2, fzlo, fzhi, fx, fy;
  SoftVal X;  // of plane z + 1
  {
    const double* t0 = tin + (long)sz * z0;
    tc = ld_step(t0 + ic);
    tn = ld_step(t0 + sz + ic);
    const double tm = ld_step(t0 - sz + ic);
    fzlo = __dmul_rn(s, __dsub_rn(tc, tm));
    fzhi = __dmul_rn(s, __dsub_rn(tn, tc));
    const int b = z0 & 1;
    const SoftVal X0 = stage(b, si, tc);
    X = stage(b ^ 1, si, tn);
    if (halo) {
      const int2 c = sm.halo[h];
      stage(b, c.y, ld_step(t0 + c.x));
      stage(b ^ 1, c.y, ld_step(t0 + sz + c.x));
    }
    __syncthreads();
    bool ok;
    const SoftVal ax = staged(b, si - 1);
    fx = softfp::soft_flux(s, ax, X0, ok);
    if (!ok) fx = hard(ax, X0);
    const SoftVal ay = staged(b, si - W);
    fy = softfp::soft_flux(s, ay, X0, ok);
    if (!ok) fy = hard(ay, X0);
    sm.fx[b][fi] = fx;
    sm.fy[b][gi] = fy;
    extra(b);
    tn2 = ld_step(tin + (long)sz * min(z0 + 2, nz) + ic);
  }
  const bool active = in_tile && x0 + tx < nx && y0 + ty < ny;
  const bool edge = x0 + tx == 0 || x0 + tx == nx - 1 || y0 + ty == 0 || y0 + ty == ny - 1;
  auto store = [&](int z, double v) {
    if (!active) return;
    if (edge || z == 0 || z == P.nz - 1)
      store_images(tout, sy, (long)sz, it.x0 + tx, it.y0 + ty, z, P.nx, P.ny, P.nz, v);
    else
      tout[(long)sz * z + ic] = v;
  };
#pragma unroll 1
  for (int z = z0;; ++z) {
    __syncthreads();
    const int buf = z & 1, nb = buf ^ 1;
    const double a = __dsub_rn(sm.fx[buf][fi + 1], fx);
    const double b = __dsub_rn(sm.fy[buf][gi + TX], fy);
    const double c = __dsub_rn(fzhi, fzlo);
    if (z + 1 >= z1) {
      store(z, __dadd_rn(tc, __dmul_rn(hdt, __dadd_rn(__dadd_rn(a, b), c))));
      break;
    }
    const double dz = __dsub_rn(tn2, tn);
    const SoftVal xl = staged(nb, si - 1);
    bool okx, oky;
    double gx = softfp::soft_flux(s, xl, X, okx);
    const double ab = __dadd_rn(a, b);
    const SoftVal yl = staged(nb, si - W);
    double gy = softfp::soft_flux(s, yl, X, oky);
    const double sum = __dadd_rn(ab, c);
    // plane z + 2 (exists: z + 1 < z1 <= nz)
    const SoftVal Xn = stage(buf, si, tn2);
    if (halo) {
      const int2 c = sm.halo[h];
      stage(buf, c.y, ld_step(tin + (long)sz * (z + 2) + c.x));
    }
    const double prod = __dmul_rn(hdt, sum);
    const double gz = __dmul_rn(s, dz);
    const double v = __dadd_rn(tc, prod);
    if (!(okx && oky)) {
      gx = hard(xl, X);
      gy = hard(yl, X);
    }
    sm.fx[nb][fi] = gx;
    sm.fy[nb][gi] = gy;
    extra(nb);
    tc = tn;
    tn = tn2;
    tn2 = ld_step(tin + (long)sz * min(z + 3, P.nz) + ic);  // past nz: read again, not used
    store(z, v);
    fx = gx;
    fy = gy;
    fzlo = fzhi;
    fzhi = gz;
    X = Xn;
  }
}

__global__ void __launch_bounds__(PT_THREADS, 4) patches_soft_kernel(const PatchDev* __restrict__ patches,
                                                                     const WorkItem* __restrict__ items, int nitems,
                                                                     const double* __restrict__ src,
                                                                     double* __restrict__ dst) {
  __shared__ PatchSoftShared sm;
  step_begin();
  for (int w = blockIdx.x; w < nitems; w += gridDim.x) {
    if (threadIdx.x == 0) {
      sm.it = items[w];
      sm.P = patches[sm.it.patch];
    }
    __syncthreads();
    patch_soft_item(sm, src, dst);
    __syncthreads();  // the staged planes and faces are reused by the next item
  }
  step_end();
}

// FP32 mode shares the ring machinery of the FP32 heat step: plane p (z0-1 <= p <= z1) lives in
// stage (p - z0 + PNS) % PNS, iteration z waits for planes up to z+1, syncs, refills the stage of
// plane z-2 with plane z+PNS-2 and computes from the stages of planes z and z+1; the z loop is
// unrolled over the ring so stages are constants.  lambda is a scalar per patch, so each face
// costs (2 lambda) * (Tb - Ta): two FP32 operations.
constexpr int PNS = 5;

// Every ghost cell of every patch of an arena takes its periodic source's value (blocks of one
// blockIdx.y share a patch, threads over the six ghost faces: z faces whole, then y faces for the
// interior z, then x faces for the interior y and z).  FP64 arenas after loading (512 patches, a launch
// each, took 1.9 ms in all); FP32 windows after a run, as the strip kernel writes no ghosts during the
// steps.
template <typename T>
__global__ void __launch_bounds__(256) patches_ghosts_kernel(const PatchDev* __restrict__ patches, int npatch,
                                                             T* __restrict__ arena) {
  for (int p = blockIdx.y; p < npatch; p += gridDim.y) {
    const PatchDev P = patches[p];
    const int nx = P.nx, ny = P.ny, nz = P.nz, gx = nx + 2, gy = ny + 2;
    T* base = arena + P.offset + 1 + gx + (long)gx * gy;  // interior (0, 0, 0)
    const long sz = (long)gx * gy;
    const long A = (long)gx * gy, B = (long)gx * nz, C = (long)ny * nz;
    for (long g = blockIdx.x * (long)blockDim.x + threadIdx.x; g < 2 * (A + B + C);
         g += (long)gridDim.x * blockDim.x) {
      int x, y, z;
      if (g < 2 * A) {
        const long q = g % A;
        z = g < A ? -1 : nz;
        y = (int)(q / gx) - 1;
        x = (int)(q % gx) - 1;
      } else if (g < 2 * (A + B)) {
        const long h = g - 2 * A, q = h % B;
        y = h < B ? -1 : ny;
        z = (int)(q / gx);
        x = (int)(q % gx) - 1;
      } else {
        const long h = g - 2 * (A + B), q = h % C;
        x = h < C ? -1 : nx;
        z = (int)(q / ny);
        y = (int)(q % ny);
      }
      const int sx = x < 0 ? x + nx : (x >= nx ? x - nx : x);
      const int syy = y < 0 ? y + ny : (y >= ny ? y - ny : y);
      const int szz = z < 0 ? z + nz : (z >= nz ? z - nz : z);
      base[x + (long)gx * y + sz * z] = base[sx + (long)gx * syy + sz * szz];
    }
  }
}

__device__ __forceinline__ void pcp_async4(uint32_t smem, const void* gmem) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(smem), "l"(gmem) : "memory");
}
__device__ __forceinline__ void pcp_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void pcp_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

// FP32 mode, row strips: an item is a strip of R rows of W = min(nx, 512) columns of one patch
// over a z range (R <= 1024 / W, the patch's rows split evenly between its strips), and the
// block's 256 threads own its cells linearly (4 each, strided by 256), so lanes have cells
// whatever the patch's shape (tiles of fixed width leave up to half the lanes idle on patches of
// 16..96 cells).  The strip plus its one-cell halo, at most (R + 2)(W + 2) <= PR_STAGE floats,
// streams through the same ring of PNS stages as the tiled kernel; each cell reads its six
// neighbours from the stage and carries its centre value and the one below it in registers.  The
// halo is read from the periodic images' sources (x = -1 -> nx - 1, ...), so no step writes
// ghost cells: nebo_patchset_run fills them once after its last step.  With lambda constant over
// a patch the six face fluxes sum to 2 lambda (sum of the neighbours - 6 T), so a cell costs 5
// adds and 2 FMAs in FP32, T' = T + (dt lambda) (sum - 6 T) with dt lambda rounded once on the
// host (the FP64 mode keeps the reference's face form, bit for bit).
constexpr int PR_CELLS = 1024;                    // cells per strip plane
constexpr int PR_CPT = PR_CELLS / PT_THREADS;     // cells per thread
constexpr int PR_MAXW = 512;
constexpr int PR_STAGE = 2056;                    // max over W of (1024 / W + 2)(W + 2), W >= 2
constexpr int PR_NCOPY = (PR_STAGE + PT_THREADS - 1) / PT_THREADS;

// strip width and rows (the same on host and device)
__host__ __device__ __forceinline__ void strip_shape(int nx, int ny, int& wfull, int& rows) {
  wfull = nx < PR_MAXW ? nx : PR_MAXW;
  const int rmax = PR_CELLS / wfull, nstrips = (ny + rmax - 1) / rmax;
  rows = (ny + nstrips - 1) / nstrips;
}

__global__ void __launch_bounds__(PT_THREADS, 2) patches_f32_strip_kernel(const PatchDev* __restrict__ patches,
                                                                          const WorkItem* __restrict__ items,
                                                                          int nitems, const float* __restrict__ src,
                                                                          float* __restrict__ dst) {
  __shared__ __align__(16) float ring[PNS * PR_STAGE];
  const int tid = threadIdx.x;
  const uint32_t ring0 = (uint32_t)__cvta_generic_to_shared(ring);
  for (int w = blockIdx.x; w < nitems; w += gridDim.x) {
    const WorkItem it = items[w];
    const PatchDev P = patches[it.patch];
    const int nx = P.nx, ny = P.ny, nz = P.nz;
    int wfull, rfull;
    strip_shape(nx, ny, wfull, rfull);
    const int W = min(wfull, nx - it.x0), R = min(rfull, ny - it.y0);
    const int SW = W + 2, PLANE = SW * (R + 2);  // stage row pitch and size
    const int sy = nx + 2;
    const long sz = (long)(nx + 2) * (ny + 2);
    const long interior = (long)1 + sy + sz;
    const float* tin = src + P.offset + interior;
    float* tout = dst + P.offset + interior;
    const float k = (float)(P.hdt * P.lam2);  // T' = T + k (sum of the 6 neighbours - 6 T)
    const int z0 = it.z0, z1 = it.z1;
    // copy slots: unit k of the (R+2) x (W+2) halo strip, halo cells at the patch's faces taken
    // from their periodic sources
    int goff[PR_NCOPY];
#pragma unroll
    for (int j = 0; j < PR_NCOPY; ++j) {
      const int k = min(tid + j * PT_THREADS, PLANE - 1);
      const int r = k / SW, c = k - r * SW;
      int x = it.x0 - 1 + c, y = it.y0 - 1 + r;
      x = x < 0 ? x + nx : (x >= nx ? x - nx : x);
      y = y < 0 ? y + ny : (y >= ny ? y - ny : y);
      goff[j] = x + sy * y;
    }
    auto issue = [&](int p, int st) {
      if (p <= z1) {
        const float* tp = tin + sz * (p < 0 ? p + nz : (p >= nz ? p - nz : p));
        const uint32_t so = ring0 + (uint32_t)(st * PR_STAGE) * sizeof(float);
#pragma unroll
        for (int j = 0; j < PR_NCOPY; ++j) {
          const int k = tid + j * PT_THREADS;
          if (k < PLANE) pcp_async4(so + (uint32_t)k * sizeof(float), tp + goff[j]);
        }
      }
    };
    issue(z0 - 1, PNS - 1);
    pcp_commit();
#pragma unroll
    for (int i = 0; i < PNS - 2; ++i) {
      issue(z0 + i, i);
      pcp_commit();
    }
    // this thread's cells: strip cell tid + 256 j -> stage index si, window offset gi (x + sy y);
    // bit j of `live`: the cell exists
    int si[PR_CPT], gi[PR_CPT];
    unsigned live = 0;
#pragma unroll
    for (int j = 0; j < PR_CPT; ++j) {
      const int c = tid + j * PT_THREADS;
      const int r = c / W, col = c - r * W;
      if (c < W * R) live |= 1u << j;
      si[j] = c < W * R ? (r + 1) * SW + col + 1 : SW + 1;
      gi[j] = (it.x0 + col) + sy * (it.y0 + r);
    }
    pcp_wait<PNS - 3>();
    __syncthreads();
    float t[PR_CPT], tb[PR_CPT];  // the cell and the one below it
#pragma unroll
    for (int j = 0; j < PR_CPT; ++j) {
      t[j] = ring[si[j]];
      tb[j] = ring[(PNS - 1) * PR_STAGE + si[j]];
    }
    for (int zb = z0; zb < z1; zb += PNS) {
#pragma unroll
      for (int i = 0; i < PNS; ++i) {
        const int z = zb + i;
        if (z >= z1) break;
        pcp_wait<PNS - 4>();
        __syncthreads();
        issue(z + PNS - 2, (i + PNS - 2) % PNS);
        pcp_commit();
        const float* T0 = ring + i * PR_STAGE;
        const float* Tn = ring + ((i + 1) % PNS) * PR_STAGE;
#pragma unroll
        for (int j = 0; j < PR_CPT; ++j) {
          const int c = si[j];
          const float tc = t[j], tn = Tn[c];
          const float nb = ((T0[c - 1] + T0[c + 1]) + (T0[c - SW] + T0[c + SW])) + (tb[j] + tn);
          if ((live >> j) & 1u) tout[(long)gi[j] + sz * z] = fmaf(k, fmaf(-6.0f, tc, nb), tc);
          tb[j] = tc;
          t[j] = tn;
        }
      }
    }
    pcp_wait<0>();
    __syncthreads();  // the ring is refilled by the next item
  }
}

// FP32 mode on bulk-copied slabs (every patch with nx <= PB_CELLS).  The FP32 working state
// holds each patch's interior only, rows padded to a multiple of 4 floats (16 bytes) and each
// patch 256-byte aligned, so every row starts on a 16-byte boundary.  An item is a strip of R
// full rows of one patch over a z range (the rows split evenly between the strips).
// Per plane three cp.async.bulk copies fill a stage of the ring: the row below the strip, its R
// rows (one contiguous run) and the row above, the two halo rows and the halo planes taken from
// their periodic sources (rows ny-1 / 0, planes nz-1 / 0); the x halo is the row's own other end.
// One thread arms the stage's mbarrier and issues the copies; each of the 256 threads owns four
// consecutive cells of a row (R pitch <= 1024): rows start on 16-byte boundaries, so the rows above,
// below and of the next plane are one 16-byte load each and the four results one store, and only
// the two cells beside the quad are single loads.  A thread with four cells 256 apart loaded each
// neighbour of each cell by itself, 54 instructions a cell, and was bound by issue (81 %); 512
// patches of 16..96 cells an edge (742 MB a step) took 170 us a step that way and take 122 us so
// (6.1 TB/s; bound by memory; 131 us with three stages, 124 with five, 138 with seven, 134 at eight
// blocks an SM, whose 32 registers spill).  The operations of a cell are those of
// patches_f32_strip_kernel in the same order.
// No ghost cells exist in this layout: nebo_patchset_sync writes whole FP64 windows.
constexpr int PB_CELLS = 4 * PT_THREADS;  // floats per strip plane, the rows' padding included
constexpr int PB_NS = 4;                  // stages

__host__ __device__ __forceinline__ int strip_rows_bulk(int nx, int ny) {
  const int rmax = PB_CELLS / ((nx + 3) / 4 * 4);
  const int nstrips = (ny + rmax - 1) / rmax;
  return (ny + nstrips - 1) / nstrips;
}

__device__ unsigned int g_patch_bulk_timeouts;

// stage_floats: floats per stage (a multiple of 4, at least (R + 2) pitch32 for every item)
__global__ void __launch_bounds__(PT_THREADS) patches_f32_bulk_kernel(const PatchDev* __restrict__ patches,
                                                                      const WorkItem* __restrict__ items, int nitems,
                                                                      const float* __restrict__ src,
                                                                      float* __restrict__ dst, int stage_floats) {
  extern __shared__ __align__(128) unsigned char pb_smem[];
  const float* ring = reinterpret_cast<const float*>(pb_smem);
  const uint32_t ring0 = (uint32_t)__cvta_generic_to_shared(pb_smem);
  const uint32_t bar0 = ring0 + (uint32_t)(PB_NS * stage_floats) * 4u;
  const int tid = threadIdx.x;
  bool ok = true;
  step_begin();
  for (int w = blockIdx.x; w < nitems; w += gridDim.x) {
    const WorkItem it = items[w];
    const PatchDev P = patches[it.patch];
    const int nx = P.nx, ny = P.ny, nz = P.nz, pitch = P.pitch32;
    const int R = min(strip_rows_bulk(nx, ny), ny - it.y0);
    const long sz = (long)ny * pitch;
    const float* base = src + P.off32;
    float* obase = dst + P.off32;
    const float k = (float)(P.hdt * P.lam2);  // T' = T + k (sum of the 6 neighbours - 6 T)
    const int z0 = it.z0, z1 = it.z1;
    const uint32_t rowb = (uint32_t)pitch * 4u;
    const int ylo = it.y0 == 0 ? ny - 1 : it.y0 - 1;
    const int yhi = it.y0 + R == ny ? 0 : it.y0 + R;
    if (tid == 0) {
      for (int st = 0; st < PB_NS; ++st) mbar_init(bar0 + 8 * st, 1);
      asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncthreads();
    // plane q of the item is z0 - 1 + q (periodic), in stage st = q % PB_NS, phase (q / PB_NS) & 1
    auto issue = [&](int q, int st) {
      const int p = z0 - 1 + q;
      if (p > z1) return;  // the last plane read is z1 (the +z neighbour of the item's last plane)
      const int pw = p < 0 ? p + nz : (p >= nz ? p - nz : p);
      const uint32_t bar = bar0 + 8 * st;
      const uint32_t so = ring0 + (uint32_t)(st * stage_floats) * 4u;
      const float* pl = base + (long)pw * sz;
      mbar_expect_tx(bar, (uint32_t)(R + 2) * rowb);
      bulk_g2s(so, pl + (long)ylo * pitch, rowb, bar);
      bulk_g2s(so + rowb, pl + (long)it.y0 * pitch, (uint32_t)R * rowb, bar);
      bulk_g2s(so + (uint32_t)(R + 1) * rowb, pl + (long)yhi * pitch, rowb, bar);
    };
    if (tid == 0)
      for (int q = 0; q < PB_NS; ++q) issue(q, q);
    // this thread's four cells of a row (fewer at the row's end: the row's last quad may hold
    // padding, which is computed and stored but never read as a neighbour) in a stage; the cells
    // left and right of them, wrapped within the row; cell `last` is the row's last one
    const int quads = pitch >> 2;
    const bool act = tid < R * quads;
    const int r = act ? tid / quads : 0, col = act ? 4 * (tid - r * quads) : 0;
    const int row = (r + 1) * pitch, si = row + col;
    const int sl = row + (col == 0 ? nx : col) - 1, sr = col + 4 >= nx ? row : si + 4;
    const int last = nx - 1 - col;
    const float* mine = ring + si;
    ok &= mbar_wait(bar0, 0) & mbar_wait(bar0 + 8, 0);
    float4 tb = *reinterpret_cast<const float4*>(mine);                // the cells below
    float4 t = *reinterpret_cast<const float4*>(mine + stage_floats);  // the cells
    float* op = obase + (long)z0 * sz + (it.y0 + r) * pitch + col;
    int cs = 1, cn = 2, ce = 0;  // stages of the centre plane q, of q + 1 and of q - 1
    uint32_t phase = 0;          // of stage cn
    for (int z = z0; z < z1; ++z) {
      __syncthreads();  // plane q-1's stage is no longer read
      if (tid == 0) {
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        issue(z - z0 + PB_NS, ce);
      }
      ok &= mbar_wait(bar0 + 8 * cn, phase);
      const float* T0 = ring + cs * stage_floats;
      const float4 tn = *reinterpret_cast<const float4*>(mine + cn * stage_floats);
      const float4 td = *reinterpret_cast<const float4*>(T0 + si - pitch);
      const float4 tu = *reinterpret_cast<const float4*>(T0 + si + pitch);
      const float tl = T0[sl], tr = T0[sr];
      auto upd = [&](float l, float c, float rr, float d, float u, float b, float n) {
        const float nb = ((l + rr) + (d + u)) + (b + n);
        return fmaf(k, fmaf(-6.0f, c, nb), c);
      };
      float4 v;
      v.x = upd(tl, t.x, last == 0 ? tr : t.y, td.x, tu.x, tb.x, tn.x);
      v.y = upd(t.x, t.y, last == 1 ? tr : t.z, td.y, tu.y, tb.y, tn.y);
      v.z = upd(t.y, t.z, last == 2 ? tr : t.w, td.z, tu.z, tb.z, tn.z);
      v.w = upd(t.z, t.w, tr, td.w, tu.w, tb.w, tn.w);
      if (act) *reinterpret_cast<float4*>(op) = v;
      op += sz;
      tb = t;
      t = tn;
      ce = cs;
      cs = cn;
      if (++cn == PB_NS) {
        cn = 0;
        phase ^= 1u;
      }
    }
    __syncthreads();  // every copy of the item has landed and been read: the barriers start over
    if (tid == 0)
      for (int st = 0; st < PB_NS; ++st) mbar_inval(bar0 + 8 * st);
  }
  step_end();
  if (!ok) atomicAdd(&g_patch_bulk_timeouts, 1u);
}

// FP64 windows -> FP32 slab layout (interiors only) and back (whole windows: each cell of a
// window takes its periodic interior source, so the ghosts are filled in the same pass).  Packing, a
// warp takes a row, four of its cells per lane in flight.  Unpacking, a thread takes four consecutive
// window elements whatever rows they fall in: windows start on 256-byte boundaries, so the results are
// two 16-byte stores on a whole sector.  Values widen and round by their bits (a hardware conversion
// issues on the FP64 pipe).  512 patches of 16..96 cells an edge back to windows (1.2 GB): an index
// division per cell 623 us, a warp per row with 8-byte stores 358, two elements a thread 348, four 287
// (4.2 TB/s).
__device__ __forceinline__ float narrow(double v) {  // rounded to nearest, subnormal floats included
  const int e = fixmath::dexp(v);
  return e <= 896 && e >= 872 ? (float)v : fixmath::f64_to_f32_rn(v);
}
__device__ __forceinline__ int wrap1(int i, int n) { return i < 0 ? n - 1 : (i == n ? 0 : i); }

__global__ void __launch_bounds__(256) patches_pack_f32_kernel(const PatchDev* __restrict__ patches, int npatch,
                                                               const double* __restrict__ a64,
                                                               float* __restrict__ a32) {
  const int lane = threadIdx.x & 31, nw = gridDim.x * (blockDim.x >> 5);
  for (int p = blockIdx.y; p < npatch; p += gridDim.y) {
    const PatchDev P = patches[p];
    const int nx = P.nx, ny = P.ny, gx = nx + 2, gy = ny + 2;
    const long rows = (long)ny * P.nz;
    for (long r = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5); r < rows; r += nw) {
      const long z = fast_div(r, ny), y = r - z * ny;
      const double* from = a64 + P.offset + 1 + gx * (y + 1 + (long)gy * (z + 1));
      float* to = a32 + P.off32 + r * P.pitch32;
      for (int x = lane; x < nx; x += 128) {
        double v[4];
#pragma unroll
        for (int k = 0; k < 4; ++k) v[k] = x + 32 * k < nx ? __ldg(from + x + 32 * k) : 0.0;
#pragma unroll
        for (int k = 0; k < 4; ++k)
          if (x + 32 * k < nx) to[x + 32 * k] = narrow(v[k]);
      }
    }
  }
}
__global__ void __launch_bounds__(256) patches_unpack_f32_kernel(const PatchDev* __restrict__ patches, int npatch,
                                                                 const float* __restrict__ a32,
                                                                 double* __restrict__ a64) {
  for (int p = blockIdx.y; p < npatch; p += gridDim.y) {
    const PatchDev P = patches[p];
    const int nx = P.nx, ny = P.ny, nz = P.nz, gx = nx + 2, gy = ny + 2;
    const long total = (long)gx * gy * (nz + 2), step = 4 * (long)gridDim.x * blockDim.x;
    double* to = a64 + P.offset;
    for (long q = 4 * (blockIdx.x * (long)blockDim.x + threadIdx.x); q < total; q += step) {
      const long r = fast_div(q, gx);
      int c = (int)(q - r * gx), z = (int)fast_div(r, gy), y = (int)(r - (long)z * gy);
      const float* from = a32 + P.off32 + ((long)wrap1(z - 1, nz) * ny + wrap1(y - 1, ny)) * P.pitch32;
      float v[4];
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        v[k] = q + k < total ? __ldg(from + wrap1(c - 1, nx)) : 0.0f;
        if (++c == gx) {  // the next window row (past the window's end none is read)
          c = 0;
          if (++y == gy) {
            y = 0;
            ++z;
          }
          from = a32 + P.off32 + ((long)wrap1(min(z, nz + 1) - 1, nz) * ny + wrap1(y - 1, ny)) * P.pitch32;
        }
      }
      double w[4];
#pragma unroll
      for (int k = 0; k < 4; ++k) w[k] = fixmath::f32_to_f64(v[k]);
      if (q + 3 < total) {
        *reinterpret_cast<double2*>(to + q) = make_double2(w[0], w[1]);
        *reinterpret_cast<double2*>(to + q + 2) = make_double2(w[2], w[3]);
      } else {
        for (int k = 0; k < 4; ++k)
          if (q + k < total) to[q + k] = w[k];
      }
    }
  }
}

}  // namespace

// Bounded waits of the patch kernels that gave up since the last call (cleared by the read).
int patch_wait_timeouts(unsigned int* count) {
  unsigned int v = 0, zero = 0;
  NEBO_CUDA_TRY(cudaMemcpyFromSymbol(&v, g_patch_bulk_timeouts, sizeof(v)));
  if (v) NEBO_CUDA_TRY(cudaMemcpyToSymbol(g_patch_bulk_timeouts, &zero, sizeof(zero)));
  *count = v;
  return NEBO_OK;
}

struct PatchSet {
  int npatch = 0;
  int dtype = NEBO_F64;
  std::vector<int> shape;  // 3 per patch
  std::vector<long long> offset;
  std::vector<double> lam, dt;
  std::vector<int> log2tx;
  long long total = 0;  // elements per arena
  void* arena[2] = {nullptr, nullptr};    // FP64 states
  float* arena32[2] = {nullptr, nullptr};  // FP32 states (FP32 mode)
  float2* arena2[2] = {nullptr, nullptr};  // two-float states (FP32X2 mode)
  PatchDev* d_patches = nullptr;
  WorkItem* d_items = nullptr;
  int nitems = 0;
  int zchunk = 16;
  int grid = 0;
  bool wide_plane = false;  // some patch plane holds 2^31 cells or more (64-bit offsets: patches_step_kernel)
  int grid32 = 0;  // resident blocks of the FP32 ring kernel (one full wave)
  bool bulk32 = false;            // FP32 mode on the slab layout (every nx <= PB_CELLS)
  std::vector<long long> off32;   // slab layout: interior offsets
  std::vector<int> pitch32;       // slab layout: row pitches
  long long total32 = 0;          // slab layout: floats per arena
  int stage32 = 0;                // slab layout: floats per ring stage
  std::map<std::pair<int, int>, cudaGraphExec_t> graphs;  // (steps, parity) -> graph
  ~PatchSet() {
    for (auto& kv : graphs) cudaGraphExecDestroy(kv.second);
    cudaFree(arena[0]);
    cudaFree(arena[1]);
    cudaFree(arena32[0]);
    cudaFree(arena32[1]);
    cudaFree(arena2[0]);
    cudaFree(arena2[1]);
    cudaFree(d_patches);
    cudaFree(d_items);
  }
};

namespace {

std::vector<WorkItem> build_items(const PatchSet& ps, const std::vector<int>& which, int zchunk) {
  std::vector<WorkItem> items;
  for (int p : which) {
    const int nx = ps.shape[3 * p], ny = ps.shape[3 * p + 1], nz = ps.shape[3 * p + 2];
    // FP32: row strips (strip_shape); otherwise tiles, one row per thread row
    int TX = 1 << ps.log2tx[p], TY = PT_THREADS / TX;
    if (ps.dtype == NEBO_F64 && !ps.wide_plane) tile_shape(nx, ny, ps.log2tx[p], TX, TY);
    if (ps.dtype == NEBO_F32) {
      if (ps.bulk32) {
        TX = nx;
        TY = strip_rows_bulk(nx, ny);
      } else {
        strip_shape(nx, ny, TX, TY);
      }
    }
    for (int z0 = 0; z0 < nz; z0 += zchunk)
      for (int y0 = 0; y0 < ny; y0 += TY)
        for (int x0 = 0; x0 < nx; x0 += TX) items.push_back(WorkItem{p, x0, y0, z0, std::min(z0 + zchunk, nz)});
  }
  // largest z-extent items first so the strided assignment ends with short items
  std::stable_sort(items.begin(), items.end(), [](const WorkItem& a, const WorkItem& b) { return (a.z1 - a.z0) > (b.z1 - b.z0); });
  return items;
}

// FP64 items' z extent: the longest of 48, 32 and 16 planes that leaves three waves of resident
// blocks (an item stages two planes beyond its own; too few items leave the last wave ragged): 128
// patches of 16..96 cells 5.53 ms per 10 steps at 48, 5.64 at 32, 5.78 at 16; 20 small ones 0.43 at 16,
// 0.70 at 48.
int f64_zchunk(const PatchSet& ps, const std::vector<int>& all) {
  for (int zc : {48, 32})
    if ((long)build_items(ps, all, zc).size() >= 3L * 4 * num_sms()) return zc;
  return 16;
}

int upload_tables(PatchSet& ps, const std::vector<WorkItem>& items, cudaStream_t s) {
  std::vector<PatchDev> pd(ps.npatch);
  for (int p = 0; p < ps.npatch; ++p) {
    pd[p].offset = ps.offset[p];
    pd[p].off32 = ps.bulk32 ? ps.off32[p] : 0;
    pd[p].pitch32 = ps.bulk32 ? ps.pitch32[p] : 0;
    pd[p].nx = ps.shape[3 * p];
    pd[p].ny = ps.shape[3 * p + 1];
    pd[p].nz = ps.shape[3 * p + 2];
    pd[p].log2tx = ps.log2tx[p];
    pd[p].lam2 = ps.lam[p] + ps.lam[p];
    pd[p].hdt = 0.5 * ps.dt[p];
  }
  if (!ps.d_patches) NEBO_CUDA_TRY(cudaMalloc((void**)&ps.d_patches, sizeof(PatchDev) * ps.npatch));
  NEBO_CUDA_TRY(cudaMemcpyAsync(ps.d_patches, pd.data(), sizeof(PatchDev) * ps.npatch, cudaMemcpyHostToDevice, s));
  cudaFree(ps.d_items);
  ps.d_items = nullptr;
  NEBO_CUDA_TRY(cudaMalloc((void**)&ps.d_items, sizeof(WorkItem) * std::max<size_t>(1, items.size())));
  NEBO_CUDA_TRY(cudaMemcpyAsync(ps.d_items, items.data(), sizeof(WorkItem) * items.size(), cudaMemcpyHostToDevice, s));
  NEBO_CUDA_TRY(cudaStreamSynchronize(s));
  ps.nitems = (int)items.size();
  for (auto& kv : ps.graphs) cudaGraphExecDestroy(kv.second);
  ps.graphs.clear();
  return NEBO_OK;
}

int launch_step(const PatchSet& ps, const WorkItem* items, int nitems, int parity, cudaStream_t s) {
  if (nitems == 0) return NEBO_OK;
  LaunchScope ls(ps.dtype == NEBO_F64 ? "patches_step_f64" : (ps.dtype == NEBO_F32 ? "patches_step_f32" : "patches_step_f32x2"), s);
  const int grid = std::min(nitems, ps.grid);
  if (ps.dtype == NEBO_F64 && ps.wide_plane)
    patches_step_kernel<PMODE_F64><<<grid, PT_THREADS, 0, s>>>(ps.d_patches, items, nitems,
                                                               (const double*)ps.arena[parity],
                                                               (double*)ps.arena[parity ^ 1]);
  else if (ps.dtype == NEBO_F64)
    launch_step_kernel(patches_soft_kernel, dim3(grid), dim3(PT_THREADS), 0, s, ps.d_patches, items, nitems,
                       (const double*)ps.arena[parity], (double*)ps.arena[parity ^ 1]);
  else if (ps.dtype == NEBO_F32 && ps.bulk32)
    launch_step_kernel(patches_f32_bulk_kernel, dim3(std::min(nitems, ps.grid32)), dim3(PT_THREADS),
                       (size_t)PB_NS * ps.stage32 * sizeof(float) + PB_NS * sizeof(uint64_t), s, ps.d_patches, items,
                       nitems, ps.arena32[parity], ps.arena32[parity ^ 1], ps.stage32);
  else if (ps.dtype == NEBO_F32)
    patches_f32_strip_kernel<<<std::min(nitems, ps.grid32), PT_THREADS, 0, s>>>(ps.d_patches, items, nitems,
                                                                               ps.arena32[parity],
                                                                               ps.arena32[parity ^ 1]);
  else
    patches_step_kernel<PMODE_F32X2><<<grid, PT_THREADS, 0, s>>>(ps.d_patches, items, nitems, ps.arena2[parity],
                                                                 ps.arena2[parity ^ 1]);
  NEBO_LAUNCH_CHECK("nebo_patchset_run");
  return NEBO_OK;
}

int default_log2tx(int nx) { return nx <= 16 ? 4 : (nx <= 40 ? 5 : 6); }

__global__ void patches_cast_kernel(const double* __restrict__ a, float* __restrict__ b, size_t n) {
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x)
    b[i] = (float)a[i];
}
__global__ void patches_split_kernel(const double* __restrict__ a, float2* __restrict__ b, size_t n) {
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) {
    const float hi = (float)a[i];
    b[i] = make_float2(hi, (float)(a[i] - (double)hi));
  }
}
__global__ void patches_widen_kernel(const float* __restrict__ a, double* __restrict__ b, size_t n) {
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x)
    b[i] = (double)a[i];
}
__global__ void patches_join_kernel(const float2* __restrict__ a, double* __restrict__ b, size_t n) {
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x)
    b[i] = (double)a[i].x + (double)a[i].y;
}

}  // namespace
}  // namespace nebo

using namespace nebo;

struct nebo_patchset : PatchSet {};

extern "C" int nebo_patchset_create(nebo_patchset** out, int npatch, const int32_t* shapes, const double* lam,
                                    const double* dt, int dtype) {
  if (!out || npatch <= 0 || !shapes || !lam || !dt)
    return fail(NEBO_ERR_INVALID, "Nebo error in nebo_patchset_create: bad arguments");
  if (dtype != NEBO_F64 && dtype != NEBO_F32 && dtype != NEBO_F32X2)
    return fail(NEBO_ERR_INVALID, "Nebo error in nebo_patchset_create: dtype");
  *out = nullptr;
  nebo_patchset* ps = new nebo_patchset();
  ps->npatch = npatch;
  ps->dtype = dtype;
  ps->shape.assign(shapes, shapes + 3 * npatch);
  ps->lam.assign(lam, lam + npatch);
  ps->dt.assign(dt, dt + npatch);
  ps->offset.resize(npatch);
  ps->log2tx.resize(npatch);
  long long off = 0;
  for (int p = 0; p < npatch; ++p) {
    const int nx = shapes[3 * p], ny = shapes[3 * p + 1], nz = shapes[3 * p + 2];
    if (nx < 2 || ny < 2 || nz < 2) {
      delete ps;
      return fail(NEBO_ERR_INVALID, "Nebo error in nebo_patchset_create: patch %d has an edge below 2", p);
    }
    ps->offset[p] = off;
    ps->wide_plane = ps->wide_plane || (long long)(nx + 2) * (ny + 2) >= (1LL << 31);
    off += (long long)(nx + 2) * (ny + 2) * (nz + 2);
    off = (off + 31) & ~31LL;  // 256-byte aligned windows
    ps->log2tx[p] = default_log2tx(nx);
  }
  ps->total = off;
  const size_t bytes = (size_t)off * sizeof(double);
  cudaError_t e = cudaMalloc(&ps->arena[0], bytes);
  if (e == cudaSuccess) e = cudaMalloc(&ps->arena[1], bytes);
  if (e == cudaSuccess) e = cudaMemset(ps->arena[0], 0, bytes);
  if (e == cudaSuccess) e = cudaMemset(ps->arena[1], 0, bytes);
  if (dtype == NEBO_F32X2) {
    const size_t b2 = (size_t)off * sizeof(float2);
    if (e == cudaSuccess) e = cudaMalloc((void**)&ps->arena2[0], b2);
    if (e == cudaSuccess) e = cudaMalloc((void**)&ps->arena2[1], b2);
    if (e == cudaSuccess) e = cudaMemset(ps->arena2[0], 0, b2);
    if (e == cudaSuccess) e = cudaMemset(ps->arena2[1], 0, b2);
  }
  if (dtype == NEBO_F32) {
    // the slab layout when every row fits a strip: interiors only, rows padded to 16 bytes
    ps->bulk32 = true;
    for (int p = 0; p < npatch; ++p) ps->bulk32 = ps->bulk32 && shapes[3 * p] <= PB_CELLS;
    if (ps->bulk32) {
      ps->off32.resize(npatch);
      ps->pitch32.resize(npatch);
      long long o32 = 0;
      int stage = 0;
      for (int p = 0; p < npatch; ++p) {
        const int nx = shapes[3 * p], ny = shapes[3 * p + 1], nz = shapes[3 * p + 2];
        const int pitch = (nx + 3) / 4 * 4;
        ps->off32[p] = o32;
        ps->pitch32[p] = pitch;
        o32 += (long long)pitch * ny * nz;
        o32 = (o32 + 63) & ~63LL;  // 256-byte aligned patches
        stage = std::max(stage, (strip_rows_bulk(nx, ny) + 2) * pitch);
      }
      ps->total32 = o32;
      ps->stage32 = stage;
    }
  }
  if (dtype == NEBO_F32) {
    const size_t b32 = (size_t)(ps->bulk32 ? ps->total32 : off) * sizeof(float);
    if (e == cudaSuccess) e = cudaMalloc((void**)&ps->arena32[0], b32);
    if (e == cudaSuccess) e = cudaMalloc((void**)&ps->arena32[1], b32);
    if (e == cudaSuccess) e = cudaMemset(ps->arena32[0], 0, b32);
    if (e == cudaSuccess) e = cudaMemset(ps->arena32[1], 0, b32);
  }
  if (e != cudaSuccess) {
    delete ps;
    return cuda_fail(e, "nebo_patchset_create");
  }
  ps->grid = num_sms() * 8;
  if (dtype == NEBO_F32) {
    ps->zchunk = 1 << 30;  // FP32 items cover the patch's whole z extent
    int per_sm = 0;
    if (ps->bulk32) {
      const size_t smem = (size_t)PB_NS * ps->stage32 * sizeof(float) + PB_NS * sizeof(uint64_t);
      if (smem > 48 * 1024 &&
          cudaFuncSetAttribute(patches_f32_bulk_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) !=
              cudaSuccess) {
        cudaGetLastError();
        delete ps;
        return fail(NEBO_ERR_UNSUPPORTED, "Nebo error in nebo_patchset_create: FP32 strips need %zu bytes of "
                                          "shared memory", smem);
      }
      if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, patches_f32_bulk_kernel, PT_THREADS, smem) !=
              cudaSuccess ||
          per_sm < 1) {
        cudaGetLastError();
        per_sm = 1;
      }
    } else if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, patches_f32_strip_kernel, PT_THREADS, 0) !=
                   cudaSuccess ||
               per_sm < 1) {
      cudaGetLastError();
      per_sm = 1;
    }
    ps->grid32 = num_sms() * per_sm;
  }
  std::vector<int> all(npatch);
  for (int p = 0; p < npatch; ++p) all[p] = p;
  if (dtype == NEBO_F64) ps->zchunk = f64_zchunk(*ps, all);
  int rc = upload_tables(*ps, build_items(*ps, all, ps->zchunk), 0);
  if (rc) {
    delete ps;
    return rc;
  }
  *out = ps;
  return NEBO_OK;
}

extern "C" int nebo_patchset_destroy(nebo_patchset* ps) {
  delete ps;
  return NEBO_OK;
}

extern "C" int nebo_patchset_info(const nebo_patchset* ps, int64_t* total_elems, int64_t* offsets, int32_t* log2tx,
                                  int32_t* nitems) {
  if (!ps) return fail(NEBO_ERR_INVALID, "Nebo error in nebo_patchset_info: null handle");
  if (total_elems) *total_elems = ps->total;
  for (int p = 0; p < ps->npatch; ++p) {
    if (offsets) offsets[p] = ps->offset[p];
    if (log2tx) log2tx[p] = ps->log2tx[p];
  }
  if (nitems) *nitems = ps->nitems;
  return NEBO_OK;
}

extern "C" void* nebo_patchset_arena(const nebo_patchset* ps, int which) {
  return (ps && (which == 0 || which == 1)) ? ps->arena[which] : nullptr;
}

// Every patch's ghosts take their periodic images (run once after filling arena 0).
extern "C" int nebo_patchset_fill_ghosts(const nebo_patchset* ps, int which, nebo_stream_t stream) {
  if (!ps || (which != 0 && which != 1)) return fail(NEBO_ERR_INVALID, "Nebo error in nebo_patchset_fill_ghosts");
  {
    LaunchScope ls("patches_ghosts_f64", (cudaStream_t)stream);
    patches_ghosts_kernel<double><<<dim3(4, std::min(ps->npatch, 4096)), 256, 0, (cudaStream_t)stream>>>(
        ps->d_patches, ps->npatch, (double*)ps->arena[which]);
    NEBO_LAUNCH_CHECK("nebo_patchset_fill_ghosts");
  }
  if (ps->dtype == NEBO_F32 && ps->bulk32) {  // the FP32 working state, slab layout
    LaunchScope ls("patches_pack_f32", (cudaStream_t)stream);
    patches_pack_f32_kernel<<<dim3(8, std::min(ps->npatch, 4096)), 256, 0, (cudaStream_t)stream>>>(
        ps->d_patches, ps->npatch, (const double*)ps->arena[which], ps->arena32[which]);
    NEBO_LAUNCH_CHECK("nebo_patchset_fill_ghosts");
  } else if (ps->dtype == NEBO_F32) {  // the FP32 working state
    LaunchScope ls("patches_cast_f32", (cudaStream_t)stream);
    patches_cast_kernel<<<num_sms() * 8, 256, 0, (cudaStream_t)stream>>>((const double*)ps->arena[which],
                                                                         ps->arena32[which], (size_t)ps->total);
    NEBO_LAUNCH_CHECK("nebo_patchset_fill_ghosts");
  } else if (ps->dtype == NEBO_F32X2) {  // split each double into (hi, lo) floats
    LaunchScope ls("patches_split_f32x2", (cudaStream_t)stream);
    patches_split_kernel<<<num_sms() * 8, 256, 0, (cudaStream_t)stream>>>((const double*)ps->arena[which],
                                                                          ps->arena2[which], (size_t)ps->total);
    NEBO_LAUNCH_CHECK("nebo_patchset_fill_ghosts");
  }
  return NEBO_OK;
}

// Bring the state of arena `which` into its FP64 arena (FP32 mode widens, FP32X2 joins hi + lo;
// FP64 mode already keeps its state there).
extern "C" int nebo_patchset_sync(const nebo_patchset* ps, int which, nebo_stream_t stream) {
  if (!ps || (which != 0 && which != 1)) return fail(NEBO_ERR_INVALID, "Nebo error in nebo_patchset_sync");
  if (ps->dtype == NEBO_F64) return NEBO_OK;
  LaunchScope ls("patches_to_f64", (cudaStream_t)stream);
  if (ps->dtype == NEBO_F32X2)
    patches_join_kernel<<<num_sms() * 8, 256, 0, (cudaStream_t)stream>>>(ps->arena2[which], (double*)ps->arena[which],
                                                                         (size_t)ps->total);
  else if (ps->bulk32)
    patches_unpack_f32_kernel<<<dim3(32, std::min(ps->npatch, 4096)), 256, 0, (cudaStream_t)stream>>>(
        ps->d_patches, ps->npatch, ps->arena32[which], (double*)ps->arena[which]);
  else
    patches_widen_kernel<<<num_sms() * 8, 256, 0, (cudaStream_t)stream>>>(ps->arena32[which],
                                                                          (double*)ps->arena[which], (size_t)ps->total);
  NEBO_LAUNCH_CHECK("nebo_patchset_sync");
  return NEBO_OK;
}

// Time each tile width on the patches of each x-extent class and keep the fastest.
// FP32 strips need no tile width; the tuner picks the z extent of the items instead (whole
// patches, or chunks of 32 or 16 planes: shorter items balance the persistent blocks better,
// longer ones refill the plane ring less often) by timing whole steps.
static int autotune_strips(nebo_patchset* ps, cudaStream_t s, int32_t* chosen_log2tx) {
  std::vector<int> all(ps->npatch);
  for (int p = 0; p < ps->npatch; ++p) all[p] = p;
  cudaEvent_t a, b;
  NEBO_CUDA_TRY(cudaEventCreate(&a));
  NEBO_CUDA_TRY(cudaEventCreate(&b));
  int rc = NEBO_OK, bestz = ps->zchunk;
  float best = 1e30f;
  const int cands[3] = {1 << 30, 32, 16};
  for (int zc : cands) {
    rc = upload_tables(*ps, build_items(*ps, all, zc), s);
    if (rc) break;
    float ms = 0.f;
    for (int rep = 0; rep < 4 && !rc; ++rep) {
      cudaEventRecord(a, s);
      rc = launch_step(*ps, ps->d_items, ps->nitems, rep & 1, s);
      cudaEventRecord(b, s);
      cudaEventSynchronize(b);
      float t = 0.f;
      cudaEventElapsedTime(&t, a, b);
      if (rep > 0) ms += t;  // first launch warms up
    }
    if (!rc && ms < best) {
      best = ms;
      bestz = zc;
    }
  }
  cudaEventDestroy(a);
  cudaEventDestroy(b);
  if (rc) return rc;
  ps->zchunk = bestz;
  rc = upload_tables(*ps, build_items(*ps, all, ps->zchunk), s);
  if (rc) return rc;
  if (chosen_log2tx)
    for (int p = 0; p < ps->npatch; ++p) chosen_log2tx[p] = ps->log2tx[p];
  return NEBO_OK;
}

extern "C" int nebo_patchset_autotune(nebo_patchset* ps, nebo_stream_t stream, int32_t* chosen_log2tx) {
  if (!ps) return fail(NEBO_ERR_INVALID, "Nebo error in nebo_patchset_autotune: null handle");
  cudaStream_t s = (cudaStream_t)stream;
  if (ps->dtype == NEBO_F32) return autotune_strips(ps, s, chosen_log2tx);
  std::map<int, std::vector<int>> classes;  // class by nx bucket of 8
  for (int p = 0; p < ps->npatch; ++p) classes[(ps->shape[3 * p] + 7) / 8].push_back(p);
  cudaEvent_t a, b;
  NEBO_CUDA_TRY(cudaEventCreate(&a));
  NEBO_CUDA_TRY(cudaEventCreate(&b));
  WorkItem* d_tmp = nullptr;
  int rc = NEBO_OK;
  for (auto& kv : classes) {
    float best = 1e30f;
    int bestl = default_log2tx(ps->shape[3 * kv.second[0]]);
    for (int l = 4; l <= 6 && !rc; ++l) {
      for (int p : kv.second) ps->log2tx[p] = l;
      std::vector<WorkItem> items = build_items(*ps, kv.second, ps->zchunk);
      cudaFree(d_tmp);
      d_tmp = nullptr;
      if (cudaMalloc((void**)&d_tmp, sizeof(WorkItem) * items.size()) != cudaSuccess) { rc = NEBO_ERR_ALLOC; break; }
      cudaMemcpyAsync(d_tmp, items.data(), sizeof(WorkItem) * items.size(), cudaMemcpyHostToDevice, s);
      // patch table must carry the candidate tile width
      std::vector<int> keep = ps->log2tx;
      rc = upload_tables(*ps, std::vector<WorkItem>(), s);
      if (rc) break;
      float ms = 0.f;
      for (int rep = 0; rep < 4 && !rc; ++rep) {
        cudaEventRecord(a, s);
        rc = launch_step(*ps, d_tmp, (int)items.size(), rep & 1, s);
        cudaEventRecord(b, s);
        cudaEventSynchronize(b);
        float t = 0.f;
        cudaEventElapsedTime(&t, a, b);
        if (rep > 0) ms += t;  // first launch warms up
      }
      if (ms < best) {
        best = ms;
        bestl = l;
      }
    }
    for (int p : kv.second) ps->log2tx[p] = bestl;
  }
  cudaFree(d_tmp);
  cudaEventDestroy(a);
  cudaEventDestroy(b);
  if (rc) return rc;
  std::vector<int> all(ps->npatch);
  for (int p = 0; p < ps->npatch; ++p) all[p] = p;
  if (ps->dtype == NEBO_F64) ps->zchunk = f64_zchunk(*ps, all);
  rc = upload_tables(*ps, build_items(*ps, all, ps->zchunk), s);
  if (rc) return rc;
  if (chosen_log2tx)
    for (int p = 0; p < ps->npatch; ++p) chosen_log2tx[p] = ps->log2tx[p];
  // the timing runs overwrote the arenas: callers autotune before loading data
  return NEBO_OK;
}

// After the steps of a run: the FP32 strip kernel writes no ghost cells, so the arena that holds
// the result gets them here (one launch).
int finish_run(const PatchSet& ps, int which, cudaStream_t s) {
  if (ps.dtype != NEBO_F32 || ps.bulk32) return NEBO_OK;  // the slab layout has no ghost cells
  LaunchScope ls("patches_ghosts_f32", s);
  patches_ghosts_kernel<float><<<dim3(4, std::min(ps.npatch, 4096)), 256, 0, s>>>(ps.d_patches, ps.npatch,
                                                                                  ps.arena32[which]);
  NEBO_LAUNCH_CHECK("nebo_patchset_run ghosts");
  return NEBO_OK;
}

// steps time steps starting from arena `start`; returns (via *final) the arena holding the result.
extern "C" int nebo_patchset_run(nebo_patchset* ps, int start, int steps, int use_graph, int* final_arena,
                                 nebo_stream_t stream) {
  if (!ps || (start != 0 && start != 1) || steps < 0) return fail(NEBO_ERR_INVALID, "Nebo error in nebo_patchset_run");
  cudaStream_t s = (cudaStream_t)stream;
  if (final_arena) *final_arena = (start + steps) & 1;
  if (steps == 0) return NEBO_OK;
  if (!use_graph) {
    for (int k = 0; k < steps; ++k) {
      int rc = launch_step(*ps, ps->d_items, ps->nitems, (start + k) & 1, s);
      if (rc) return rc;
    }
    return finish_run(*ps, (start + steps) & 1, s);
  }
  const std::pair<int, int> key(steps, start);
  auto it = ps->graphs.find(key);
  if (it == ps->graphs.end()) {
    cudaStream_t cap;
    NEBO_CUDA_TRY(cudaStreamCreateWithFlags(&cap, cudaStreamNonBlocking));
    NEBO_CUDA_TRY(cudaStreamBeginCapture(cap, cudaStreamCaptureModeThreadLocal));
    int rc = NEBO_OK;
    for (int k = 0; k < steps && !rc; ++k) rc = launch_step(*ps, ps->d_items, ps->nitems, (start + k) & 1, cap);
    if (!rc) rc = finish_run(*ps, (start + steps) & 1, cap);
    cudaGraph_t g = nullptr;
    cudaError_t e = cudaStreamEndCapture(cap, &g);
    cudaStreamDestroy(cap);
    if (rc) {
      if (g) cudaGraphDestroy(g);
      return rc;
    }
    if (e != cudaSuccess) return cuda_fail(e, "nebo_patchset_run capture");
    cudaGraphExec_t exec;
    e = cudaGraphInstantiate(&exec, g, 0);
    cudaGraphDestroy(g);
    if (e != cudaSuccess) return cuda_fail(e, "nebo_patchset_run instantiate");
    it = ps->graphs.emplace(key, exec).first;
  }
  NEBO_CUDA_TRY(cudaGraphLaunch(it->second, s));
  return NEBO_OK;
}
