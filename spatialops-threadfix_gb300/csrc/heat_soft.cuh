// The exact FP64 heat step on precomputed face coefficients with face fluxes on the integer pipe
// (soft_flux, softflux.cuh): the bits of heat_step_kernel (heat.cu, where the operator stands).
//
// What bounds it.  heat_step_kernel keeps the FP64 pipe 82 % busy at 16 operations per cell (34 in
// general spacing) while 17 % of the issue slots are used.  Here:
//   * the face coefficients RN(la + lb) come from a pass per run (face_coef_kernel): 3 operations
//     fewer, 16 bytes more per cell, which HBM has to spare;
//   * unit spacing: the x and y fluxes are integer work (60 ALU instructions each), the z flux and
//     the update 9 FP64 operations: FP64 70 % and ALU 59 % busy together.  (z flux in integers too:
//     368 against 357 us at 256^3 with 3 blocks per SM, the ALU then bounds it.)
//   * general spacing: the reference multiplies both cells of a face by 1/d and both faces of a cell
//     again; each product is taken once per cell and axis (face and axis) instead, and all three
//     fluxes are integer work: 13 FP64 operations per cell.  (z flux in FP64: 669 against 595 us.)
// A 32 x 8 tile marches in z: values are unpacked once and staged with their halo two planes ahead,
// and the FP64 update of plane z runs beside the integer fluxes of plane z + 1, so one covers the
// other's latency (without that overlap 408 us at 256^3).  32 x 16 tiles, with fewer halo faces per
// cell but 512 threads at a barrier, were slower (365 us).
// Measured per step (heat_step_kernel -> this, GB300): unit 256^3 552 -> 348 us, 128^3 82 -> 57,
// 64^3 14.5 -> 12.4 (in a graph 12.6 -> 10.0); spacing (0.5, 0.8, 1.25) 256^3 1098 -> 622,
// 203 x 131 x 98 207 -> 123.
#pragma once

#include "common.cuh"
#include "softflux.cuh"

namespace nebo {
namespace {

constexpr int HS_X = 32, HS_Y = 8;

struct SoftHeatParams {
  double hdt;    // UNIT: dt/2; else dt
  double c1[3];  // 1/d per axis (not UNIT)
};

// lfx, lfy, lfz: face_coef_kernel's arrays (HALF in general spacing), same layout as tin.
template <bool UNIT>
__global__ void __launch_bounds__(HS_X* HS_Y, UNIT ? 4 : 3) heat_soft_kernel(
    const double* __restrict__ tin, double* __restrict__ tout, const double* __restrict__ lfx,
    const double* __restrict__ lfy, const double* __restrict__ lfz, int sy, int sz, int nx, int ny, int nz, int zchunk,
    SoftHeatParams p) {
  constexpr bool SOFTZ = !UNIT;
  constexpr int W = HS_X + 2, H = HS_Y + 2;
  constexpr int NV = UNIT ? 1 : 2;  // staged values per cell: scaled for the x and the y faces
  __shared__ long long sM[2][NV][H * W];
  __shared__ int sE[2][NV][H * W];
  __shared__ double sfx[2][HS_Y][HS_X + 1];
  __shared__ double sfy[2][HS_Y + 1][HS_X];
  using softfp::SoftVal;
  const int tx = threadIdx.x, ty = threadIdx.y;
  const int x0 = blockIdx.x * HS_X, y0 = blockIdx.y * HS_Y;
  const int z0 = blockIdx.z * zchunk, z1 = min(z0 + zchunk, nz);
  const int xc = min(x0 + tx, nx), yc = min(y0 + ty, ny);
  auto scaled = [&](double t, int axis) { return UNIT ? t : __dmul_rn(t, p.c1[axis]); };
  auto hard = [&](double s, SoftVal a, SoftVal b) {
    return __dmul_rn(s, __dsub_rn(softfp::pack(b), softfp::pack(a)));
  };
  auto stage = [&](int buf, int i, double t) {
    const SoftVal v = softfp::unpack(scaled(t, 0));
    sM[buf][0][i] = v.m;
    sE[buf][0][i] = v.e;
    if (!UNIT) {
      const SoftVal w = softfp::unpack(scaled(t, 1));
      sM[buf][NV - 1][i] = w.m;
      sE[buf][NV - 1][i] = w.e;
    }
    return v;
  };
  auto staged = [&](int buf, int axis, int i) {
    SoftVal v;
    v.m = sM[buf][axis ? NV - 1 : 0][i];
    v.e = sE[buf][axis ? NV - 1 : 0][i];
    return v;
  };
  // halo cells of the staged plane: warp 1 the columns x0 + 32 (its first 8 lanes) and x0 - 1 (the
  // next 8), warp 2 the row below, warp 3 the row above; clamped into the window (a clamped cell
  // feeds no active face)
  const int si = (ty + 1) * W + tx + 1;  // the cell's staged index
  // the halo cell's offset in a plane and staged index (UNIT keeps them in shared memory: its 64
  // registers are taken)
  __shared__ int2 shalo[3][HS_X];
  int2 h0 = make_int2(0, 0);
  const bool halo = (ty == 1 && tx < 2 * HS_Y) || ty == 2 || ty == 3;
  if (halo) {
    const int r = tx & (HS_Y - 1);
    int2 h;
    if (ty == 1) {
      h.x = (tx < HS_Y ? min(x0 + HS_X, nx) : x0 - 1) + sy * min(y0 + r, ny);
      h.y = (r + 1) * W + (tx < HS_Y ? HS_X + 1 : 0);
    } else {
      h.x = xc + sy * (ty == 2 ? y0 - 1 : min(y0 + HS_Y, ny));
      h.y = (ty == 2 ? 0 : (HS_Y + 1) * W) + tx + 1;
    }
    if (UNIT) shalo[ty - 1][tx] = h;
    h0 = h;
  }
  const int ic = xc + sy * yc;  // the cell's offset in a plane (fewer than 2^31 cells)
  // the extra faces: warp 0 those above the tile, the first lanes of warp 1 those right of it
  const bool xface = (ty == 0 && y0 + HS_Y <= ny && x0 + tx <= nx) ||
                     (ty == 1 && tx < HS_Y && x0 + HS_X <= nx && y0 + tx < ny);
  auto halo_at = [&]() { return UNIT ? shalo[ty - 1][tx] : h0; };
  struct Coef {
    double x, y, z, e;  // of the cell's low x and y faces and its high z face; of the extra face
  };
  auto load = [&](int z) {
    Coef k;
    const long o = (long)sz * z;
    k.x = ld_step(lfx + o + ic);
    k.y = ld_step(lfy + o + ic);
    k.z = ld_step(lfz + o + sz + ic);  // plane z + 1 <= nz
    k.e = 0.0;
    if (xface) {
      k.e = ty == 0 ? ld_step(lfy + o + xc + sy * (y0 + HS_Y)) : ld_step(lfx + o + x0 + HS_X + sy * (y0 + tx));
    }
    return k;
  };
  auto extra = [&](int buf, double s) {
    if (xface) {
      const bool up = ty == 0;
      const int i = up ? HS_Y * W + tx + 1 : (tx + 1) * W + HS_X;
      const SoftVal a = staged(buf, up, i), b = staged(buf, up, i + (up ? W : 1));
      bool ok;
      double f = softfp::soft_flux(s, a, b, ok);
      if (!ok) f = hard(s, a, b);
      *(up ? &sfy[buf][HS_Y][tx] : &sfx[buf][tx][HS_X]) = f;
    }
  };

  step_begin();
  // plane z0: staged, its low z face and its other faces
  double tc, tn, tn2, hn = 0.0, fzlo, fzhi, fx, fy;
  SoftVal X, Z;  // of plane z + 1 (in general spacing scaled for its x and z faces)
  Coef k = load(z0);
  {
    const double* t0 = tin + (long)sz * z0;
    tc = ld_step(t0 + ic);
    tn = ld_step(t0 + sz + ic);
    const double tm = ld_step(t0 - sz + ic);
    fzlo = __dmul_rn(ld_step(lfz + (long)sz * z0 + ic), __dsub_rn(scaled(tc, 2), scaled(tm, 2)));
    const int b = z0 & 1;
    const SoftVal X0 = stage(b, si, tc);
    X = stage(b ^ 1, si, tn);
    if (SOFTZ) Z = softfp::unpack(scaled(tn, 2));
    if (halo) {
      const int2 h = halo_at();
      stage(b, h.y, ld_step(t0 + h.x));
      stage(b ^ 1, h.y, ld_step(t0 + sz + h.x));
    }
    __syncthreads();
    fzhi = __dmul_rn(k.z, __dsub_rn(scaled(tn, 2), scaled(tc, 2)));
    bool ok;
    const SoftVal ax = staged(b, 0, si - 1);
    fx = softfp::soft_flux(k.x, ax, X0, ok);
    if (!ok) fx = hard(k.x, ax, X0);
    const SoftVal ay = staged(b, 1, si - W), by = UNIT ? X0 : staged(b, 1, si);
    fy = softfp::soft_flux(k.y, ay, by, ok);
    if (!ok) fy = hard(k.y, ay, by);
    sfx[b][ty][tx] = fx;
    sfy[b][ty][tx] = fy;
    extra(b, k.e);
    const long o2 = (long)sz * min(z0 + 2, nz);
    tn2 = ld_step(tin + o2 + ic);
    if (!UNIT) hn = halo ? ld_step(tin + o2 + halo_at().x) : 0.0;
    if (z0 + 1 < z1) k = load(z0 + 1);
  }
  auto store = [&](int z, double v) {
    const int x = x0 + tx, y = y0 + ty;
    if (x < nx && y < ny) {
      tout[(long)sz * z + ic] = v;
      if (x == 0 || x == nx - 1 || y == 0 || y == ny - 1 || z == 0 || z == nz - 1)
        store_images_only(tout, sy, sz, x, y, z, nx, ny, nz, v);
    }
  };
#pragma unroll 1
  for (int z = z0;; ++z) {
    __syncthreads();
    // The update of plane z (FP64) runs beside the fluxes of plane z + 1 (integers): neither
    // depends on the other, so the FP64 latencies are covered by the integer instructions.
    const int buf = z & 1, nb = buf ^ 1;
    const double fxhi = sfx[buf][ty][tx + 1], fyhi = sfy[buf][ty + 1][tx];
    double a, b, c;
    if (UNIT) {
      a = __dsub_rn(fxhi, sfx[buf][ty][tx]);
      b = __dsub_rn(fyhi, fy);
      c = __dsub_rn(fzhi, fzlo);
    } else {
      a = __dsub_rn(__dmul_rn(fxhi, p.c1[0]), __dmul_rn(sfx[buf][ty][tx], p.c1[0]));
      b = __dsub_rn(__dmul_rn(fyhi, p.c1[1]), __dmul_rn(sfy[buf][ty][tx], p.c1[1]));
      c = __dsub_rn(__dmul_rn(fzhi, p.c1[2]), __dmul_rn(fzlo, p.c1[2]));
    }
    if (z + 1 >= z1) {
      step_end();
      store(z, __dadd_rn(tc, __dmul_rn(p.hdt, __dadd_rn(__dadd_rn(a, b), c))));
      break;
    }
    const double dz = SOFTZ ? 0.0 : __dsub_rn(tn2, tn);
    const SoftVal xl = staged(nb, 0, si - 1);
    bool okx, oky, okz = true;
    double gx = softfp::soft_flux(k.x, xl, X, okx);
    const double ab = __dadd_rn(a, b);
    const SoftVal yl = staged(nb, 1, si - W), Y = UNIT ? X : staged(nb, 1, si);
    double gy = softfp::soft_flux(k.y, yl, Y, oky);
    const double sum = __dadd_rn(ab, c);
    // plane z + 2 (exists: z + 1 < z1 <= nz)
    const SoftVal Xn = stage(buf, si, tn2);
    if (halo) {
      const int2 h = halo_at();
      stage(buf, h.y, UNIT ? ld_step(tin + (long)sz * (z + 2) + h.x) : hn);
    }
    const double prod = __dmul_rn(p.hdt, sum);
    double gz;
    SoftVal Zn;
    if (SOFTZ) {
      Zn = softfp::unpack(scaled(tn2, 2));
      gz = softfp::soft_flux(k.z, Z, Zn, okz);
    } else {
      gz = __dmul_rn(k.z, dz);
    }
    const double v = __dadd_rn(tc, prod);
    if (!(okx && oky && okz)) {
      gx = hard(k.x, xl, X);
      gy = hard(k.y, yl, Y);
      if (SOFTZ) gz = hard(k.z, Z, Zn);
    }
    sfx[nb][ty][tx] = gx;
    sfy[nb][ty][tx] = gy;
    extra(nb, k.e);
    // loads of the next iteration: plane z + 3 (clamped to nz, then unused) and the coefficients
    // of plane z + 2's faces (unused in the last iteration)
    const long o3 = (long)sz * min(z + 3, nz);
    tc = tn;
    tn = tn2;
    tn2 = ld_step(tin + o3 + ic);
    if (!UNIT) hn = halo ? ld_step(tin + o3 + halo_at().x) : 0.0;
    k = load(min(z + 2, z1 - 1));
    store(z, v);
    fy = gy;
    fzlo = fzhi;
    fzhi = gz;
    X = Xn;
    if (SOFTZ) Z = Zn;
  }
}

}  // namespace
}  // namespace nebo
