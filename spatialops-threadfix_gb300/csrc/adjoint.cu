// Adjoint of the fused heat step (no counterpart in the reference, which has no differentiation):
// gradients of  J = 1/2 * sum_interior (T_N - T_target)^2  with respect to T_0 and lambda, for
// T_{k+1} = T_k + dt * sum_d Div_d(Interp_d(lambda) * Grad_d(T_k)) on a periodic SVol patch with
// one ghost layer and unit spacing (the forward step is nebo_heat_step's, bit-exact FP64).
//
// Reverse step (abar' = dJ/dT_{k+1}, both with periodic ghost images):
//   abar[c]  = abar'[c] + dt * sum_d ( lf[c+s] (abar'[c+s]-abar'[c]) - lf[c] (abar'[c]-abar'[c-s]) )
//              -- the forward operator applied to abar' (it is self-adjoint on the periodic
//                 grid; the ghost fill's transpose folds ghost contributions onto their
//                 interior images, which the periodic ghost reads express);
//   glam[c] -= (dt/2) * sum_d ( (T[c]-T[c-s])(abar'[c]-abar'[c-s]) + (T[c+s]-T[c])(abar'[c+s]-abar'[c]) )
//              -- lambda[c] enters the face coefficients lf[c] and lf[c+s] with weight 1/2.
// One kernel per reverse step computes both, with every face quantity computed once and shared
// through shared memory (x, y) or carried in a register (z), and writes abar's ghost images.
//
// Memory: sqrt(N) checkpointing.  The forward sweep keeps T at every L-th step (L = ceil(sqrt N))
// and the states of the last segment; the reverse sweep recomputes each earlier segment's states
// from its checkpoint into a segment buffer and walks it backwards, so device memory grows like
// 2*sqrt(N) fields, not N, and the forward work is about 2N - sqrt(N) steps.
#include <cmath>
#include <vector>

#include <type_traits>

#include "common.cuh"
#include "fp64_int.cuh"
#include "softflux.cuh"

namespace nebo {
namespace {

constexpr int BX = 32;
constexpr int BY = 8;

// A forward state as a double (FP32 states widen exactly).
__device__ __forceinline__ double to_f64(double v) { return v; }
__device__ __forceinline__ double to_f64(float v) { return fixmath::f32_to_f64(v); }  // by its bits: a
// hardware conversion issues on the FP64 pipe

__device__ __forceinline__ void store_images1(double* base, int sy, long sz, int x, int y, int z, int nx, int ny, int nz,
                                              double v) {
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

// One reverse step.  Per face (a, b = a + s) the thread that owns the face computes
//   dA = A[b] - A[a],  dT = T[b] - T[a]                                   (FP64)
// and shares them (x, y through shared memory, z in a register).  Per cell c:
//   Aout[c] = A[c] + (dt/2) * sum_faces +-lf_face * dA_face              (FP64 FMA chain)
//   glam[c] -= (dt/2) * sum_faces dT_face * dA_face
// with lf_face = lambda[a] + lambda[b] either read from precomputed face arrays (LF) or summed
// from lambda.  EXACT: the face products dT*dA in FP64 (an FMA chain).  Otherwise each face
// product is an FP32 product of the FP32-rounded FP64 differences (relative error ~1e-7; the
// differences themselves are exact FP64, so no cancellation is amplified), their sum is FP32 and
// only the fold into glam is FP64: 6 FP64 operations per cell fewer, and the adjoint state A,
// hence dJ/dT0, is unaffected.
template <bool EXACT, bool LF, typename S = double>
__global__ void __launch_bounds__(BX* BY, sizeof(S) == 4 ? 3 : 4) heat_adjoint_kernel(const S* __restrict__ T, const double* __restrict__ Ain,
                                                              double* __restrict__ Aout, const double* __restrict__ L,
                                                              const double* __restrict__ lfx,
                                                              const double* __restrict__ lfy,
                                                              const double* __restrict__ lfz, double* __restrict__ glam,
                                                              int sy, long sz, int nx, int ny, int nz, int zchunk,
                                                              double hdt) {
  typedef typename std::conditional<EXACT, double, float>::type P;  // face-product operand type
  __shared__ double sax[2][BY][BX + 1];
  __shared__ double say[2][BY + 1][BX];
  __shared__ P stx[2][BY][BX + 1];
  __shared__ P sty[2][BY + 1][BX];
  const int tx = threadIdx.x, ty = threadIdx.y;
  const int x0 = blockIdx.x * BX, y0 = blockIdx.y * BY;
  const int x = x0 + tx, y = y0 + ty;
  const int z0 = blockIdx.z * zchunk, z1 = min(z0 + zchunk, nz);
  const bool active = x < nx && y < ny;
  const int xc = min(x, nx), yc = min(y, ny);
  auto at = [&](int i, int j, int k) { return (long)i + (long)sy * j + sz * k; };
  // (dA, dT) of face (a, b); dT as the product operand type
  auto face = [&](long a, long b, double& da, P& dt) {
    da = __ldg(Ain + b) - __ldg(Ain + a);
    const double d = to_f64(__ldg(T + b)) - to_f64(__ldg(T + a));  // exact for FP32 states too
    if constexpr (EXACT) dt = d; else dt = fixmath::f32_trunc(d);
  };
  auto coef = [&](const double* lf, long a, long b) { return LF ? __ldg(lf + b) : __ldg(L + a) + __ldg(L + b); };
  double dazl;
  P dtzl;
  face(at(xc, yc, z0 - 1), at(xc, yc, z0), dazl, dtzl);
  for (int z = z0; z < z1; ++z) {
    const int buf = z & 1;
    const long c = at(xc, yc, z);
    double dazh, dax, day;
    P dtzh, dtx, dty;
    face(c, c + sz, dazh, dtzh);
    face(c - 1, c, dax, dtx);
    face(c - sy, c, day, dty);
    sax[buf][ty][tx] = dax;
    stx[buf][ty][tx] = dtx;
    say[buf][ty][tx] = day;
    sty[buf][ty][tx] = dty;
    if (ty == 0) {
      const int yh = y0 + BY;
      if (yh <= ny && x <= nx) face(at(xc, yh - 1, z), at(xc, yh, z), say[buf][BY][tx], sty[buf][BY][tx]);
    } else if (ty == 1 && tx < BY) {
      const int xh = x0 + BX, yr = y0 + tx;
      if (xh <= nx && yr < ny) face(at(xh - 1, yr, z), at(xh, yr, z), sax[buf][tx][BX], stx[buf][tx][BX]);
    }
    __syncthreads();
    if (active) {
      const double daxh = sax[buf][ty][tx + 1], dayh = say[buf][ty + 1][tx];
      const P dtxh = stx[buf][ty][tx + 1], dtyh = sty[buf][ty + 1][tx];
      double s = dazh * coef(lfz, c, c + sz);
      s = fma(-dazl, coef(lfz, c - sz, c), s);
      s = fma(dayh, coef(lfy, c, c + sy), s);
      s = fma(-day, coef(lfy, c - sy, c), s);
      s = fma(daxh, coef(lfx, c, c + 1), s);
      s = fma(-dax, coef(lfx, c - 1, c), s);
      store_images1(Aout, sy, sz, x, y, z, nx, ny, nz, fma(hdt, s, Ain[c]));
      double ps;
      if constexpr (EXACT) {
        ps = dtzh * dazh;
        ps = fma(dtzl, dazl, ps);
        ps = fma(dtyh, dayh, ps);
        ps = fma(dty, day, ps);
        ps = fma(dtxh, daxh, ps);
        ps = fma(dtx, dax, ps);
      } else {
        using fixmath::f32_trunc;
        float q = dtzh * f32_trunc(dazh);
        q = fmaf(dtzl, f32_trunc(dazl), q);
        q = fmaf(dtyh, f32_trunc(dayh), q);
        q = fmaf(dty, f32_trunc(day), q);
        q = fmaf(dtxh, f32_trunc(daxh), q);
        q = fmaf(dtx, f32_trunc(dax), q);
        ps = fixmath::f32_to_f64(q);
      }
      glam[c] = fma(-hdt, ps, glam[c]);
    }
    dazl = dazh;
    dtzl = dtzh;
  }
}

// The reverse step on precomputed face coefficients and FP64 states with the x and y differences on
// the integer pipe (soft_sub, softflux.cuh), arranged as in heat_soft.cuh: T and A are unpacked once
// and staged with their halo two planes ahead, and the FP64 chains of plane z run beside the integer
// differences of plane z + 1 of other warps.  The operations and their order are
// heat_adjoint_kernel's, the bits too: 16 FP64 operations per cell instead of 20, 98 -> 86 us at
// 128^3 (three blocks per SM at 76 registers; the differences of T alone, 64 registers: 90 to 93; the
// differences without their fallback branches, so that chains and integers interleave, 89 at 80
// registers).
constexpr int AS_W = BX + 2;
struct AdjShared {
  long long m[2][2][(BY + 2) * AS_W];  // [buffer][T, A]
  int e[2][2][(BY + 2) * AS_W];
  double ax[2][BY][BX + 1], ay[2][BY + 1][BX];
  double tx[2][BY][BX + 1], ty[2][BY + 1][BX];
};

template <bool EXACT>
__global__ void __launch_bounds__(BX* BY, 3) heat_adjoint_soft_kernel(
    const double* __restrict__ T, const double* __restrict__ Ain, double* __restrict__ Aout,
    const double* __restrict__ lfx, const double* __restrict__ lfy, const double* __restrict__ lfz,
    double* __restrict__ glam, int sy, int sz, int nx, int ny, int nz, int zchunk, double hdt) {
  __shared__ AdjShared sm;
  using softfp::SoftVal;
  const int tx = threadIdx.x, ty = threadIdx.y;
  const int x0 = blockIdx.x * BX, y0 = blockIdx.y * BY;
  const int z0 = blockIdx.z * zchunk, z1 = min(z0 + zchunk, nz);
  const int xc = min(x0 + tx, nx), yc = min(y0 + ty, ny);
  const int ic = xc + sy * yc, si = (ty + 1) * AS_W + tx + 1;
  auto stage = [&](int buf, int f, int i, double v) {
    const SoftVal u = softfp::unpack(v);
    sm.m[buf][f][i] = u.m;
    sm.e[buf][f][i] = u.e;
    return u;
  };
  auto staged = [&](int buf, int f, int i) {
    SoftVal v;
    v.m = sm.m[buf][f][i];
    v.e = sm.e[buf][f][i];
    return v;
  };
  auto sub = [&](SoftVal a, SoftVal b) {
    bool ok;
    double d = softfp::soft_sub(a, b, ok);
    if (!ok) d = __dsub_rn(softfp::pack(b), softfp::pack(a));
    return d;
  };
  // halo cells: warp 1 the columns x0 + 32 (its first 8 lanes) and x0 - 1 (the next 8), warp 2 the
  // row below, warp 3 the row above; clamped into the window (a clamped cell feeds no active face)
  const bool halo = (ty == 1 && tx < 2 * BY) || ty == 2 || ty == 3;
  int ih, hi;
  if (ty == 1) {
    const int r = tx & (BY - 1);
    ih = (tx < BY ? min(x0 + BX, nx) : x0 - 1) + sy * min(y0 + r, ny);
    hi = (r + 1) * AS_W + (tx < BY ? BX + 1 : 0);
  } else {
    ih = xc + sy * (ty == 2 ? y0 - 1 : min(y0 + BY, ny));
    hi = (ty == 2 ? 0 : (BY + 1) * AS_W) + tx + 1;
  }
  // the extra faces: warp 0 those above the tile, the first lanes of warp 1 those right of it
  const bool xface = (ty == 0 && y0 + BY <= ny && x0 + tx <= nx) ||
                     (ty == 1 && tx < BY && x0 + BX <= nx && y0 + tx < ny);
  auto extra = [&](int buf) {
    if (xface) {
      const bool up = ty == 0;
      const int i = up ? BY * AS_W + tx + 1 : (tx + 1) * AS_W + BX, j = i + (up ? AS_W : 1);
      *(up ? &sm.ty[buf][BY][tx] : &sm.tx[buf][tx][BX]) = sub(staged(buf, 0, i), staged(buf, 0, j));
      *(up ? &sm.ay[buf][BY][tx] : &sm.ax[buf][tx][BX]) = sub(staged(buf, 1, i), staged(buf, 1, j));
    }
  };
  // differences across the low x and y faces of a staged plane, into the shared faces
  double dax, day, dtx, dty;
  auto faces = [&](int buf, SoftVal t, SoftVal a) {
    dtx = sub(staged(buf, 0, si - 1), t);
    dax = sub(staged(buf, 1, si - 1), a);
    dty = sub(staged(buf, 0, si - AS_W), t);
    day = sub(staged(buf, 1, si - AS_W), a);
    sm.tx[buf][ty][tx] = dtx;
    sm.ax[buf][ty][tx] = dax;
    sm.ty[buf][ty][tx] = dty;
    sm.ay[buf][ty][tx] = day;
    extra(buf);
  };
  step_begin();
  double tn, an, ac, tn2, an2, dazl, dtzl, dazh, dtzh;
  SoftVal X, Y;  // T and A of plane z + 1
  {
    const double* t0 = T + (long)sz * z0;
    const double* a0 = Ain + (long)sz * z0;
    const double tc = ld_step(t0 + ic);
    ac = ld_step(a0 + ic);
    tn = ld_step(t0 + sz + ic);
    an = ld_step(a0 + sz + ic);
    dazl = ac - ld_step(a0 - sz + ic);
    dtzl = tc - ld_step(t0 - sz + ic);
    dazh = an - ac;
    dtzh = tn - tc;
    const int b = z0 & 1;
    const SoftVal X0 = stage(b, 0, si, tc), Y0 = stage(b, 1, si, ac);
    X = stage(b ^ 1, 0, si, tn);
    Y = stage(b ^ 1, 1, si, an);
    if (halo) {
      stage(b, 0, hi, ld_step(t0 + ih));
      stage(b, 1, hi, ld_step(a0 + ih));
      stage(b ^ 1, 0, hi, ld_step(t0 + sz + ih));
      stage(b ^ 1, 1, hi, ld_step(a0 + sz + ih));
    }
    __syncthreads();
    faces(b, X0, Y0);
    const long o2 = (long)sz * min(z0 + 2, nz);
    tn2 = ld_step(T + o2 + ic);
    an2 = ld_step(Ain + o2 + ic);
  }
  const bool active = x0 + tx < nx && y0 + ty < ny;
  auto chain = [&](double kxl, double kxh, double kyl, double kyh, double kzl, double kzh, double daxh, double dayh) {
    double s = dazh * kzh;
    s = fma(-dazl, kzl, s);
    s = fma(dayh, kyh, s);
    s = fma(-day, kyl, s);
    s = fma(daxh, kxh, s);
    return fma(-dax, kxl, s);
  };
  auto products = [&](double daxh, double dayh, double dtxh, double dtyh) {
    if constexpr (EXACT) {
      double ps = dtzh * dazh;
      ps = fma(dtzl, dazl, ps);
      ps = fma(dtyh, dayh, ps);
      ps = fma(dty, day, ps);
      ps = fma(dtxh, daxh, ps);
      return fma(dtx, dax, ps);
    } else {
      using fixmath::f32_trunc;
      float q = f32_trunc(dtzh) * f32_trunc(dazh);
      q = fmaf(f32_trunc(dtzl), f32_trunc(dazl), q);
      q = fmaf(f32_trunc(dtyh), f32_trunc(dayh), q);
      q = fmaf(f32_trunc(dty), f32_trunc(day), q);
      q = fmaf(f32_trunc(dtxh), f32_trunc(daxh), q);
      q = fmaf(f32_trunc(dtx), f32_trunc(dax), q);
      return fixmath::f32_to_f64(q);
    }
  };
  auto store = [&](int z, double v, double gn) {
    if (active) {
      glam[(long)sz * z + ic] = gn;
      store_images1(Aout, sy, sz, x0 + tx, y0 + ty, z, nx, ny, nz, v);
    }
  };
#pragma unroll 1
  for (int z = z0;; ++z) {
    __syncthreads();
    const int buf = z & 1, nb = buf ^ 1;
    const long o = (long)sz * z + ic;
    const double daxh = sm.ax[buf][ty][tx + 1], dayh = sm.ay[buf][ty + 1][tx];
    const double dtxh = sm.tx[buf][ty][tx + 1], dtyh = sm.ty[buf][ty + 1][tx];
    const double kzh = ld_step(lfz + o + sz), kzl = ld_step(lfz + o), kyh = ld_step(lfy + o + sy), kyl = ld_step(lfy + o),
                 kxh = ld_step(lfx + o + 1), kxl = ld_step(lfx + o);
    const double g = active ? ld_step(glam + o) : 0.0;
    const double v = fma(hdt, chain(kxl, kxh, kyl, kyh, kzl, kzh, daxh, dayh), ac);
    const double gn = fma(-hdt, products(daxh, dayh, dtxh, dtyh), g);
    const bool more = z + 1 < z1;
    if (more) {
      dazl = dazh;
      dtzl = dtzh;
      dazh = an2 - an;
      dtzh = tn2 - tn;
      faces(nb, X, Y);
      // plane z + 2 (exists: z + 1 < z1 <= nz)
      X = stage(buf, 0, si, tn2);
      Y = stage(buf, 1, si, an2);
      if (halo) {
        stage(buf, 0, hi, ld_step(T + (long)sz * (z + 2) + ih));
        stage(buf, 1, hi, ld_step(Ain + (long)sz * (z + 2) + ih));
      }
    }
    if (!more) step_end();
    store(z, v, gn);
    if (!more) break;
    ac = an;
    tn = tn2;
    an = an2;
    const long o3 = (long)sz * min(z + 3, nz);  // past nz: read again, not used
    tn2 = ld_step(T + o3 + ic);
    an2 = ld_step(Ain + o3 + ic);
  }
}

// dst = src rounded to FP32 (whole windows of the same layout).
__global__ void to_f32_kernel(const double* __restrict__ src, float* __restrict__ dst, long n) {
  for (long i = blockIdx.x * (long)blockDim.x + threadIdx.x; i < n; i += (long)gridDim.x * blockDim.x)
    dst[i] = fixmath::f64_to_f32_rn(src[i]);
}

// abar_N = T_N - T_target on the interior (+ images); per-block partial sums of (T_N - T_target)^2.
template <typename S>
__global__ void loss_seed_kernel(const S* __restrict__ T, const double* __restrict__ Tt, double* __restrict__ A,
                                 int sy, long sz, int nx, int ny, int nz, double* __restrict__ partial) {
  double acc = 0.0;
  const long total = (long)nx * ny * nz;
  for (long i = blockIdx.x * (long)blockDim.x + threadIdx.x; i < total; i += (long)gridDim.x * blockDim.x) {
    const int x = (int)(i % nx), y = (int)((i / nx) % ny), z = (int)(i / ((long)nx * ny));
    const long c = (long)x + (long)sy * y + sz * z;
    const double d = to_f64(T[c]) - Tt[c];
    acc = fma(d, d, acc);
    store_images1(A, sy, sz, x, y, z, nx, ny, nz, d);
  }
  for (int o = 16; o > 0; o >>= 1) acc += __shfl_down_sync(0xffffffffu, acc, o);
  __shared__ double sh[32];
  if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = acc;
  __syncthreads();
  if (threadIdx.x == 0) {
    double t = 0.0;
    for (int i = 0; i < (int)(blockDim.x + 31) / 32; ++i) t += sh[i];
    partial[blockIdx.x] = t;
  }
}

}  // namespace

int heat_step_dispatch(const nebo_field* T, const nebo_field* To, const nebo_field* L, double dt, const double sp[3],
                       cudaStream_t s);  // heat.cu

}  // namespace nebo

using namespace nebo;

// One reverse step (exposed for tests): Aout, glam from T_k, A_{k+1}; all windows one ghost
// layer, same shape; A_{k+1} and T_k must hold periodic ghost images (lam too).
extern "C" int nebo_heat_adjoint_step(const nebo_field* Tk, const nebo_field* Ain, const nebo_field* Aout,
                                      const nebo_field* lam, const nebo_field* glam, double dt, nebo_stream_t stream) {
  const nebo_field* fs[5] = {Tk, Ain, Aout, lam, glam};
  for (int i = 0; i < 5; ++i) {
    int rc = check_field(fs[i], "nebo_heat_adjoint_step");
    if (rc) return rc;
    if (fs[i]->dtype != NEBO_F64) return fail(NEBO_ERR_UNSUPPORTED, "Nebo error in nebo_heat_adjoint_step: FP64 only");
    if ((rc = check_periodic_patch(fs[i], 1, "nebo_heat_adjoint_step"))) return rc;
    if (i && (rc = check_same_layout(Tk, fs[i], "nebo_heat_adjoint_step"))) return rc;
  }
  int n[3];
  interior_extent(*Tk, n);
  const View<double> vt = make_view<double>(*Tk), va = make_view<double>(*Ain), vo = make_view<double>(*Aout),
                     vl = make_view<double>(*lam), vg = make_view<double>(*glam);
  const int gxb = (n[0] + BX - 1) / BX, gyb = (n[1] + BY - 1) / BY;
  static std::atomic<int> per_sm{0};  // z chunks in whole waves of resident blocks
  const int zchunk = wave_zchunk((long)gxb * gyb,
                                 (long)num_sms() * blocks_per_sm(heat_adjoint_kernel<true, false>, BX * BY, per_sm),
                                 n[2], 1, 8, 1);
  const int chunks = (n[2] + zchunk - 1) / zchunk;
  cudaStream_t s = (cudaStream_t)stream;
  LaunchScope ls("heat_adjoint_step", s);
  heat_adjoint_kernel<true, false><<<dim3(gxb, gyb, chunks), dim3(BX, BY), 0, s>>>(
      vt.base, va.base, vo.base, vl.base, nullptr, nullptr, nullptr, vg.base, vt.sy, vt.sz, n[0], n[1], n[2], zchunk,
      0.5 * dt);
  NEBO_LAUNCH_CHECK("nebo_heat_adjoint_step");
  return NEBO_OK;
}

namespace {
// One reverse step of the gradient driver: precomputed face coefficients (View bases of the
// three face arrays, same layout as T), exact or FP32 face products.
template <typename S>
int adjoint_step_lf(const nebo_field* Tk, const nebo_field* Ain, const nebo_field* Aout, const double* lfx,
                    const double* lfy, const double* lfz, const nebo_field* glam, double dt, bool exact,
                    cudaStream_t s) {
  int n[3];
  interior_extent(*Tk, n);
  const View<S> vt = make_view<S>(*Tk);
  const View<double> va = make_view<double>(*Ain), vo = make_view<double>(*Aout), vg = make_view<double>(*glam);
  const int gxb = (n[0] + BX - 1) / BX, gyb = (n[1] + BY - 1) / BY;
  if constexpr (std::is_same<S, double>::value) {
    if (heat_faces_ok(Tk)) {
      static std::atomic<int> per_sm[2];  // z chunks in whole waves of resident blocks (zero: not queried)
      auto go = [&](auto kern, std::atomic<int>& cache) {
        const int zchunk =
            wave_zchunk((long)gxb * gyb, (long)num_sms() * blocks_per_sm(kern, BX * BY, cache), n[2], 2, 4, 1);
        LaunchScope ls("heat_adjoint_step", s);
        launch_step_kernel(kern, dim3(gxb, gyb, (n[2] + zchunk - 1) / zchunk), dim3(BX, BY), 0, s,
            vt.base, va.base, vo.base, lfx, lfy, lfz, vg.base, vt.sy, (int)vt.sz, n[0], n[1], n[2], zchunk, 0.5 * dt);
      };
      if (exact)
        go(heat_adjoint_soft_kernel<true>, per_sm[1]);
      else
        go(heat_adjoint_soft_kernel<false>, per_sm[0]);
      NEBO_LAUNCH_CHECK("nebo_heat_gradient (reverse step)");
      return NEBO_OK;
    }
  }
  static std::atomic<int> per_sm[2];  // z chunks in whole waves of resident blocks (zero: not queried)
  const int bps = exact ? blocks_per_sm(heat_adjoint_kernel<true, true, S>, BX * BY, per_sm[1])
                        : blocks_per_sm(heat_adjoint_kernel<false, true, S>, BX * BY, per_sm[0]);
  const int zchunk = wave_zchunk((long)gxb * gyb, (long)num_sms() * bps, n[2], 1, 8, 1);
  const int chunks = (n[2] + zchunk - 1) / zchunk;
  LaunchScope ls("heat_adjoint_step", s);
  if (exact)
    heat_adjoint_kernel<true, true, S><<<dim3(gxb, gyb, chunks), dim3(BX, BY), 0, s>>>(
        vt.base, va.base, vo.base, nullptr, lfx, lfy, lfz, vg.base, vt.sy, vt.sz, n[0], n[1], n[2], zchunk, 0.5 * dt);
  else
    heat_adjoint_kernel<false, true, S><<<dim3(gxb, gyb, chunks), dim3(BX, BY), 0, s>>>(
        vt.base, va.base, vo.base, nullptr, lfx, lfy, lfz, vg.base, vt.sy, vt.sz, n[0], n[1], n[2], zchunk, 0.5 * dt);
  NEBO_LAUNCH_CHECK("nebo_heat_gradient (reverse step)");
  return NEBO_OK;
}
}  // namespace

namespace {
// The state buffers (element type S, `stride` elements apart): [0, nck) checkpoints T_0, T_L, ...;
// [nck, nck+L) segment states; two forward temporaries; for FP32 states one more for the FP32
// copy of lambda.  The FP64 buffers: two adjoint states, three face-coefficient arrays, then 256
// doubles of loss partials.
template <typename S>
int gradient_impl(S* spool, size_t stride, double* dpool, size_t cells, int nck, int L, const nebo_field* T0,
                  const nebo_field* lam, const nebo_field* Ttarget, int steps, double dt, bool exact,
                  const nebo_field* gT0, const nebo_field* glam, double* J, nebo_stream_t stream) {
  constexpr bool f64 = std::is_same<S, double>::value;
  cudaStream_t s = (cudaStream_t)stream;
  const size_t bytes = cells * sizeof(double);
  auto sbuf = [&](size_t i) { return spool + i * stride; };
  auto dbuf = [&](size_t i) { return dpool + i * cells; };
  double* partial = dpool + 5 * cells;
  auto state_at = [&](S* p) {
    nebo_field f = *T0;
    f.data = p;
    f.dtype = f64 ? NEBO_F64 : NEBO_F32;
    return f;
  };
  auto field_at = [&](double* p) {
    nebo_field f = *T0;
    f.data = p;
    return f;
  };
  const double unit[3] = {1.0, 1.0, 1.0};
  int rc = NEBO_OK;
  nebo_field lamf = *lam;
  int n[3];
  interior_extent(*T0, n);
  // lambda's ghosts must be periodic images (they are read at boundary faces); face coefficients
  if ((rc = fill_periodic_any(&lamf, s))) return rc;
  double* A0 = dbuf(0);
  double* A1 = dbuf(1);
  S* tmp0 = sbuf(nck + L);
  S* tmp1 = sbuf(nck + L + 1);
  const View<double> vl = make_view<double>(lamf);
  const long origin = vl.base - (const double*)lamf.data;  // interior origin within a window
  double* lf[3] = {dbuf(2) + origin, dbuf(3) + origin, dbuf(4) + origin};
  if ((rc = heat_face_coef(&lamf, lf, false, s))) return rc;
  // the forward sweep's lambda and T_0 in the state type
  nebo_field lamS = lamf;
  if constexpr (!f64) {
    lamS = state_at(sbuf(nck + L + 2));
    LaunchScope ls("to_f32", s);
    to_f32_kernel<<<num_sms() * 4, 256, 0, s>>>((const double*)lamf.data, (float*)lamS.data, (long)cells);
    to_f32_kernel<<<num_sms() * 4, 256, 0, s>>>((const double*)T0->data, (float*)sbuf(0), (long)cells);
    NEBO_LAUNCH_CHECK("nebo_heat_gradient (FP32 forward copies)");
  } else {
    NEBO_CUDA_TRY(cudaMemcpyAsync(sbuf(0), T0->data, bytes, cudaMemcpyDeviceToDevice, s));
  }
  // FP64 steps share the reverse sweep's face coefficients
  const bool faces = f64 && heat_faces_ok(T0);
  auto forward_step = [&](const nebo_field* a, const nebo_field* b) {
    return faces ? heat_step_faces(a, b, lf, dt, unit, s) : heat_step_dispatch(a, b, &lamS, dt, unit, s);
  };
  // forward sweep: checkpoints every L steps; the last segment's states go straight to the
  // segment buffers (they need no recomputation)
  const int klast = (nck - 1) * L;
  {
    nebo_field c0 = state_at(sbuf(0));
    if ((rc = fill_periodic_any(&c0, s))) return rc;
  }
  S* cur = sbuf(0);
  for (int k = 0; k < steps && !rc; ++k) {
    const int j = k + 1;  // state being written
    S* nxt;
    if (j == steps)
      nxt = cur == tmp0 ? tmp1 : tmp0;
    else if (j % L == 0)
      nxt = sbuf(j / L);
    else if (j > klast)
      nxt = sbuf(nck + (j - klast - 1));
    else
      nxt = cur == tmp0 ? tmp1 : tmp0;
    nebo_field a = state_at(cur), b = state_at(nxt);
    rc = forward_step(&a, &b);
    cur = nxt;
  }
  if (rc) return rc;
  // seed: abar_N = T_N - T_target, J
  const View<S> vt = make_view<S>(state_at(cur));
  const View<double> vtt = make_view<double>(*Ttarget);
  const View<double> va = make_view<double>(field_at(A0));
  {
    LaunchScope ls("loss_seed", s);
    loss_seed_kernel<S><<<256, 256, 0, s>>>(vt.base, vtt.base, va.base, vt.sy, vt.sz, n[0], n[1], n[2], partial);
  }
  NEBO_CUDA_TRY(cudaGetLastError());
  double hp[256];
  NEBO_CUDA_TRY(cudaMemcpyAsync(hp, partial, sizeof(hp), cudaMemcpyDeviceToHost, s));
  NEBO_CUDA_TRY(cudaMemsetAsync(glam->data, 0, bytes, s));
  // reverse sweep, segment by segment
  double* Ain = A0;
  double* Aout = A1;
  for (int seg = nck - 1; seg >= 0 && !rc; --seg) {
    const int k0 = seg * L, k1 = (k0 + L < steps) ? k0 + L : steps;  // states k0 .. k1-1
    // recompute states k0+1 .. k1-1 into the segment buffers (state k0 is the checkpoint)
    for (int k = k0; seg != nck - 1 && k + 1 < k1 && !rc; ++k) {
      nebo_field a = state_at(k == k0 ? sbuf(seg) : sbuf(nck + (k - k0 - 1)));
      nebo_field b = state_at(sbuf(nck + (k - k0)));
      rc = forward_step(&a, &b);
    }
    for (int k = k1 - 1; k >= k0 && !rc; --k) {
      nebo_field tk = state_at(k == k0 ? sbuf(seg) : sbuf(nck + (k - k0 - 1)));
      nebo_field ai = field_at(Ain), ao = field_at(Aout);
      rc = adjoint_step_lf<S>(&tk, &ai, &ao, lf[0], lf[1], lf[2], glam, dt, exact, s);
      double* t = Ain;
      Ain = Aout;
      Aout = t;
    }
  }
  if (rc) return rc;
  NEBO_CUDA_TRY(cudaMemcpyAsync(gT0->data, Ain, bytes, cudaMemcpyDeviceToDevice, s));
  NEBO_CUDA_TRY(cudaStreamSynchronize(s));
  if (J) {
    double t = 0.0;
    for (int i = 0; i < 256; ++i) t += hp[i];
    *J = 0.5 * t;
  }
  return rc;
}

int gradient_entry(const nebo_field* T0, const nebo_field* lam, const nebo_field* Ttarget, int steps, double dt,
                   int checkpoint_every, bool exact, bool forward_f32, const nebo_field* gT0, const nebo_field* glam,
                   double* J, nebo_stream_t stream, const char* what) {
  const nebo_field* fs[5] = {T0, lam, Ttarget, gT0, glam};
  for (int i = 0; i < 5; ++i) {
    int rc = check_field(fs[i], what);
    if (rc) return rc;
    if (fs[i]->dtype != NEBO_F64) return fail(NEBO_ERR_UNSUPPORTED, "Nebo error in %s: FP64 only", what);
    if ((rc = check_periodic_patch(fs[i], 1, what))) return rc;
    if (i && (rc = check_same_layout(T0, fs[i], what))) return rc;
  }
  if (steps < 1) return fail(NEBO_ERR_INVALID, "Nebo error in %s: steps < 1", what);
  cudaStream_t s = (cudaStream_t)stream;
  const size_t cells = (size_t)T0->glob[0] * T0->glob[1] * T0->glob[2];
  const size_t ssize = forward_f32 ? sizeof(float) : sizeof(double);
  const size_t stride = (cells + 63) / 64 * 64;  // state buffers 256-byte aligned
  const size_t dbytes = 5 * cells * sizeof(double) + 256 * sizeof(double);
  int L = checkpoint_every > 0 ? checkpoint_every : (int)std::ceil(std::sqrt((double)steps));
  if (L > steps) L = steps;  // a segment never holds more than the run's states
  if (checkpoint_every == NEBO_CHECKPOINT_AUTO) {
    // every state kept (no recomputation) when all of them fit in 80 % of the free memory
    size_t free_b = 0, total_b = 0;
    if (cudaMemGetInfo(&free_b, &total_b) == cudaSuccess) {
      if (((size_t)steps + 4) * stride * ssize + dbytes <= free_b / 10 * 8) L = 1;
    } else {
      cudaGetLastError();
    }
  }
  const int nck = (steps + L - 1) / L;  // checkpoints at steps 0, L, 2L, ...
  // state buffers: nck checkpoints + L segment states + 2 forward temporaries (+ FP32 lambda),
  // ~ 2 sqrt(N) fields; FP64: 2 adjoint states + 3 face-coefficient arrays
  const size_t nstate = (size_t)nck + (size_t)L + 2 + (forward_f32 ? 1 : 0);
  void* spool = nullptr;
  double* dpool = nullptr;
  pool_retain();
  NEBO_CUDA_TRY(cudaMallocAsync(&spool, nstate * stride * ssize, s));
  cudaError_t e = cudaMallocAsync((void**)&dpool, dbytes, s);
  if (e != cudaSuccess) {
    cudaFreeAsync(spool, s);
    return cuda_fail(e, what);
  }
  const int rc = forward_f32
                     ? gradient_impl<float>((float*)spool, stride, dpool, cells, nck, L, T0, lam, Ttarget, steps, dt,
                                            exact, gT0, glam, J, stream)
                     : gradient_impl<double>((double*)spool, stride, dpool, cells, nck, L, T0, lam, Ttarget, steps, dt,
                                             exact, gT0, glam, J, stream);
  cudaFreeAsync(spool, s);
  cudaFreeAsync(dpool, s);
  return rc;
}
}  // namespace

// Full gradient with sqrt(N) checkpointing.  T0, lam, Ttarget: windows (1 ghost, periodic patch);
// gT0, glam: outputs (windows; interiors written, glam overwritten); J: host result.
// checkpoint_every 0 (or below, other than NEBO_CHECKPOINT_AUTO) selects ceil(sqrt(steps));
// NEBO_CHECKPOINT_AUTO keeps every state when they fit in device memory.
extern "C" int nebo_heat_gradient(const nebo_field* T0, const nebo_field* lam, const nebo_field* Ttarget, int steps,
                                  double dt, int checkpoint_every, const nebo_field* gT0, const nebo_field* glam,
                                  double* J, nebo_stream_t stream) {
  return gradient_entry(T0, lam, Ttarget, steps, dt, checkpoint_every, true, false, gT0, glam, J, stream,
                        "nebo_heat_gradient");
}

extern "C" int nebo_heat_gradient_ex(const nebo_field* T0, const nebo_field* lam, const nebo_field* Ttarget, int steps,
                                     double dt, int checkpoint_every, int products, const nebo_field* gT0,
                                     const nebo_field* glam, double* J, nebo_stream_t stream) {
  const int prod = products & ~NEBO_FORWARD_F32;
  if (prod != NEBO_PRODUCTS_F64 && prod != NEBO_PRODUCTS_F32)
    return fail(NEBO_ERR_INVALID, "Nebo error in nebo_heat_gradient_ex: products %d", products);
  return gradient_entry(T0, lam, Ttarget, steps, dt, checkpoint_every, prod == NEBO_PRODUCTS_F64,
                        (products & NEBO_FORWARD_F32) != 0, gT0, glam, J, stream, "nebo_heat_gradient_ex");
}
