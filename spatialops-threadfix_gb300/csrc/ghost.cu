// Periodic ghost exchange inside one GPU's memory: every ghost cell of a uniform-ghost patch
// takes the value of its wrapped interior image.  This is the single-patch stand-in for the
// halo exchange that callers of the reference perform between patches (the reference itself
// has no periodic support; its heat driver fills ghosts by copy before each step).
#include "common.cuh"

namespace nebo {
namespace {

// Up to FILL_MAX fields of one shape, blockIdx.y the field (base: its interior (0,0,0)).
constexpr int FILL_MAX = 6;
struct FillArgs {
  void* base[FILL_MAX];
  int wide[FILL_MAX];  // 1: doubles
  int sy;
  long sz;
  int nx, ny, nz, g;
};

// The ghost shell is split into the two z slabs (full x,y extent), the two y slabs (interior z) and
// the two x slabs (interior y,z), so every ghost cell is visited exactly once and no interior cell
// is touched.  A warp takes a row of a z or y slab (gx cells, one index computation for all of
// them, eight loads in flight), or the 2 g x-ghosts of 32 interior rows, one row per lane.  What
// bounds it: latency.  Five fields of 324^3 with two ghost layers: 90 us in five launches with a
// division per cell, 40 in one.
template <typename T>
__device__ __forceinline__ void fill_shell(T* __restrict__ base, const FillArgs& a) {
  const int gx = a.nx + 2 * a.g, gy = a.ny + 2 * a.g, g = a.g;
  const long zrows = 2L * g * gy, yrows = 2L * g * a.nz, inner = (long)a.ny * a.nz;
  const long total = zrows + yrows + (inner + 31) / 32;
  const int lane = threadIdx.x & 31;
  const long nw = (long)gridDim.x * (blockDim.x >> 5);
  auto wrap = [](int i, int n) { return i < 0 ? i + n : (i >= n ? i - n : i); };  // g <= n
  for (long w = (long)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5); w < total; w += nw) {
    if (w < zrows + yrows) {
      int y, z;
      if (w < zrows) {
        const int k = (int)fast_div(w, gy);
        y = (int)(w - (long)k * gy) - g;
        z = k < g ? k - g : a.nz + (k - g);
      } else {
        const long q = w - zrows;
        z = (int)fast_div(q, 2 * g);
        const int k = (int)(q - (long)z * (2 * g));
        y = k < g ? k - g : a.ny + (k - g);
      }
      T* to = base + (long)a.sy * y + a.sz * z;
      const T* from = base + (long)a.sy * wrap(y, a.ny) + a.sz * wrap(z, a.nz);
      for (int i = lane; i < gx; i += 256) {  // eight loads in flight
        T v[8];
#pragma unroll
        for (int k = 0; k < 8; ++k) v[k] = i + 32 * k < gx ? from[wrap(i + 32 * k - g, a.nx)] : T(0);
#pragma unroll
        for (int k = 0; k < 8; ++k)
          if (i + 32 * k < gx) to[i + 32 * k - g] = v[k];
      }
    } else {
      const long q = (w - zrows - yrows) * 32 + lane;
      if (q < inner) {
        const long z = fast_div(q, a.ny);
        T* row = base + (long)a.sy * (q - z * a.ny) + a.sz * z;
        for (int k = 0; k < g; ++k) {
          const T hi = row[k - g + a.nx], lo = row[k];
          row[k - g] = hi;
          row[a.nx + k] = lo;
        }
      }
    }
  }
}

__global__ void __launch_bounds__(256) fill_periodic_kernel(const __grid_constant__ FillArgs a) {
  if (a.wide[blockIdx.y])
    fill_shell(static_cast<double*>(a.base[blockIdx.y]), a);
  else
    fill_shell(static_cast<float*>(a.base[blockIdx.y]), a);
}

}  // namespace

int fill_periodic_fields(const nebo_field* const* fs, int count, cudaStream_t s) {
  const nebo_field* f = fs[0];
  int rc = check_field(f, "nebo_fill_periodic");
  if (rc) return rc;
  const int g = f->ghost_minus[0];
  if ((rc = check_periodic_patch(f, g, "nebo_fill_periodic"))) return rc;
  if (g == 0) return NEBO_OK;
  if (count > FILL_MAX) return fail(NEBO_ERR_INVALID, "Nebo error in nebo_fill_periodic: %d fields", count);
  int n[3];
  interior_extent(*f, n);
  FillArgs a{};
  a.sy = f->glob[0];
  a.sz = (long)f->glob[0] * f->glob[1];
  a.nx = n[0];
  a.ny = n[1];
  a.nz = n[2];
  a.g = g;
  for (int i = 0; i < count; ++i) {
    a.wide[i] = fs[i]->dtype == NEBO_F64;
    a.base[i] = a.wide[i] ? (void*)make_view<double>(*fs[i]).base : (void*)make_view<float>(*fs[i]).base;
  }
  const long warps = 2L * g * (n[1] + 2 * g) + 2L * g * n[2] + ((long)n[1] * n[2] + 31) / 32;
  const long want = (warps + 7) / 8;
  const int blocks = (int)(want < (long)num_sms() * 16 ? want : (long)num_sms() * 16);
  LaunchScope ls("fill_periodic", s);
  fill_periodic_kernel<<<dim3(blocks, count), 256, 0, s>>>(a);
  NEBO_LAUNCH_CHECK("nebo_fill_periodic");
  return NEBO_OK;
}

int fill_periodic_any(const nebo_field* f, cudaStream_t s) { return fill_periodic_fields(&f, 1, s); }

}  // namespace nebo

extern "C" int nebo_fill_periodic(const nebo_field* f, nebo_stream_t stream) {
  return nebo::fill_periodic_any(f, (cudaStream_t)stream);
}
