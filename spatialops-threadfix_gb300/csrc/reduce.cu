// Reductions nebo_sum / nebo_max / nebo_min / nebo_norm (and _interior) over one field
// (spatialops/NeboReductions.h:45-240).  The reference folds serially on the CPU; here a
// deterministic tree runs on the device:
//   per thread: batches of 8 independent loads, each batch summed exactly in 128-bit fixed point
//               and folded into a Neumaier-compensated FP64 sum (or max/min keys); a region that is
//               one run of memory is walked as such, others a warp per row;
//   per block:  the threads' sums (and compensations) add exactly in 128-bit fixed point, max/min
//               as order-preserving integer keys: one (sum, rest) pair or extremum per block;
//   last step:  the blocks' pairs add the same way, rounded once.
// What bounds it: a small field its chain of dependent steps, a large one the integer pipe (about 50
// instructions per element of a sum beside 0.6 FP64 operations; 20 us of HBM time at 256^3).  An FP64
// instruction holds its SM's pipe for 16 clocks a warp, so a shuffle tree of compensated adds (35
// of them per warp) cost more than reading a 66^3 field: 23 us a field plus 11 us for the merge;
// the integer tree takes none.  Measured, kernels of one nebo_sum: 66^3 34 -> 5 us (with nebo_reduce's
// single launch and no device-to-host copy 60 -> 23 us per call from Python, 14.6 from C), 258^3 FP64
// 63 us, max 35 us.
// FP32 fields are accumulated in FP64.  max/min use the reference's comparisons
// ((r < v) ? v : r and (r > v) ? v : r: NaNs never win), so they are exact; equal zeros of opposite
// sign may come back with either sign.
#include <algorithm>
#include <atomic>
#include <climits>
#include <cmath>
#include <mutex>

#include "common.cuh"
#include "fp64_int.cuh"
#include "reduce4.cuh"

namespace nebo {
namespace {

constexpr int RED_THREADS = 256;
constexpr int RED_MAX_BLOCKS = 1024;

struct Acc {
  double s, c;  // sum and running compensation (sum/norm), or the extremum's key in c
};

// a += v, the rounding error kept in a.c (Neumaier; magnitudes compared on the integer pipe)
__device__ __forceinline__ void two_sum_add(Acc& a, double v) {
  const double t = a.s + v;
  const unsigned long long ms = (unsigned long long)__double_as_longlong(a.s) << 1,
                           mv = (unsigned long long)__double_as_longlong(v) << 1;
  const bool big = ms >= mv;
  const double x = big ? a.s : v, y = big ? v : a.s;
  a.c += (x - t) + y;
  a.s = t;
}

// The sum of every thread's s and c as a pair (s: rounded to nearest, c: what that leaves), valid in
// thread 0 of the block (RED_THREADS threads).  With E the largest biased exponent of all of them,
// each becomes an integer in units of 2^(E-1134) (|x| < 2^112; anything down to 2^-59 of the
// largest keeps its 53 bits, the rest is within 2^-113 of it) and the 512 integers add exactly.
// Infinities of one sign give that infinity, others and NaNs NaN (s decides: a compensation beside an
// infinite s is NaN); scales whose result could leave the normal range add in FP64.
__device__ __forceinline__ Acc block_sum(Acc a) {
  __shared__ int she[RED_THREADS / 32];
  __shared__ fixmath::fix128 shs[RED_THREADS / 32];
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  int E = __reduce_max_sync(0xffffffffu, max(fixmath::dexp(a.s), fixmath::dexp(a.c)));
  __syncthreads();  // the arrays may still be read from a previous call
  if (lane == 0) she[wid] = E;
  __syncthreads();
#pragma unroll
  for (int i = 0; i < RED_THREADS / 32; ++i) E = max(E, she[i]);
  if (E < 140 || E > 2020) {  // block-uniform
    if (E == 0x7ff) {
      const long long PINF = 0x7ff0000000000000LL, b = __double_as_longlong(a.s);
      const bool nan = (b & ~(1LL << 63)) > PINF;
      const bool pos = __syncthreads_or(nan || b == PINF), neg = __syncthreads_or(nan || b == (PINF | (1LL << 63)));
      a.s = __longlong_as_double(pos == neg ? 0x7ff8000000000000LL : (pos ? PINF : PINF | (1LL << 63)));
      a.c = 0.0;
      return a;
    }
    if (!__syncthreads_or(((unsigned long long)__double_as_longlong(a.s) << 1) != 0 ||
                          ((unsigned long long)__double_as_longlong(a.c) << 1) != 0)) {
      a.s = a.c = 0.0;
      return a;
    }
    __shared__ Acc sha[RED_THREADS];
    sha[threadIdx.x] = a;
    __syncthreads();
    if (threadIdx.x == 0) {
      Acc r = sha[0];
      for (int i = 1; i < RED_THREADS; ++i) {
        two_sum_add(r, sha[i].s);
        r.c += sha[i].c;
      }
      if (fixmath::dexp(r.s) == 0x7ff) r.c = 0.0;
      a = r;
    }
    return a;
  }
  fixmath::fix128 t = fixmath::to_units(a.s, E + 10) + fixmath::to_units(a.c, E + 10);
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    const unsigned long long lo = __shfl_down_sync(0xffffffffu, (unsigned long long)t, o);
    const long long hi = __shfl_down_sync(0xffffffffu, (long long)(t >> 64), o);
    t += fixmath::make128(hi, lo);
  }
  if (lane == 0) shs[wid] = t;
  __syncthreads();
  if (threadIdx.x == 0) {
    t = shs[0];
#pragma unroll
    for (int i = 1; i < RED_THREADS / 32; ++i) t += shs[i];
    const int u = E + 10 - 1144;
    a.s = fixmath::units_to_double0(t, u);
    a.c = fixmath::units_to_double0(t - fixmath::to_units(a.s, E + 10), u);
  }
  return a;
}

// The largest key of the block, valid in thread 0.
__device__ __forceinline__ long long block_max_key(long long k) {
  __shared__ long long shk[RED_THREADS / 32];
  auto warp_max = [](long long v) {
    const int hi = __reduce_max_sync(0xffffffffu, (int)(v >> 32));
    const unsigned lo = __reduce_max_sync(0xffffffffu, (int)(v >> 32) == hi ? (unsigned)v : 0u);
    return (long long)(((unsigned long long)(unsigned)hi << 32) | lo);
  };
  k = warp_max(k);
  __syncthreads();
  if ((threadIdx.x & 31) == 0) shk[threadIdx.x >> 5] = k;
  __syncthreads();
  if (threadIdx.x < 32) k = warp_max(shk[threadIdx.x & (RED_THREADS / 32 - 1)]);
  return k;
}

// FP32 elements widen exactly through integer operations (a hardware f32 -> f64 conversion issues
// on the FP64 pipe, which the accumulation itself needs).
__device__ __forceinline__ double widen(double v) { return v; }
__device__ __forceinline__ double widen(float v) { return fixmath::f32_to_f64(v); }

// The region of a reduction: rows of w elements, or (flat) one run of w elements.
template <typename T>
struct Region {
  const T* base;  // first element
  long w;         // elements per row; flat: of the region
  int sy;         // row pitch
  long sz;
  int ny;         // rows per plane
  int nrows;      // flat: 0
};

// f8(v[8], m) for batches of up to 8 elements per lane, their loads issued together: v[i] exists
// where bit i of m is set, the others are 0.
template <typename T, class F8>
__device__ __forceinline__ void walk(const Region<T>& g, F8&& f8) {
  auto batch = [&](const T* p, long x, long step) {
    T e[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) e[i] = x + i * step < g.w ? __ldg(p + x + i * step) : T(0);
    double v[8];
    unsigned m = 0;
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      v[i] = widen(e[i]);
      m |= (x + i * step < g.w ? 1u : 0u) << i;
    }
    f8(v, m);
  };
  const int tid = blockIdx.x * RED_THREADS + threadIdx.x;
  const long threads = (long)gridDim.x * RED_THREADS;
  if (g.nrows == 0) {
    for (long x = tid; x < g.w; x += 8 * threads) batch(g.base, x, threads);
    return;
  }
  const int lane = threadIdx.x & 31, nwarps = (int)(threads >> 5);
  for (int r = tid >> 5; r < g.nrows; r += nwarps) {
    const int z = r / g.ny, y = r - z * g.ny;
    const T* row = g.base + (long)g.sy * y + g.sz * z;
    for (long x = lane; x < g.w; x += 256) batch(row, x, 32);
  }
}

// Sum of 8 in pairs (7 FP64 adds), and of their squares (4 multiplies folded into 4 FMAs).
__device__ __forceinline__ double sum8(const double* v) {
  return ((v[0] + v[1]) + (v[2] + v[3])) + ((v[4] + v[5]) + (v[6] + v[7]));
}
__device__ __forceinline__ double sumsq8(const double* v) {
  const double a = fma(v[0], v[0], v[1] * v[1]), b = fma(v[2], v[2], v[3] * v[3]);
  const double c = fma(v[4], v[4], v[5] * v[5]), d = fma(v[6], v[6], v[7] * v[7]);
  return (a + b) + (c + d);
}

// a += the 8 values of q, with their rounding errors (every element counts as in one compensated
// sum).  With E their largest biased exponent each becomes an integer in units of 2^(E-1141); the
// integers add exactly and enter a as a pair: 5 FP64 operations per batch where compensated adds of
// the elements take 5 each (250^3: 137 us of nebo_sum).  Scales whose result could leave the normal
// range, infinities and NaNs take those.
__device__ __forceinline__ void add8(Acc& a, const double* q) {
  unsigned top = 0u;
#pragma unroll
  for (int i = 0; i < 8; ++i) top = max(top, (unsigned)(__double_as_longlong(q[i]) >> 32) & 0x7fffffffu);
  const int E = (int)(top >> 20);
  if (E < 140 || E > 2020) {
    unsigned long long any = 0ull;
#pragma unroll
    for (int i = 0; i < 8; ++i) any |= (unsigned long long)__double_as_longlong(q[i]) << 1;
    if (any) {
#pragma unroll
      for (int i = 0; i < 8; ++i) two_sum_add(a, q[i]);
    }
    return;
  }
  fixmath::fix128 t = 0;
#pragma unroll
  for (int i = 0; i < 8; ++i) t += fixmath::to_units(q[i], E + 3);
  const int u = E + 3 - 1144;
  const double s = fixmath::units_to_double0(t, u);
  two_sum_add(a, s);
  a.c += fixmath::units_to_double0(t - fixmath::to_units(s, E + 3), u);
}

// One thread's share of a reduction: a (sum, compensation) pair, or the extremum's key in c's place.
template <typename T, int OP>
__device__ __forceinline__ Acc reduce_region(const Region<T>& g) {
  constexpr bool ext = OP == NEBO_RED_MAX || OP == NEBO_RED_MIN;
  Acc a{0.0, 0.0};
  long long key = LLONG_MIN;
  walk(g, [&](const double* v, unsigned m) {
    if constexpr (ext) {
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        const long long k = order_key(v[i]);
        // a NaN's key lies outside [key(-inf), key(inf)]; the minimum is the largest ~key
        if ((m >> i & 1u) && k >= KEY_NINF && k <= KEY_PINF) {
          const long long q = OP == NEBO_RED_MAX ? k : ~k;
          key = q > key ? q : key;
        }
      }
    } else {
      double q[8];
#pragma unroll
      for (int i = 0; i < 8; ++i) q[i] = OP == NEBO_RED_NORM ? __dmul_rn(v[i], v[i]) : v[i];
      add8(a, q);
    }
  });
  if constexpr (ext) a.c = __longlong_as_double(key);
  return a;
}

template <int OP>
__device__ __forceinline__ Acc block_acc(Acc a) {
  if constexpr (OP == NEBO_RED_MAX || OP == NEBO_RED_MIN)
    a.c = __longlong_as_double(block_max_key(__double_as_longlong(a.c)));
  else
    a = block_sum(a);
  return a;
}

// The blocks' partials (read through L2) into the result, by one block.
template <int OP>
__device__ __forceinline__ void finish(const Acc* partials, int n, double* out) {
  constexpr bool ext = OP == NEBO_RED_MAX || OP == NEBO_RED_MIN;
  Acc a{0.0, ext ? __longlong_as_double(LLONG_MIN) : 0.0};
  // fixed assignment of partials to threads -> deterministic result
  for (int i = threadIdx.x; i < n; i += RED_THREADS) {
    Acc b;
    b.s = __ldcg(&partials[i].s);
    b.c = __ldcg(&partials[i].c);
    if constexpr (ext) {
      const long long ka = __double_as_longlong(a.c), kb = __double_as_longlong(b.c);
      a.c = __longlong_as_double(ka > kb ? ka : kb);
    } else {
      two_sum_add(a, b.s);
      a.c += b.c;
    }
  }
  a = block_acc<OP>(a);
  if (threadIdx.x == 0) {
    double r;
    if constexpr (ext) {
      const long long k = __double_as_longlong(a.c);
      r = k == LLONG_MIN ? (OP == NEBO_RED_MAX ? -INFINITY : INFINITY) : from_key(OP == NEBO_RED_MAX ? k : ~k);
    } else {
      r = a.s + a.c;
      if (OP == NEBO_RED_NORM) r = sqrt(r);
    }
    *out = r;
  }
}

template <typename T, int OP>
__global__ void __launch_bounds__(RED_THREADS, 4) reduce_rows_kernel(Region<T> g, Acc* __restrict__ partials) {
  const Acc a = block_acc<OP>(reduce_region<T, OP>(g));
  if (threadIdx.x == 0) partials[blockIdx.x] = a;
}

template <int OP>
__global__ void __launch_bounds__(RED_THREADS, 4) reduce_final_kernel(const Acc* __restrict__ partials, int n,
                                                                   double* __restrict__ out) {
  finish<OP>(partials, n, out);
}

// Both passes in one launch for nebo_reduce, which waits for its result: the partials live in one of
// RED_SLOTS fixed slots that the caller holds until then, and the block that draws the last ticket
// (which atomicInc wraps back to 0) finishes.  No block waits for another.
constexpr int RED_SLOTS = 8;
struct Slot {
  Acc partials[RED_MAX_BLOCKS];
  unsigned ticket;
};
__device__ Slot g_slots[RED_SLOTS];

template <typename T, int OP>
__global__ void __launch_bounds__(RED_THREADS, 4) reduce_slot_kernel(Region<T> g, int slot, double* __restrict__ out) {
  __shared__ bool last;
  Slot& s = g_slots[slot];
  const Acc a = block_acc<OP>(reduce_region<T, OP>(g));
  if (threadIdx.x == 0) {
    s.partials[blockIdx.x] = a;
    __threadfence();
    last = atomicInc(&s.ticket, gridDim.x - 1) == gridDim.x - 1;
  }
  __syncthreads();
  if (!last) return;
  __threadfence();
  finish<OP>(s.partials, gridDim.x, out);
}

// Free slots (bit set: taken) and the host words their results go to.
std::atomic<unsigned> g_slots_taken{0};
std::mutex g_slot_mu;
double* g_slot_results = nullptr;

// A free slot and the device address of its host word; false when all are taken or the words cannot
// be had (the caller then takes scratch from the pool).
bool take_slot(int* slot, double** host, double** dev) {
  unsigned taken = g_slots_taken.load();
  for (;;) {
    int i = 0;
    while (i < RED_SLOTS && (taken >> i & 1u)) ++i;
    if (i == RED_SLOTS) return false;
    if (g_slots_taken.compare_exchange_weak(taken, taken | 1u << i)) {
      *slot = i;
      break;
    }
  }
  void* d = nullptr;
  {
    std::lock_guard<std::mutex> g(g_slot_mu);
    // asked every time: a cudaDeviceReset frees the words
    if (!g_slot_results || cudaHostGetDevicePointer(&d, g_slot_results, 0) != cudaSuccess) {
      cudaGetLastError();
      void* p = nullptr;
      d = nullptr;
      g_slot_results = nullptr;
      if (cudaHostAlloc(&p, RED_SLOTS * sizeof(double), cudaHostAllocPortable | cudaHostAllocMapped) == cudaSuccess &&
          cudaHostGetDevicePointer(&d, p, 0) == cudaSuccess)
        g_slot_results = (double*)p;
      else
        cudaGetLastError();
    }
    *host = g_slot_results;
  }
  if (!*host || !d) {
    g_slots_taken.fetch_and(~(1u << *slot));
    return false;
  }
  *host += *slot;
  *dev = (double*)d + *slot;
  return true;
}

// Per-call scratch from the stream-ordered pool: concurrent reductions on different streams
// never share partials.
int scratch_alloc(Acc** partials, double** result, cudaStream_t s) {
  void* p = nullptr;
  pool_retain();
  NEBO_CUDA_TRY(cudaMallocAsync(&p, RED_MAX_BLOCKS * sizeof(Acc) + 64, s));
  *partials = (Acc*)p;
  *result = (double*)((char*)p + RED_MAX_BLOCKS * sizeof(Acc));
  return NEBO_OK;
}

}  // namespace

// Region of a field reduction in glob coordinates: whole window (valid ghosts included) or the
// window minus its valid ghosts (interior, BC cells included), as nebo_fold does.
void reduction_region(const nebo_field& f, int interior, int lo[3], int hi[3]) {
  for (int i = 0; i < 3; ++i) {
    const int gm = f.extent[i] <= 1 ? 0 : f.ghost_minus[i];
    const int gp = f.extent[i] <= 1 ? 0 : f.ghost_plus[i];
    lo[i] = f.offset[i] + (interior ? gm : 0);
    hi[i] = f.offset[i] + f.extent[i] - (interior ? gp : 0);
  }
}

namespace {

// The region of a reduction and the blocks that walk it (8 elements per thread, at most four blocks
// per SM and max_blocks); 0 blocks: empty.
template <typename T>
int plan(const nebo_field& f, int interior, int max_blocks, Region<T>* g) {
  int lo[3], hi[3];
  reduction_region(f, interior, lo, hi);
  const long nrows = (long)(hi[1] - lo[1]) * (hi[2] - lo[2]), w = hi[0] - lo[0];
  if (hi[1] <= lo[1] || nrows <= 0 || w <= 0) return 0;
  g->sy = f.glob[0];
  g->sz = (long)f.glob[0] * f.glob[1];
  g->base = (const T*)f.data + lo[0] + (long)g->sy * lo[1] + g->sz * lo[2];
  g->ny = hi[1] - lo[1];
  const bool flat = w == f.glob[0] && (hi[2] - lo[2] == 1 || g->ny == f.glob[1]);
  g->w = flat ? w * nrows : w;
  g->nrows = flat ? 0 : (int)nrows;
  const long want = flat ? (g->w + 8 * RED_THREADS - 1) / (8 * RED_THREADS) : (nrows + RED_THREADS / 32 - 1) / (RED_THREADS / 32);
  return (int)std::min(want, std::min((long)num_sms() * 4, (long)max_blocks));
}

template <typename T>
void launch_rows(const Region<T>& g, int op, int blocks, Acc* partials, cudaStream_t s) {
  switch (op) {
    case NEBO_RED_SUM: reduce_rows_kernel<T, NEBO_RED_SUM><<<blocks, RED_THREADS, 0, s>>>(g, partials); break;
    case NEBO_RED_MAX: reduce_rows_kernel<T, NEBO_RED_MAX><<<blocks, RED_THREADS, 0, s>>>(g, partials); break;
    case NEBO_RED_MIN: reduce_rows_kernel<T, NEBO_RED_MIN><<<blocks, RED_THREADS, 0, s>>>(g, partials); break;
    default: reduce_rows_kernel<T, NEBO_RED_NORM><<<blocks, RED_THREADS, 0, s>>>(g, partials);
  }
}
void launch_final(int op, const Acc* partials, int n, double* out, cudaStream_t s) {
  switch (op) {
    case NEBO_RED_SUM: reduce_final_kernel<NEBO_RED_SUM><<<1, RED_THREADS, 0, s>>>(partials, n, out); break;
    case NEBO_RED_MAX: reduce_final_kernel<NEBO_RED_MAX><<<1, RED_THREADS, 0, s>>>(partials, n, out); break;
    case NEBO_RED_MIN: reduce_final_kernel<NEBO_RED_MIN><<<1, RED_THREADS, 0, s>>>(partials, n, out); break;
    default: reduce_final_kernel<NEBO_RED_NORM><<<1, RED_THREADS, 0, s>>>(partials, n, out);
  }
}
template <typename T>
void launch_slot(const Region<T>& g, int op, int blocks, int slot, double* out, cudaStream_t s) {
  switch (op) {
    case NEBO_RED_SUM: reduce_slot_kernel<T, NEBO_RED_SUM><<<blocks, RED_THREADS, 0, s>>>(g, slot, out); break;
    case NEBO_RED_MAX: reduce_slot_kernel<T, NEBO_RED_MAX><<<blocks, RED_THREADS, 0, s>>>(g, slot, out); break;
    case NEBO_RED_MIN: reduce_slot_kernel<T, NEBO_RED_MIN><<<blocks, RED_THREADS, 0, s>>>(g, slot, out); break;
    default: reduce_slot_kernel<T, NEBO_RED_NORM><<<blocks, RED_THREADS, 0, s>>>(g, slot, out);
  }
}

// Both passes on s with the given partials (room for RED_MAX_BLOCKS).
template <typename T>
int reduce_two_pass(const nebo_field* f, int op, int interior, double* d_result, Acc* partials, const char* what,
                    cudaStream_t s) {
  Region<T> g;
  const int blocks = plan(*f, interior, RED_MAX_BLOCKS, &g);
  if (!blocks) return fail(NEBO_ERR_INVALID, "Nebo error in %s: empty region", what);
  {
    LaunchScope ls("reduce_rows", s);
    launch_rows(g, op, blocks, partials, s);
  }
  {
    LaunchScope ls("reduce_final", s);
    launch_final(op, partials, blocks, d_result, s);
  }
  NEBO_LAUNCH_CHECK(what);
  return NEBO_OK;
}

}  // namespace

int reduce_field_into(const nebo_field* f, int op, int interior, double* d_result, Acc* partials, const char* what,
                      cudaStream_t s) {
  return f->dtype == NEBO_F64 ? reduce_two_pass<double>(f, op, interior, d_result, partials, what, s)
                              : reduce_two_pass<float>(f, op, interior, d_result, partials, what, s);
}

static int check_reduce_args(const nebo_field* f, int op) {
  int rc = check_field(f, "nebo_reduce");
  if (rc) return rc;
  if (op < NEBO_RED_SUM || op > NEBO_RED_NORM) return fail(NEBO_ERR_INVALID, "Nebo error in nebo_reduce: bad op %d", op);
  return NEBO_OK;
}

}  // namespace nebo

using namespace nebo;

extern "C" int nebo_reduce_async(const nebo_field* f, int op, int interior, double* d_result, nebo_stream_t stream) {
  int rc = check_reduce_args(f, op);
  if (rc) return rc;
  if (!d_result) return fail(NEBO_ERR_INVALID, "Nebo error in nebo_reduce_async: null result pointer");
  Acc* partials;
  double* dres;
  cudaStream_t s = (cudaStream_t)stream;
  if ((rc = scratch_alloc(&partials, &dres, s))) return rc;
  rc = reduce_field_into(f, op, interior, d_result, partials, "nebo_reduce", s);
  cudaFreeAsync(partials, s);
  return rc;
}

extern "C" int nebo_reduce(const nebo_field* f, int op, int interior, double* result, nebo_stream_t stream) {
  int rc = check_reduce_args(f, op);
  if (rc) return rc;
  if (!result) return fail(NEBO_ERR_INVALID, "Nebo error in nebo_reduce: null result pointer");
  cudaStream_t s = (cudaStream_t)stream;
  int slot;
  double *hres, *sres;
  if (take_slot(&slot, &hres, &sres)) {  // held until the result has been read
    auto one_pass = [&](auto g) -> int {
      const int blocks = plan(*f, interior, RED_MAX_BLOCKS, &g);
      if (!blocks) return fail(NEBO_ERR_INVALID, "Nebo error in nebo_reduce: empty region");
      {
        LaunchScope ls("reduce_slot", s);
        launch_slot(g, op, blocks, slot, sres, s);
      }
      // whatever the launch check says, a kernel that did start has left the slot before it is free
      const cudaError_t launched = cudaGetLastError(), ended = cudaStreamSynchronize(s);
      if (launched != cudaSuccess || ended != cudaSuccess)
        return cuda_fail(launched != cudaSuccess ? launched : ended, "nebo_reduce");
      *result = *(volatile double*)hres;
      return NEBO_OK;
    };
    rc = f->dtype == NEBO_F64 ? one_pass(Region<double>{}) : one_pass(Region<float>{});
    g_slots_taken.fetch_and(~(1u << slot));
    return rc;
  }
  Acc* partials;
  double* dres;
  if ((rc = scratch_alloc(&partials, &dres, s))) return rc;
  rc = reduce_field_into(f, op, interior, dres, partials, "nebo_reduce", s);
  if (!rc) {
    cudaError_t e = cudaMemcpyAsync(result, dres, sizeof(double), cudaMemcpyDeviceToHost, s);
    if (e != cudaSuccess) rc = cuda_fail(e, "nebo_reduce copy");
  }
  cudaFreeAsync(partials, s);
  if (rc) return rc;
  NEBO_CUDA_TRY(cudaStreamSynchronize(s));
  return NEBO_OK;
}

// ------------------------------------------------------------------------------------------
// Reduction without any allocation.
//
// nebo_reduce / nebo_reduce_async take their block partials from the stream-ordered pool on
// every call.  Callers that must not enter the CUDA allocator at that point (a host framework
// that has reserved the device memory up front in its own pool, so a further cudaMalloc fails or
// breaks its accounting; code that runs where the allocator may not be entered) use
// nebo_reduce_noalloc instead: the same two kernels, with the partials in the fixed array below.
//
// The array lives in this module's device memory for every GPU that loads the library, until the
// process exits.  Host code cannot use the symbol's name as a device address, so the first call
// on each device (with that device current) looks the address up with cudaGetSymbolAddress and
// caches it (a cudaDeviceReset voids the cached address: a process that resets a device must not
// call this entry point on it afterwards); that first call should come before any stream capture.
// A reduction takes at most 1024 blocks, one slot each.  All calls share the array
// and it keeps the last call's contents: pass 1 writes every slot that pass 2 reads, so nothing
// needs clearing, but calls whose kernels overlap on the GPU (different streams, no ordering
// between them) race on it.
namespace nebo {
namespace {

constexpr int NOALLOC_MAX_PARTIALS = 1024;  // 16 KiB: one (sum, compensation) pair per block
constexpr long NOALLOC_MAX_ROWS = 2147483647L;  // rows (y * z) of the reduced region
constexpr int NOALLOC_MAX_DEVICES = 64;
static __device__ __align__(256) Acc g_noalloc_partials[NOALLOC_MAX_PARTIALS];

std::mutex g_noalloc_mu;
Acc* g_noalloc_addr[NOALLOC_MAX_DEVICES] = {nullptr};

int noalloc_partials(Acc** out) {
  int dev = 0;
  NEBO_CUDA_TRY(cudaGetDevice(&dev));
  if (dev < 0 || dev >= NOALLOC_MAX_DEVICES)
    return fail(NEBO_ERR_UNSUPPORTED, "Nebo error in nebo_reduce_noalloc: device index %d beyond %d", dev,
                NOALLOC_MAX_DEVICES);
  std::lock_guard<std::mutex> g(g_noalloc_mu);
  if (!g_noalloc_addr[dev]) {
    void* p = nullptr;
    cudaError_t e = cudaGetSymbolAddress(&p, g_noalloc_partials);
    if (e != cudaSuccess) return cuda_fail(e, "nebo_reduce_noalloc (cudaGetSymbolAddress)");
    g_noalloc_addr[dev] = static_cast<Acc*>(p);
  }
  *out = g_noalloc_addr[dev];
  return NEBO_OK;
}

}  // namespace
}  // namespace nebo

extern "C" int nebo_reduce_noalloc(const nebo_field* f, int op, int interior, double* d_result,
                                   nebo_stream_t stream) {
  int rc = check_reduce_args(f, op);
  if (rc) return rc;
  if (!d_result) return fail(NEBO_ERR_INVALID, "Nebo error in nebo_reduce_noalloc: null result pointer");
  int lo[3], hi[3];
  reduction_region(*f, interior, lo, hi);
  const long nrows = (long)(hi[1] - lo[1]) * (hi[2] - lo[2]);
  if (nrows <= 0 || hi[0] <= lo[0]) return fail(NEBO_ERR_INVALID, "Nebo error in nebo_reduce_noalloc: empty region");
  // The row walk takes an int row count; larger regions are refused before any CUDA call.
  if (nrows > NOALLOC_MAX_ROWS)
    return fail(NEBO_ERR_INVALID,
                "Nebo error in nebo_reduce_noalloc: the region has %ld rows, more than the %ld this entry point takes",
                nrows, (long)NOALLOC_MAX_ROWS);
  // One partial slot per block, and never more blocks than slots (plan): the strided walk covers any
  // region with fewer blocks, so the fixed array suffices whatever the SM count.
  static_assert(RED_MAX_BLOCKS <= NOALLOC_MAX_PARTIALS, "one slot per block");
  Acc* partials = nullptr;
  if ((rc = noalloc_partials(&partials))) return rc;
  return reduce_field_into(f, op, interior, d_result, partials, "nebo_reduce_noalloc", (cudaStream_t)stream);
}

// ------------------------------------------------------------------------------------------
// All four reductions in one pass over the field (nebo_sum, nebo_max, nebo_min, nebo_norm of
// the same region), for callers that need several of them: the field is read once instead of
// four times.  FP64 is the scarce unit on this GPU, so each element costs two FP64 operations
// (one add for the sum, one fused multiply-add for the sum of squares); max and min compare
// order-preserving 64-bit integer keys of the doubles on the integer pipe.  Per-thread partial
// sums are plain (at most a few hundred terms each); partials are combined with Neumaier
// compensation.  NaNs are skipped by max/min, as the reference's comparisons skip them; equal
// zeros of opposite sign may come back with either sign.
namespace nebo {
namespace {

__device__ __forceinline__ Acc4 block_acc4(Acc4 a) {
  const Acc s = block_sum(Acc{a.s, a.sc}), q = block_sum(Acc{a.q, a.qc});
  return Acc4{s.s, s.c, q.s, q.c, block_max_key(a.mx), ~block_max_key(~a.mn)};
}

template <typename T>
__global__ void __launch_bounds__(RED_THREADS, 4) reduce4_rows_kernel(Region<T> g, Acc4* __restrict__ partials) {
  Acc4 a = acc4_identity();
  walk(g, [&](const double* v, unsigned m) {
    a.s += sum8(v);
    a.q += sumsq8(v);
#pragma unroll
    for (int i = 0; i < 8; ++i)
      if (m >> i & 1u) keys_add(a.mx, a.mn, order_key(v[i]));  // NaNs never win a comparison
  });
  a = block_acc4(a);
  if (threadIdx.x == 0) partials[blockIdx.x] = a;
}

// out = {sum, max, min, norm} of the partial accumulators (one block).
__global__ void __launch_bounds__(RED_THREADS, 4) reduce4_final_kernel(const Acc4* __restrict__ partials, int n,
                                                                    double* __restrict__ out) {
  Acc4 a = acc4_identity();
  for (int i = threadIdx.x; i < n; i += RED_THREADS) merge4(a, partials[i]);
  a = block_acc4(a);
  if (threadIdx.x == 0) {
    out[0] = pair_sum(a.s, a.sc);
    out[1] = a.mx == LLONG_MIN ? -INFINITY : from_key(a.mx);
    out[2] = a.mn == LLONG_MAX ? INFINITY : from_key(a.mn);
    out[3] = sqrt(pair_sum(a.q, a.qc));
  }
}

template <typename T>
int reduce4_two_pass(const nebo_field* f, int interior, double* d_out4, cudaStream_t s) {
  Region<T> g;
  const int blocks = plan(*f, interior, RED_MAX_BLOCKS, &g);
  if (!blocks) return fail(NEBO_ERR_INVALID, "Nebo error in nebo_reduce_all: empty region");
  Acc4* partials = nullptr;
  pool_retain();
  NEBO_CUDA_TRY(cudaMallocAsync((void**)&partials, sizeof(Acc4) * blocks, s));
  {
    LaunchScope ls("reduce4_rows", s);
    reduce4_rows_kernel<T><<<blocks, RED_THREADS, 0, s>>>(g, partials);
  }
  {
    LaunchScope ls("reduce4_final", s);
    reduce4_final_kernel<<<1, RED_THREADS, 0, s>>>(partials, blocks, d_out4);
  }
  const cudaError_t le = cudaGetLastError();
  cudaFreeAsync(partials, s);
  if (le != cudaSuccess) return cuda_fail(le, "nebo_reduce_all");
  return NEBO_OK;
}

}  // namespace
}  // namespace nebo

extern "C" int nebo_reduce_all(const nebo_field* f, int interior, double* d_out4, nebo_stream_t stream) {
  int rc = check_reduce_args(f, NEBO_RED_SUM);
  if (rc) return rc;
  if (!d_out4) return fail(NEBO_ERR_INVALID, "Nebo error in nebo_reduce_all: null result pointer");
  cudaStream_t s = (cudaStream_t)stream;
  return f->dtype == NEBO_F64 ? reduce4_two_pass<double>(f, interior, d_out4, s)
                              : reduce4_two_pass<float>(f, interior, d_out4, s);
}
