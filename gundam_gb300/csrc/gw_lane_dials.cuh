// gw_lane_dials.cuh -- dial evaluation of the lanes-over-points kernel
// (gw_lanes.cu): one dial at a lane's KR points, from the tile's pre-decoded
// headers (make_lane_header) and its payload by 32-bit shared-memory addresses.
// The arithmetic is that of gw_dials.cuh; what differs is the index work around
// it, which is most of a warp's instructions (64 points, warp instructions per
// dial with the generic dial_values and now: grid dial 67 -> 47, general spline
// 229 -> 197, graph 205 -> 144, bilinear surface 266 -> 222, norm 56 -> 26).
#pragma once
#include "gw_device.cuh"

namespace gw {
namespace {

// Shared-memory loads by 32-bit address (the address of a generic pointer takes
// two registers and 64-bit arithmetic).
__device__ __forceinline__ uint2 lds64(uint32_t a) {
  uint2 r;
  asm volatile("ld.shared.v2.u32 {%0, %1}, [%2];" : "=r"(r.x), "=r"(r.y) : "r"(a));
  return r;
}
__device__ __forceinline__ uint4 lds128(uint32_t a) {
  uint4 r;
  asm volatile("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(r.x), "=r"(r.y), "=r"(r.z), "=r"(r.w) : "r"(a));
  return r;
}

template <typename T>
__device__ __forceinline__ T lds(uint32_t a) {
  T r;
  if constexpr (sizeof(T) == 4) {
    asm volatile("ld.shared.f32 %0, [%1];" : "=f"(r) : "r"(a));
  } else if constexpr (kIsDf<T>) {
    asm volatile("ld.shared.v2.f32 {%0, %1}, [%2];" : "=f"(r.hi), "=f"(r.lo) : "r"(a));
  } else {
    asm volatile("ld.shared.f64 %0, [%1];" : "=d"(r) : "r"(a));
  }
  return r;
}

// Coefficient block of a grid dial (16-byte aligned, as the payloads are).
__device__ __forceinline__ float block_cubic(uint32_t a, float u) {
  const uint4 q = lds128(a);
  return __uint_as_float(q.x) +
         u * (__uint_as_float(q.y) + u * (__uint_as_float(q.z) + u * __uint_as_float(q.w)));
}
__device__ __forceinline__ double block_cubic(uint32_t a, double u) {
  const uint4 p = lds128(a), q = lds128(a + 16);
  const double c0 = __hiloint2double((int)p.y, (int)p.x), c1 = __hiloint2double((int)p.w, (int)p.z);
  const double c2 = __hiloint2double((int)q.y, (int)q.x), c3 = __hiloint2double((int)q.w, (int)q.z);
  return c0 + u * (c1 + u * (c2 + u * c3));
}
__device__ __forceinline__ dfloat block_cubic(uint32_t a, dfloat u) {
  const uint4 p = lds128(a), q = lds128(a + 16);
  auto f = [](uint32_t h, uint32_t l) { return dfloat(__uint_as_float(h), __uint_as_float(l)); };
  return f(p.x, p.y) + u * (f(p.z, p.w) + u * (f(q.x, q.y) + u * f(q.z, q.w)));
}

// Address of the record of the interval that holds x, among n - 1 intervals
// whose knots lie at key, key + stride, ...: the last of the records 0 .. n - 2
// whose knot is below x (`strict`; else not above x), or record 0.  Halving
// steps that stay in range, the same for every point of a dial: a load, a
// comparison and a select per point and step, where the five-step searches of
// eval_general and eval_graph test every candidate's index as well.  Knots do
// not decrease, so both find the same interval.
template <typename T, int KR, bool strict>
__device__ __forceinline__ void find_interval(uint32_t rec, uint32_t key, int stride, int n, const T (&x)[KR],
                                              uint32_t (&a)[KR]) {
#pragma unroll
  for (int j = 0; j < KR; ++j) a[j] = rec;
  for (int len = n - 1; len > 1;) {
    const int half = len >> 1;
    const uint32_t by = (uint32_t)(half * stride);
#pragma unroll
    for (int j = 0; j < KR; ++j) {
      const T k = lds<T>(a[j] + by + key);
      if (strict ? above(x[j], k) : !above(k, x[j])) a[j] += by;
    }
    len -= half;
  }
}

// General spline at KR points: eval_general's operations on the interval.
template <typename T, int KR>
__device__ __forceinline__ void general_values(uint32_t d, int n, const T (&xin)[KR], bool trunc, T (&val)[KR]) {
  constexpr uint32_t S = (uint32_t)sizeof(T);
  T x[KR];
#pragma unroll
  for (int j = 0; j < KR; ++j) x[j] = xin[j];
  if (trunc) {
    const T lo = lds<T>(d + 2 * S), hi = lds<T>(d + (3 * (n - 1) + 2) * S);
#pragma unroll
    for (int j = 0; j < KR; ++j) {
      if (x[j] <= lo) x[j] = lo;
      else if (x[j] >= hi) x[j] = hi;
    }
  }
  uint32_t a[KR];
  find_interval<T, KR, true>(d, 2 * S, 3 * S, n, x, a);
#pragma unroll
  for (int j = 0; j < KR; ++j) {
    const T p1 = lds<T>(a[j]), s1 = lds<T>(a[j] + S), x1 = lds<T>(a[j] + 2 * S);
    const T p2 = lds<T>(a[j] + 3 * S), s2 = lds<T>(a[j] + 4 * S), x2 = lds<T>(a[j] + 5 * S);
    const T step = x2 - x1;
    const T fx = fdiv(x[j] - x1, step);
    const T m1 = s1 * step;
    const T m2 = s2 * step;
    val[j] = hermite(p1, m1, p2, m2, fx);
  }
}

// Graph at KR points: eval_graph's operations on the interval.
template <typename T, int KR>
__device__ __forceinline__ void graph_values(uint32_t d, int n, const T (&x)[KR], bool trunc, T (&val)[KR]) {
  constexpr uint32_t S = (uint32_t)sizeof(T);
  if (n < 2) {
    const T y = lds<T>(d);
#pragma unroll
    for (int j = 0; j < KR; ++j) val[j] = y;
    return;
  }
  uint32_t a[KR];
  find_interval<T, KR, true>(d, S, 2 * S, n, x, a);
#pragma unroll
  for (int j = 0; j < KR; ++j) {
    const T p1 = lds<T>(a[j]), x1 = lds<T>(a[j] + S), p2 = lds<T>(a[j] + 2 * S), x2 = lds<T>(a[j] + 3 * S);
    const T step = x2 - x1;
    const T fx = fdiv(x[j] - x1, step);
    const T m = p2 - p1;
    val[j] = p1 + fx * m;
  }
  if (trunc) {
    const T y0 = lds<T>(d), x0 = lds<T>(d + S);
    const T yn = lds<T>(d + (2 * n - 2) * S), xn = lds<T>(d + (2 * n - 1) * S);
#pragma unroll
    for (int j = 0; j < KR; ++j) {
      if (x[j] <= x0) val[j] = y0;
      else if (x[j] >= xn) val[j] = yn;
    }
  }
}

// Bilinear surface at KR points: eval_bilinear's operations on the facet.
template <typename T, int KR>
__device__ __forceinline__ void bilinear_values(uint32_t d, const T (&xin)[KR], const T (&yin)[KR], bool trunc,
                                                T (&val)[KR]) {
  constexpr uint32_t S = (uint32_t)sizeof(T);
  const int nx = (int)lds<T>(d), ny = (int)lds<T>(d + S);
  const uint32_t xx = d + 2 * S, yy = xx + nx * S, z = yy + ny * S;
  T x[KR], y[KR];
#pragma unroll
  for (int j = 0; j < KR; ++j) {
    x[j] = xin[j];
    y[j] = yin[j];
  }
  if (trunc) {
    const T x0 = lds<T>(xx), xn = lds<T>(xx + (nx - 1) * S), y0 = lds<T>(yy), yn = lds<T>(yy + (ny - 1) * S);
#pragma unroll
    for (int j = 0; j < KR; ++j) {
      if (x[j] < x0) x[j] = x0;
      if (x[j] > xn) x[j] = xn;
      if (y[j] < y0) y[j] = y0;
      if (y[j] > yn) y[j] = yn;
    }
  }
  uint32_t ax[KR], ay[KR];
  find_interval<T, KR, false>(xx, 0u, (int)S, nx, x, ax);
  find_interval<T, KR, false>(yy, 0u, (int)S, ny, y, ay);
#pragma unroll
  for (int j = 0; j < KR; ++j) {
    const uint32_t row = z + (ax[j] - xx) * (uint32_t)ny + (ay[j] - yy), up = row + (uint32_t)ny * S;
    const T ka[2] = {lds<T>(ax[j]), lds<T>(ax[j] + S)}, kb[2] = {lds<T>(ay[j]), lds<T>(ay[j] + S)};
    const T q[4] = {lds<T>(row), lds<T>(row + S), lds<T>(up), lds<T>(up + S)};
    val[j] = bilinear_facet(q, 2, ka, kb, x[j], y[j]);
  }
}

// A parameter's values at the points k0, k0 + kstep, ...
template <typename T, int KR>
__device__ __forceinline__ void points_of(const DevView& v, uint32_t par, int k0, int kstep, T (&x)[KR]) {
  const T* p = (const T*)v.x + (par * (uint32_t)v.kpad + (uint32_t)k0);
#pragma unroll
  for (int j = 0; j < KR; ++j) x[j] = p[j * kstep];
}

// The intervals and fractions of a knot grid at those points, and the values of
// a dial on the grid, before the response clamp (pl: the tile's payload).
template <typename T, int KR>
struct GridPoints {
  GridPoint<T> g[KR];
};
template <typename T, int KR>
__device__ __forceinline__ void grid_points(const DevView& v, uint32_t grid, int k0, int kstep, GridPoints<T, KR>& r) {
  const GridPoint<T>* gp = (const GridPoint<T>*)v.grid_pts + (grid * (uint32_t)v.kpad + (uint32_t)k0);
#pragma unroll
  for (int j = 0; j < KR; ++j) r.g[j] = gp[j * kstep];
}
template <typename T, int KR>
__device__ __forceinline__ void grid_values(uint32_t h, uint32_t pl, const GridPoints<T, KR>& r, T (&val)[KR]) {
  const uint32_t a = pl + lhdr_off(h);
#pragma unroll
  for (int j = 0; j < KR; ++j) val[j] = block_cubic(a + (uint32_t)r.g[j].jb * (uint32_t)sizeof(T), r.g[j].u);
}

// Response clamp of a dial: the common [0, 1e20], a table's, a grid's, the
// parameter's as given (norm dials) or within [-1e20, 1e20] (Calculate*.h).
// The common one (the default lower bound of a dial collection, no upper bound)
// is known from the header, so that nothing is loaded.  Checking the bits of an
// event's responses instead of clamping each, and evaluating an event again
// when one had left the range, saved three instructions a dial but cost more:
// of 64 draws from the prior some parameter lies beyond its knots in most events.
template <typename T, int KR>
__device__ __forceinline__ void clamp_common(T (&val)[KR]) {
#pragma unroll
  for (int j = 0; j < KR; ++j) val[j] = clamp_response(val[j], T(0.0f), T(1e20));
}
// The largest value of a type, the upper clamp of a parameter without one.
template <typename T>
__device__ __forceinline__ T open_bound() {
  return sizeof(T) == 4 ? T(FLT_MAX) : T(DBL_MAX);
}

// Tabulated.h:27-28 and Kriged.cpp:14-21, clamped to the table's bounds (q: the
// table; d, n: the dial's payload); per-point tables are laid out [entry][kpad].
template <typename T, int KR>
__device__ __forceinline__ void table_values(const DevView& v, int type, uint32_t q, const T* d, int n, int k0,
                                             int kstep, T (&val)[KR]) {
  const TableDesc td = v.tables[q];
  const int64_t st = td.per_k ? v.kpad : 1;
  const T* tab = (const T*)v.table_arena + td.offset;
  const T lo = (T)td.lower, hi = (T)td.upper;
#pragma unroll
  for (int j = 0; j < KR; ++j) {
    const int64_t kk = td.per_k ? (int64_t)(k0 + j * kstep) : 0;
    if (type == kTabulated) {
      const T f = d[0];
      const int idx = (int)d[1];
      val[j] = f * tab[idx * st + kk] + (T(1) - f) * tab[(idx + 1) * st + kk];
    } else {
      T a = T(0);
      for (int i = 0; i < n; ++i) a += d[n + i] * tab[(int64_t)(int)d[i] * st + kk];
      val[j] = a;
    }
  }
#pragma unroll
  for (int j = 0; j < KR; ++j) val[j] = clamp_response(val[j], lo, hi);
}

// The responses of a parameter's dials, before the response clamp (da, d: the
// dial's payload).
template <typename T, int KR>
__device__ __forceinline__ void parameter_values(const DevView& v, uint32_t h, uint32_t hy, uint32_t da, const T* d,
                                                 int k0, int kstep, T (&val)[KR]) {
  const int type = lhdr_type(h), n = lhdr_n(h);
  const bool trunc = (h & kLhTrunc) != 0;
  T x[KR];
  points_of<T, KR>(v, hy & 0xFFFFu, k0, kstep, x);
  if (type == kGeneral) {
    general_values<T, KR>(da, n, x, trunc, val);
  } else if (type == kGraph) {
    graph_values<T, KR>(da, n, x, trunc, val);
  } else if (type == kNorm) {
#pragma unroll
    for (int j = 0; j < KR; ++j) val[j] = x[j];
  } else if (type == kBilinear || type == kBicubic) {
    T y[KR];
    points_of<T, KR>(v, hy >> 16, k0, kstep, y);
    if (type == kBilinear) {
      bilinear_values<T, KR>(da, x, y, trunc, val);
    } else {
#pragma unroll
      for (int j = 0; j < KR; ++j) val[j] = eval_bicubic<T>(d, x[j], y[j], trunc);
    }
  } else if (v.spline_coefs) {  // monotonic, uniform and compact splines outside the grids
    coef_values<T, KR>(d, n, x, trunc, val);
  } else if (v.spline_knots && type == kMonotonic) {
#pragma unroll
    for (int j = 0; j < KR; ++j) val[j] = eval_knots<T, true>(d, n, x[j], trunc);
  } else if (v.spline_knots && type == kCompact) {
#pragma unroll
    for (int j = 0; j < KR; ++j) val[j] = eval_knots<T, false>(d, n, x[j], trunc);
  } else if (type == kUniform) {
    prepared_values<T, false, KR>(d, n, x, trunc, val);
  } else {
    prepared_values<T, true, KR>(d, n, x, trunc, val);
  }
}

// The clamped responses of the dials that the kernel has no shorter path for (h,
// hy: the header's two words; pl, base: the tile's payload; g: a grid dial's
// points, when `have_grid`).  A clamp that is not the common one is loaded before the
// response is formed (kEarly) or after it, see k_batched.
template <typename T, int KR, bool have_grid, bool kEarly>
__device__ __forceinline__ void other_values(const DevView& v, uint32_t h, uint32_t hy, uint32_t pl, const T* base,
                                             int k0, int kstep, GridPoints<T, KR>& g, T (&val)[KR]) {
  using V2 = typename Vec2<T>::type;
  const int type = lhdr_type(h);
  const uint32_t da = pl + lhdr_off(h), q = hy & 0xFFFFu;
  const T* d = kEarly ? (const T*)((const unsigned char*)base + lhdr_off(h))
                      : reinterpret_cast<const T*>(__cvta_shared_to_generic(da));
  auto grid = [&]() {
    if constexpr (!have_grid) grid_points<T, KR>(v, q, k0, kstep, g);
    grid_values<T, KR>(h, pl, g, val);
  };
  auto clamp = [&](const V2& c) {
    T lo = c.x, hi = c.y;
    if (type != kNorm && type != kGrid) {
      if (lo < T(-1e20)) lo = T(-1e20);
      if (hi > T(1e20)) hi = T(1e20);
    }
#pragma unroll
    for (int j = 0; j < KR; ++j) val[j] = clamp_response(val[j], lo, hi);
  };
  const bool common = (h & kLhCommonClamp) && type != kNorm;
  if constexpr (kEarly) {
    if (type >= kTabulated) {
      if (type == kGrid) {
        const V2 c = ((const V2*)v.grid_clamp)[q];
        grid();
        clamp(c);
      } else {
        table_values<T, KR>(v, type, q, d, lhdr_n(h), k0, kstep, val);
      }
      return;
    }
    V2 c;
    if (!common) c = ((const V2*)v.pclamp)[q];
    parameter_values<T, KR>(v, h, hy, da, d, k0, kstep, val);
    if (common) clamp_common<T, KR>(val);
    else clamp(c);
  } else {
    if (type == kGrid) {
      grid();
    } else if (type >= kTabulated) {
      table_values<T, KR>(v, type, q, d, lhdr_n(h), k0, kstep, val);
      return;
    } else {
      parameter_values<T, KR>(v, h, hy, da, d, k0, kstep, val);
    }
    if (common) clamp_common<T, KR>(val);
    else clamp(((const V2*)(type == kGrid ? v.grid_clamp : v.pclamp))[q]);
  }
}

}  // namespace
}  // namespace gw
