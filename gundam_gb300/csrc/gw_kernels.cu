// gw_kernels.cu -- the sm_103a kernels of the reweighting engine.
//
// One likelihood evaluation of K parameter points is four launches:
//   k_params    mirror the parameters (DialInputBuffer.cpp:44-89) and compute
//               the prior penalty (LikelihoodInterface.cpp:186-215);
//   k_table_fn  (only with device table functions) refill per-point tables;
//   k_plain / k_batched
//               stream the bin-sorted tiles through shared memory with bulk
//               (TMA) copies, evaluate every dial, form each event's weight as
//               an ordered product (EventDialCache.cpp:156-171) and reduce the
//               weights and squared weights per (tile, bin) in FP64;
//   k_bins_llh  add the (tile, bin) partial sums of each bin in a fixed order
//               (Histogram.cpp:107-135), evaluate the per-bin likelihood
//               (PoissonLogLikelihood.h:19-53 / BarlowBeestonBanff2022.h:150-294)
//               and reduce it, deterministically, to one value per point.
// The reference needs ~1 + n_types + 2*(2 + log2 max bin occupancy) launches
// for the same work (CacheWeights.cpp:153-183, CacheRecursiveSums.cpp:282-352).
#include <algorithm>
#include <mutex>

#include "gw.h"
#include "gw_device.cuh"

namespace gw {
namespace {

// ---------------------------------------------------------------------------
// Parameter update: mirror into the dial inputs, prior penalty.
// ---------------------------------------------------------------------------
// Grid (K, 1 + n_pen): block (k, 0) mirrors the parameters of point k and forms
// its knot-grid intervals; block (k, 1 + q) forms the part of the penalty
// delta^T C^-1 delta that rows [q, q + 1) * kPenRows of C^-1 give.
//
// The penalty is P^2 FP64 multiply-adds per point, and an SM issues two of them
// per cycle: as one block (one thread per row, rows read with a stride of P)
// it took 38 us at P = 200, a sixth of a K = 1 evaluation of 1M events.  Cut
// over blocks of kPenRows rows, thread p taking column p (coalesced), the
// launch takes 6.8 us at K = 1 and 15 us at K = 64.  The parts are added in
// a fixed order by k_bins_llh.
template <typename T>
__global__ void __launch_bounds__(256) k_params(const DevView v, const double* __restrict__ params) {
  extern __shared__ double sp[];  // raw parameter vector of point k [, original values]
  dep_launch();  // not itself a dependent launch: what it reads was complete before it started
  const int k = blockIdx.x;
  const int P = v.n_params;
  if (blockIdx.y > 0) {
    // on the parameters as given (the eigen parameters of decomposed blocks,
    // as the reference's penalty in eigen mode); u_p = sum_j C^-1[j][p] delta_j
    for (int p = threadIdx.x; p < P; p += blockDim.x) sp[p] = params[(size_t)k * P + p] - v.prior_mean[p];
    __syncthreads();
    const int j0 = ((int)blockIdx.y - 1) * kPenRows, j1 = min(P, j0 + kPenRows);
    double acc = 0;
    for (int p = threadIdx.x; p < P; p += blockDim.x) {
      const double* col = v.prior_icov + (size_t)j0 * P + p;
      double c[kPenRows];
#pragma unroll
      for (int j = 0; j < kPenRows; ++j) c[j] = j0 + j < j1 ? col[(size_t)j * P] : 0.0;
      double u = 0;
#pragma unroll
      for (int j = 0; j < kPenRows; ++j)
        if (j0 + j < j1) u += c[j] * sp[j0 + j];
      acc += sp[p] * u;
    }
    __shared__ double red[8];
    for (int o = 16; o; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (lane == 0) red[warp] = acc;
    __syncthreads();
    if (threadIdx.x == 0) {
      double t = 0;
      for (int w = 0; w < 8; ++w) t += red[w];
      v.penalty[(size_t)(blockIdx.y - 1) * v.kpad + k] = t;
    }
    return;
  }
  for (int p = threadIdx.x; p < P; p += blockDim.x) sp[p] = params[(size_t)k * P + p];
  __syncthreads();
  // eigen-decomposed blocks back to the original parameters
  // (ParameterSet::propagateEigenToOriginal, ParameterSet.cpp:766-780)
  const double* so = sp;
  if (v.n_eigen > 0) {
    double* orig = sp + P;
    for (int p = threadIdx.x; p < P; p += blockDim.x) orig[p] = sp[p];
    __syncthreads();
    for (int b = 0; b < v.n_eigen; ++b) {
      const int f = v.eig_first[b], n = v.eig_n[b];
      const double* V = v.eig_V + v.eig_off[b];
      for (int i = threadIdx.x; i < n; i += blockDim.x) {
        double acc = 0.0;
        for (int j = 0; j < n; ++j) acc = fma(V[(size_t)i * n + j], sp[f + j], acc);
        orig[f + i] = acc;
      }
    }
    __syncthreads();
    so = orig;
  }
  T* xs = (T*)v.x;
  for (int p = threadIdx.x; p < P; p += blockDim.x) {
    double x = so[p];
    const double lo = v.mirror_lo[p], hi = v.mirror_hi[p];
    if (lo > -DBL_MAX && hi < DBL_MAX) {
      // DialInputBuffer.cpp:56-70
      const double range = hi - lo;
      double t = fabs(fmod(x - lo, 2 * range));
      if (t > range) {
        t -= 2 * range;
        t = -t;
      }
      x = t + lo;
    }
    xs[(size_t)p * v.kpad + k] = (T)x;
  }
  if (v.n_grids > 0) {
    // the grid form: interval and fraction of every knot grid at this point,
    // the operations eval_coef applies per dial
    __syncthreads();
    GridPoint<T>* gp = (GridPoint<T>*)v.grid_pts;
    for (int g = threadIdx.x; g < v.n_grids; g += blockDim.x) {
      const GridDesc gd = v.grids[g];
      T xx = xs[(size_t)gd.p0 * v.kpad + k] * (T)gd.b + (T)gd.a;
      GridPoint<T> r;
      r.jb = 4 * coef_interval(xx, gd.n, gd.trunc != 0, r.u);
      gp[(size_t)g * v.kpad + k] = r;
    }
  }
}

// Device table functions: one thread per (entry, kTabPts points), the points on
// grid.z.  The FP64 sine and divisions are what it costs, and an SM issues a
// warp of them every 16 cycles: with one thread per entry for all points, the
// 4096 entries of a kriging table kept 16 SMs busy (511 us at 100 points); the
// points spread them over the chip, and the logarithm of the entry's node is
// taken once per kTabPts points.
constexpr int kTabPts = 4;
template <typename T>
__global__ void __launch_bounds__(128) k_table_fn(const DevView v, int K) {
  dep_launch();
  dep_wait();
  const TableFn fn = v.table_fns[blockIdx.y];
  const TableDesc td = v.tables[fn.table];
  const int j = blockIdx.x * blockDim.x + threadIdx.x;
  if (j >= td.size) return;
  const T* xs = (const T*)v.x;
  const double E = v.table_nodes[fn.nodes + j];
  T* arena = (T*)v.table_arena;
  const double logE = fn.kind == 1 ? log(E) : 0.0;
  const int k0 = blockIdx.z * kTabPts, k1 = min(K, k0 + kTabPts);
  for (int k = k0; k < k1; ++k) {
    double q[6];
#pragma unroll
    for (int i = 0; i < 6; ++i) q[i] = (double)xs[(size_t)fn.par[i] * v.kpad + k];
    double val = 1.0;
    if (fn.kind == 1) {
      const double s = sin(q[1] * 1.267 / E + q[2]);
      val = 1.0 - q[0] * s * s * (1.0 + q[3] * (logE - q[4])) * q[5];
    }
    arena[td.offset + (int64_t)j * v.kpad + k] = (T)val;
  }
}

// ---------------------------------------------------------------------------
// K = 1: type-ordered dial evaluation, one thread per dial.
// ---------------------------------------------------------------------------
template <typename T>
__global__ void __launch_bounds__(kPlainThreads) k_plain(const DevView v) {
  extern __shared__ __align__(128) unsigned char smem[];
  const int TB = v.tile_payload_bytes;
  unsigned char* stage0 = smem;
  unsigned char* stage1 = smem + TB;
  T* dval = (T*)(smem + 2 * TB);                       // [1024]
  double* wsh = (double*)(smem + 2 * TB + 1024 * sizeof(T));  // [kMaxTileEvents]
  uint16_t* sev = (uint16_t*)(wsh + kMaxTileEvents);  // [kMaxTileEvents]
  __shared__ uint64_t bar[2];
  __shared__ int s_bstart[kMaxLocalBins], s_bend[kMaxLocalBins];

  const int tid = threadIdx.x;
  if (tid == 0) {
    mbar_init(&bar[0], 1);
    mbar_init(&bar[1], 1);
    fence_mbar_init();
  }
  __syncthreads();

  int tile = blockIdx.x;
  if (tid == 0 && tile < v.n_tiles) issue_tile(v, tile, stage0, &bar[0]);
  dep_launch();
  dep_wait();  // the points (k_params, k_table_fn); the first tile's copy travels meanwhile
  for (int it = 0; tile < v.n_tiles; ++it, tile += gridDim.x) {
    const int st = it & 1;
    const uint32_t parity = (uint32_t)((it >> 1) & 1);
    const int next = tile + gridDim.x;
    if (tid == 0 && next < v.n_tiles) issue_tile(v, next, st ? stage0 : stage1, &bar[st ^ 1]);

    const TileDesc td = v.tiles[tile];
    uint64_t h[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int i = tid + j * kPlainThreads;
      h[j] = (i < td.ndials) ? v.hdr[td.dial0 + i] : 0ull;
    }
    T w0 = T(1);
    uint16_t evi = 0;
    if (tid < td.nevents) {
      evi = v.evinfo[td.event0 + tid];
      w0 = ((const T*)v.w0)[td.event0 + tid];
      sev[tid] = evi;
    }
    if (tid < kMaxLocalBins) {
      s_bstart[tid] = 0;
      s_bend[tid] = 0;
    }
    const bool ok = mbar_wait_bounded(&bar[st], parity, kWaitLimitNs);
    if (__syncthreads_or(!ok)) {
      if (tid == 0) {
        atomicOr(v.status, kStatusCopyTimeout);
        if (next < v.n_tiles) mbar_wait_bounded(&bar[st ^ 1], (uint32_t)(((it + 1) >> 1) & 1), kWaitLimitNs);
      }
      return;
    }
    const T* pl = (const T*)(st ? stage1 : stage0);

#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int i = tid + j * kPlainThreads;
      if (i < td.ndials) {
        T val[1];
        dial_values<T, 1>(v, h[j], pl, 0, 0, val);
        dval[hdr_slot(h[j])] = val[0];
      }
    }
    __syncthreads();

    if (tid < td.nevents) {
      const int s0 = ev_slot(evi);
      const int s1 = (tid + 1 < td.nevents) ? ev_slot(sev[tid + 1]) : (int)td.ndials;
      T w = T(1);
      for (int s = s0; s < s1; ++s) w *= dval[s];
      if (v.has_cap && w > (T)v.cap) w = (T)v.cap;
      w = w0 * w;
      wsh[tid] = (double)w;
      if (v.event_weights) v.event_weights[v.sorted_to_result[td.event0 + tid]] = (double)w;
      const int lb = ev_lbin(evi);
      if (tid == 0 || ev_lbin(sev[tid - 1]) != lb) s_bstart[lb] = tid;
      if (tid + 1 == td.nevents || ev_lbin(sev[tid + 1]) != lb) s_bend[lb] = tid + 1;
    }
    __syncthreads();

    // One warp per local bin: fixed-order FP64 reduction of w and w^2.
    const int warp = tid >> 5, lane = tid & 31;
    if (warp < (int)td.nbins) {
      const int b0 = s_bstart[warp], b1 = s_bend[warp];
      if (b1 > b0) {
        double s = 0.0, s2 = 0.0;
        for (int e = b0 + lane; e < b1; e += 32) {
          const double w = wsh[e];
          s += w;
          s2 += w * w;
        }
        for (int o = 16; o; o >>= 1) {
          s += __shfl_xor_sync(0xffffffffu, s, o);
          s2 += __shfl_xor_sync(0xffffffffu, s2, o);
        }
        if (lane == 0) {
          const int slot = (warp == 0) ? (int)td.slot0 : v.bin_slot[td.bin0 + warp];
          v.partials[(size_t)slot * v.kpad] = make_double2(s, s2);
        }
      }
    }
    __syncthreads();
  }
}

// ---------------------------------------------------------------------------
// K = 1, warp-specialised.  Warps 0..5 (evaluators) evaluate the type-ordered
// dials of a tile into one of two dial-value buffers while warps 6..7
// (reducers) form the ordered products and the bin partials of the previous
// tile from the other buffer, so the serial per-tile phases run beside the
// next tile's evaluation instead of behind a block barrier.  Hand-over per
// buffer b: FULL_b, a named barrier at which the evaluators arrive and the
// reducers wait, and ebar[b], an mbarrier at which the reducer warps arrive and
// the evaluators wait.  The evaluator warps do not meet: a tile's types differ in
// cost, and a warp that is done goes on with the next tile, up to the buffer the
// reducers still hold.  Double-float is the exception: its dial code is several
// times as long, and warps on different tiles run different types' code, so there
// the evaluators meet at the end of a tile (1M events, eight warps: 400 us so, 521
// without; FP64 the other way round, 348 and 333 us for 500k).  The last evaluator warp to be done with a tile issues
// the copies of the tile after next into its stage.  Every CTA runs the same
// number of iterations on both sides and every mbarrier wait is bounded; a
// timed-out wait marks the block failed and the protocol runs on without work:
// no further copy is issued, no header is decoded, and before the CTA exits
// thread 0 waits (bounded) for every copy in flight.
// ---------------------------------------------------------------------------
// NEV evaluator threads (192: six warps, the default; 256: eight warps, for
// double-float, whose tiles hold fewer dials than one round of 192 threads
// would cover evenly) and two reducer warps.
constexpr int kWsRed = 64;
constexpr int kBarFull = 2, kBarEval = 4, kBarRed = 6;

template <typename T, int NEV>
__global__ void __launch_bounds__(NEV + kWsRed, sizeof(T) == 4 ? 3 : 2) k_plain_ws(const DevView v) {
  constexpr int kWsEval = NEV, NT = NEV + kWsRed;
  extern __shared__ __align__(128) unsigned char smem[];
  const int TB = v.tile_payload_bytes;
  const int HB = v.tile_hdr_bytes;
  uint64_t* shdr = (uint64_t*)(smem + 2 * TB);                // [2][HB / 8], tile order
  T* dval = (T*)(smem + 2 * TB + 2 * HB);                     // [2][1024]
  double* wsh = (double*)(smem + 2 * TB + 2 * HB + 2048 * sizeof(T));  // [kMaxTileEvents]
  uint16_t* sev = (uint16_t*)(wsh + kMaxTileEvents);      // [kMaxTileEvents]
  __shared__ uint64_t bar[2], ebar[2];
  __shared__ int s_bstart[kMaxLocalBins], s_bend[kMaxLocalBins];
  __shared__ int s_done[2];                 // evaluator warps done with a stage's tile
  __shared__ volatile int s_fail, s_issued;  // s_issued: tiles whose copies the CTA has started

  const int tid = threadIdx.x;
  const int ntile = (int)blockIdx.x < v.n_tiles ? (v.n_tiles - (int)blockIdx.x + (int)gridDim.x - 1) / (int)gridDim.x
                                                : 0;
  const int hstride = HB / (int)sizeof(uint64_t);
  if (tid == 0) {
    mbar_init(&bar[0], 1);
    mbar_init(&bar[1], 1);
    mbar_init(&ebar[0], kWsRed / 32);
    mbar_init(&ebar[1], kWsRed / 32);
    fence_mbar_init();
    s_fail = 0;
    s_done[0] = s_done[1] = 0;
    s_issued = ntile < 2 ? ntile : 2;
    if (ntile > 0) issue_tile_hdr(v, blockIdx.x, smem, shdr, &bar[0]);
    if (ntile > 1) issue_tile_hdr(v, blockIdx.x + gridDim.x, smem + TB, shdr + hstride, &bar[1]);
  }
  dep_launch();
  dep_wait();  // the points (k_params, k_table_fn); the first tiles' copies travel meanwhile
  __syncthreads();

  if (tid < kWsEval) {
    // a tile's payload and headers arrive together by bulk copy; only the
    // dial count comes from the descriptor, loaded one tile ahead
    int nd = 0, nd_next = 0;
    if (ntile > 0) nd = v.tiles[blockIdx.x].ndials;
    if (ntile > 1) nd_next = v.tiles[blockIdx.x + gridDim.x].ndials;
    for (int it = 0; it < ntile; ++it) {
      const int tile = blockIdx.x + it * gridDim.x;
      const int st = it & 1;
      bool ok = !s_fail && mbar_wait_bounded(&bar[st], (uint32_t)((it >> 1) & 1), kWaitLimitNs);
      if (it >= 2)  // the reducers are done with buffer st (tile it - 2), after a failure too
        ok &= mbar_wait_bounded(&ebar[st], (uint32_t)(((it >> 1) - 1) & 1), kWaitLimitNs);
      if (!ok) s_fail = 1;
      T* dv = dval + st * 1024;
      // after any failed wait the stages hold nothing trustworthy: headers
      // are not decoded, so no shared-memory index comes from them
      if (ok && !s_fail) {
        const T* pl = (const T*)(smem + st * TB);
        const uint64_t* hs = shdr + st * hstride;
        for (int i = tid; i < nd; i += kWsEval) {
          const uint64_t h = hs[i];
          T val[1];
          dial_values<T, 1>(v, h, pl, 0, 0, val);
          dv[hdr_slot(h)] = val[0];
        }
      }
      named_arrive(kBarFull + st, NT);
      if constexpr (kIsDf<T>) named_sync(kBarEval, kWsEval);
      __syncwarp();
      if ((tid & 31) == 0) {
        __threadfence_block();  // this warp's reads of the stage come first
        if (atomicAdd(&s_done[st], 1) == kWsEval / 32 - 1) {
          s_done[st] = 0;
          // after a failed wait no further copy is issued: a stage whose copy
          // timed out may still be written by it
          if (it + 2 < ntile && !s_fail) {
            issue_tile_hdr(v, tile + 2 * gridDim.x, smem + st * TB, shdr + st * hstride, &bar[st]);
            s_issued = it + 3;
          }
        }
      }
      nd = nd_next;
      if (it + 2 < ntile) nd_next = v.tiles[tile + 2 * gridDim.x].ndials;
    }
  } else {
    const int r = tid - kWsEval;
    const int rwarp = r >> 5, lane = r & 31;
    // Reducer thread r handles events r, r + 64, ... of each tile.  The next
    // tile's descriptor, its event words and this thread's base weights are
    // loaded one tile ahead, so their latency overlaps the current tile's
    // products and sums instead of opening each tile.
    constexpr int kEvPer = kMaxTileEvents / kWsRed;
    TileDesc tdn;
    uint16_t pev[kEvPer];
    T pw0[kEvPer];
    auto prefetch = [&](int t) {
      tdn = v.tiles[t];
#pragma unroll
      for (int j = 0; j < kEvPer; ++j) {
        const int e = r + j * kWsRed;
        if (e < (int)tdn.nevents) {
          pev[j] = v.evinfo[tdn.event0 + e];
          pw0[j] = ((const T*)v.w0)[tdn.event0 + e];
        }
      }
    };
    if (ntile > 0) prefetch(blockIdx.x);
    for (int it = 0; it < ntile; ++it) {
      const int tile = blockIdx.x + it * gridDim.x;
      const int b = it & 1;
      const TileDesc td = tdn;
      T w0r[kEvPer];
#pragma unroll
      for (int j = 0; j < kEvPer; ++j) {
        const int e = r + j * kWsRed;
        if (e < (int)td.nevents) sev[e] = pev[j];
        w0r[j] = pw0[j];
      }
      if (it + 1 < ntile) prefetch(tile + gridDim.x);
      if (r < kMaxLocalBins) {
        s_bstart[r] = 0;
        s_bend[r] = 0;
      }
      named_sync(kBarRed, kWsRed);
      named_sync(kBarFull + b, NT);  // buffer b holds this tile's values
      const T* dv = dval + b * 1024;
#pragma unroll
      for (int j = 0; j < kEvPer; ++j) {
        const int e = r + j * kWsRed;
        if (e >= (int)td.nevents) break;
        const uint16_t evi = sev[e];
        const int s0 = ev_slot(evi);
        const int s1 = (e + 1 < td.nevents) ? ev_slot(sev[e + 1]) : (int)td.ndials;
        T w = T(1);
        for (int q = s0; q < s1; ++q) w *= dv[q];
        if (v.has_cap && w > (T)v.cap) w = (T)v.cap;
        w = w0r[j] * w;
        wsh[e] = (double)w;
        if (v.event_weights) v.event_weights[v.sorted_to_result[td.event0 + e]] = (double)w;
        const int lb = ev_lbin(evi);
        if (e == 0 || ev_lbin(sev[e - 1]) != lb) s_bstart[lb] = e;
        if (e + 1 == td.nevents || ev_lbin(sev[e + 1]) != lb) s_bend[lb] = e + 1;
      }
      __syncwarp();
      if (lane == 0) mbar_arrive(&ebar[b]);  // buffer b consumed
      named_sync(kBarRed, kWsRed);
      // one warp per local bin (two warps: bins w, w + 2): fixed-order FP64 sums
      for (int lb = rwarp; lb < (int)td.nbins; lb += 2) {
        const int b0 = s_bstart[lb], b1 = s_bend[lb];
        if (b1 > b0) {
          double sw = 0.0, sw2 = 0.0;
          for (int e = b0 + lane; e < b1; e += 32) {
            const double w = wsh[e];
            sw += w;
            sw2 += w * w;
          }
          for (int o = 16; o; o >>= 1) {
            sw += __shfl_xor_sync(0xffffffffu, sw, o);
            sw2 += __shfl_xor_sync(0xffffffffu, sw2, o);
          }
          if (lane == 0) {
            const int slot = (lb == 0) ? (int)td.slot0 : v.bin_slot[td.bin0 + lb];
            v.partials[(size_t)slot * v.kpad] = make_double2(sw, sw2);
          }
        }
      }
      named_sync(kBarRed, kWsRed);  // sev, wsh and the markers are reused
    }
  }
  __syncthreads();
  if (tid == 0 && s_fail) {
    atomicOr(v.status, kStatusCopyTimeout);
    // the copies that may still be in flight, the last two issued, land
    // (bounded) before the CTA's shared memory is released
    const int n = s_issued;
    for (int j = n > 2 ? n - 2 : 0; j < n; ++j)
      mbar_wait_bounded(&bar[j & 1], (uint32_t)((j >> 1) & 1), kWaitLimitNs);
  }
}

// ---------------------------------------------------------------------------
// Bin sums and likelihood.
// ---------------------------------------------------------------------------
// One block covers BT bins of KT points, 256 threads:
//   1. a bin's slots belong to eight runs, slot i0 + r to run r % 8: thread (point
//      kk, slot lane sl, bin bb), points fastest so that the reads of a slot's row
//      are contiguous, adds the slots of its runs sl, sl + SL, ... in order; the
//      runs are added in order, so that a point's sums do not depend on how many
//      points share the call;
//   2. thread (bin, point), bins fastest, writes the sums and evaluates the
//      likelihood term; the BT terms of a point are added;
//   3. these parts are added in the order of kLlhGroup, by the last block of the
//      point tile, or, where that block would have more than kOneLevel of them per
//      thread, by the last block of each group of 256 bins and then by the last of
//      all, which adds the penalty's.
// A Barlow-Beeston term is ~85 FP64 operations and an SM issues one warp of
// them every 16 cycles (10000 bins, 100 points: 189 us, 232 with CUDA's logarithm, a
// third square root and FP64 compares; see llh_bb_oa2021), so the terms are cut
// into many small blocks with full warps: 256 bins per block left 140 SMs idle at
// K = 1 (19.2 us for 3000 bins, now 12.5 us; the launch alone is 5 us).  The small
// KT give their threads to the slots of a bin instead, whose reads are a chain of
// L2 latencies.  Adding the parts in two levels takes a second arrival (1 us), in
// one level the parts go through a single SM (10000 bins, 100 points: 208 us that
// way; 100000 bins, 16 points: 140 us of 616), so the line lies where a thread of
// the last block would wait for more than a few rounds of loads.
constexpr int kOneLevel = 16;
template <int KT, int BT>
__global__ void __launch_bounds__(256) k_bins_llh(const DevView v, int K, double* sums, double* sums2,
                                                  double* llh, double* llh_stat) {
  constexpr int NT = 256, SL = NT / (KT * BT);
  static_assert(SL >= 1 && SL * KT * BT == NT && BT <= 32 && NT % KT == 0, "tile shape");
  constexpr int kRuns = 8, kParts = SL > 1 ? kRuns : 1;  // one thread per bin and point adds its runs itself
  static_assert(kRuns % SL == 0, "whole runs per slot lane");
  __shared__ double2 part[kParts][BT][KT + (KT > 1 ? 1 : 0)];
  __shared__ int slots[BT];
  __shared__ double red[kLlhRuns * KT];
  __shared__ bool last;
  const int tid = threadIdx.x;
  const int kb = blockIdx.y * KT, b0 = blockIdx.x * BT;
  dep_wait();
  {
    const int kk = tid % KT, sl = (tid / KT) % SL, bb = tid / (KT * SL);
    const int b = b0 + bb, k = kb + kk;
    const int i0 = b < v.n_bins ? v.bin_slot[b] : 0;
    const int n = b < v.n_bins && k < K ? v.bin_slot[b + 1] - i0 : 0;
    const double2* src = v.partials + (size_t)i0 * v.kpad + k;
    if constexpr (SL > 1) {
      if (kk == 0 && sl == 0) slots[bb] = n;
      constexpr int A = kRuns / SL, R = 4;  // runs of this thread, rows in flight
      static_assert(R % A == 0, "whole periods");
      double s[A] = {}, s2[A] = {};
      int r = sl;
      for (; r + (R - 1) * SL < n; r += R * SL) {
        double2 p[R];
#pragma unroll
        for (int q = 0; q < R; ++q) p[q] = src[(size_t)(r + q * SL) * v.kpad];
#pragma unroll
        for (int q = 0; q < R; ++q) {
          s[q % A] += p[q].x;
          s2[q % A] += p[q].y;
        }
      }
      if constexpr (A == 1) {  // most lanes have no slot: nothing is issued for them
        for (; r < n; r += SL) {
          const double2 p = src[(size_t)r * v.kpad];
          s[0] += p.x;
          s2[0] += p.y;
        }
      } else {
        double2 p[R - 1];
#pragma unroll
        for (int q = 0; q < R - 1; ++q)
          if (r + q * SL < n) p[q] = src[(size_t)(r + q * SL) * v.kpad];
#pragma unroll
        for (int q = 0; q < R - 1; ++q)
          if (r + q * SL < n) {
            s[q % A] += p[q].x;
            s2[q % A] += p[q].y;
          }
      }
#pragma unroll
      for (int q = 0; q < A; ++q) part[sl + q * SL][bb][kk] = make_double2(s[q], s2[q]);
    } else {
      // additions of rows that are there only: even one that adds zero takes its 16
      // cycles; four rows in flight
      double s = 0.0, s2 = 0.0;
      auto row = [&](int i) { return src[(size_t)i * v.kpad]; };
      auto add = [](double& x, double& y, const double2& p) {
        x += p.x;
        y += p.y;
      };
      if (n <= kRuns) {  // a slot per run at most: the runs in order are the slots in order
        int r = 0;
        for (; r + 3 < n; r += 4) {
          double2 p[4];
#pragma unroll
          for (int q = 0; q < 4; ++q) p[q] = row(r + q);
#pragma unroll
          for (int q = 0; q < 4; ++q) add(s, s2, p[q]);
        }
        for (; r < n; ++r) add(s, s2, row(r));
      } else if (n < 2 * kRuns) {  // two slots in the first n - 8 runs, one in the others
        const int two = n - kRuns;
        int h = 0;
        for (; h + 1 < two; h += 2) {
          double2 p[4];
#pragma unroll
          for (int q = 0; q < 4; ++q) p[q] = row(h + (q >> 1) + (q & 1) * kRuns);
          s += p[0].x + p[1].x;
          s2 += p[0].y + p[1].y;
          s += p[2].x + p[3].x;
          s2 += p[2].y + p[3].y;
        }
        if (h < two) {
          const double2 p = row(h), q = row(h + kRuns);
          s += p.x + q.x;
          s2 += p.y + q.y;
        }
        h = two;
        for (; h + 3 < kRuns; h += 4) {
          double2 p[4];
#pragma unroll
          for (int q = 0; q < 4; ++q) p[q] = row(h + q);
#pragma unroll
          for (int q = 0; q < 4; ++q) add(s, s2, p[q]);
        }
        for (; h < kRuns; ++h) add(s, s2, row(h));
      } else {
#pragma unroll 1
        for (int h = 0; h < kRuns; h += 4) {  // four runs at a time, each a sum of its own
          double2 t[4] = {};
          int i = h;
#pragma unroll 1
          for (; i + 3 < n; i += kRuns) {
            double2 p[4];
#pragma unroll
            for (int q = 0; q < 4; ++q) p[q] = row(i + q);
#pragma unroll
            for (int q = 0; q < 4; ++q) add(t[q].x, t[q].y, p[q]);
          }
#pragma unroll
          for (int q = 0; q < 3; ++q)
            if (i + q < n) add(t[q].x, t[q].y, row(i + q));
#pragma unroll
          for (int q = 0; q < 4; ++q) add(s, s2, t[q]);
        }
      }
      part[0][bb][kk] = make_double2(s, s2);
    }
  }
  __syncthreads();
  const bool want_llh = v.llh_type != 0 && (llh != nullptr || llh_stat != nullptr);
  if (tid < KT * BT) {
    const int bb = tid % BT, kk = tid / BT;
    const int b = b0 + bb, k = kb + kk;
    const bool in = b < v.n_bins && k < K;
    double term = 0.0;
    if (in) {
      double s = 0.0, s2 = 0.0;
      {
        const double2 p = part[0][bb][kk];
        s = p.x;
        s2 = p.y;
      }
      if constexpr (kParts > 1)
        for (int q = 1; q < min(slots[bb], kParts); ++q) {  // the runs that have a slot
          const double2 p = part[q][bb][kk];
          s += p.x;
          s2 += p.y;
        }
      if (sums) sums[(size_t)k * v.n_bins + b] = s;
      if (sums2) sums2[(size_t)k * v.n_bins + b] = s2;
      if (want_llh) {
        if (v.llh_type == 1)
          term = llh_poisson(v.data[b], s);
        else if (v.llh_type == 2)  // BinContent::sqrtSumSqWeights, squared again by the LLH
          term = llh_bb_bin(v.data[b], v.log_data[b], s, sqrt(s2));
      }
    }
    if (want_llh) {
      // whole warps are in this branch (KT * BT is a multiple of 32)
      term = neighbour_tree<1, BT>(term);
      if (in && bb == 0) v.llh_blocks[(size_t)blockIdx.x * v.kpad + k] = term;
    }
  }
  if (!want_llh) return;
  static_assert(NT == 32 * kLlhRuns && kLlhGroup % BT == 0 && KT <= 32, "a warp per run, whole blocks per group");
  constexpr int PG = kLlhGroup / BT;  // parts per group
  const int warp = tid >> 5, kk = tid % KT, sub = (tid & 31) / KT, k = kb + kk;
  const int parts = gridDim.x, groups = (parts + PG - 1) / PG;
  unsigned int* const counter = v.llh_counter + (size_t)blockIdx.y * (groups + 1);  // per group, and one for all
  auto part_of = [&](int i) { return i < parts && k < K ? __ldcg(&v.llh_blocks[(size_t)i * v.kpad + k]) : 0.0; };
  // whether this block is the last of `of` to arrive at counter c, its own results visible
  auto last_of = [&](int c, int of) {
    __threadfence();
    __syncthreads();
    if (tid == 0) {
      last = atomicAdd(&counter[c], 1u) == (unsigned)of - 1;
      if (last) counter[c] = 0u;
    }
    __syncthreads();
    if (last) __threadfence();
    return last;
  };
  // one level: a warp, L lanes per point and group, X parts per lane, G groups at a time
  constexpr int L = 32 / KT < PG ? 32 / KT : PG, X = PG / L, G = 32 / KT / L;
  double t = 0.0;
  if (X > kOneLevel || (groups + kLlhRuns * G - 1) / (kLlhRuns * G) * X > kOneLevel) {
    // this block's group: P neighbouring parts per thread, T threads per point
    constexpr int P = PG * KT > NT ? PG * KT / NT : 1, T = PG / P, W = T * KT > 32 ? T * KT / 32 : 1;
    const int g = blockIdx.x / PG, j0 = tid / KT * P;
    if (!last_of(g, min(parts - g * PG, PG))) return;
    double y[P];
#pragma unroll
    for (int j = 0; j < P; ++j) y[j] = j0 < PG ? part_of(g * PG + j0 + j) : 0.0;
#pragma unroll
    for (int h = 1; h < P; h <<= 1)
#pragma unroll
      for (int j = 0; j < P; j += 2 * h) y[j] += y[j + h];
    t = neighbour_tree<KT, W == 1 ? T * KT : 32>(y[0]);
    if (sub == 0) red[warp * KT + kk] = t;
    __syncthreads();
    if (tid < KT && k < K) {
      double w[W];
#pragma unroll
      for (int i = 0; i < W; ++i) w[i] = red[i * KT + kk];
#pragma unroll
      for (int h = 1; h < W; h <<= 1)
#pragma unroll
        for (int i = 0; i < W; i += 2 * h) w[i] += w[i + h];
      if (groups > 1) v.llh_groups[(size_t)g * v.kpad + k] = w[0];
      t = w[0];
    }
    if (groups > 1) {
      if (!last_of(groups, groups)) return;
      t = 0.0;
      // 32 / KT groups of the run at a time, added in order
      constexpr int S = 32 / KT;
#pragma unroll 4
      for (int g0 = warp; g0 < groups; g0 += kLlhRuns * S) {
        const int i = g0 + kLlhRuns * sub;
        const double x = i < groups && k < K ? __ldcg(&v.llh_groups[(size_t)i * v.kpad + k]) : 0.0;
#pragma unroll
        for (int q = 0; q < S; ++q) t += S > 1 ? __shfl_sync(0xffffffffu, x, q * KT + kk) : x;
      }
    } else {
      if (tid >= KT) t = 0.0;  // the one group is run 0, the others are empty
      __syncthreads();
    }
  } else {
    if (!last_of(groups, parts)) return;
    constexpr int U = X < 4 ? 4 / X : 1;  // rounds in flight
    for (int g0 = warp; g0 < groups; g0 += kLlhRuns * G * U) {
      double y[U][X];
#pragma unroll
      for (int u = 0; u < U; ++u)
#pragma unroll
        for (int j = 0; j < X; ++j) y[u][j] = part_of((g0 + kLlhRuns * (u * G + sub / L)) * PG + sub % L * X + j);
#pragma unroll
      for (int u = 0; u < U; ++u) {
        if (g0 + kLlhRuns * u * G >= groups) break;
#pragma unroll
        for (int h = 1; h < X; h <<= 1)
#pragma unroll
          for (int j = 0; j < X; j += 2 * h) y[u][j] += y[u][j + h];
        const double x = neighbour_tree<KT, KT * L>(y[u][0]);
#pragma unroll
        for (int q = 0; q < G; ++q) t += G > 1 ? __shfl_sync(0xffffffffu, x, q * L * KT + kk) : x;
      }
    }
  }
  if (sub == 0) red[warp * KT + kk] = t;
  __syncthreads();
  if (tid < KT && k < K) {
    double r[kLlhRuns];
#pragma unroll
    for (int w = 0; w < kLlhRuns; ++w) r[w] = red[w * KT + tid];
    t = ((r[0] + r[1]) + (r[2] + r[3])) + ((r[4] + r[5]) + (r[6] + r[7]));
    double pen = 0.0;
    for (int q = 0; q < v.n_pen; ++q) pen += v.penalty[(size_t)q * v.kpad + k];
    if (llh_stat) llh_stat[k] = t;
    if (llh) llh[k] = t + pen;
  }
}

// log(data) per bin, taken once when the data are set instead of per bin and
// point in every evaluation.
__global__ void k_log_data(const double* __restrict__ data, double* __restrict__ log_data, int n) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) log_data[i] = log_data_of(data[i]);
}

}  // namespace

// ---------------------------------------------------------------------------
// Launchers.
// ---------------------------------------------------------------------------
size_t plain_smem_bytes(const DevView& v) {
  const size_t tsz = v.precision == 1 ? sizeof(float) : sizeof(double);
  const size_t dv = (v.plain_kind >= 1 ? 2048 : 1024) * tsz;
  const size_t hb = v.plain_kind >= 1 ? 2 * (size_t)v.tile_hdr_bytes : 0;
  return 2 * (size_t)v.tile_payload_bytes + hb + dv + kMaxTileEvents * sizeof(double) +
         kMaxTileEvents * sizeof(uint16_t);
}

size_t batched_smem_bytes(const DevView& v, const BatchedShape& b) {
  const size_t tsz = v.precision == 1 ? sizeof(float) : sizeof(double);
  if (b.kind == 3) return ws_smem_bytes(v, b.kc);  // k_ws
  if (b.kind == 1) {  // k_multi
    return (size_t)b.stages * v.tile_payload_bytes + 1024 * sizeof(uint64_t) +
           (size_t)kMaxTileEvents * b.kc * sizeof(double) + (size_t)1024 * b.kc * tsz + kMaxTileEvents * tsz +
           (kMaxTileEvents + 1) * sizeof(uint16_t);
  }
  const int nw = b.threads / 32;
  // k_batched: per stage the payload, the headers (sized for the engine's
  // largest tile) and the event buffers; then the bin partials
  return (size_t)b.stages * ((size_t)v.tile_payload_bytes + (size_t)v.tile_hdr_bytes + lanes_ev_bytes(tsz)) +
         (size_t)(nw + kMaxLocalBins - 1) * b.kr * 32 * sizeof(double2);
}

template <typename T>
static const void* plain_fn(int kind) {
  if (kind == 2) return (const void*)k_plain_ws<T, 256>;
  return kind == 1 ? (const void*)k_plain_ws<T, 192> : (const void*)k_plain<T>;
}

// threads of a K = 1 kernel kind (0: k_plain, 1: k_plain_ws with six
// evaluator warps, 2: with eight)
static int plain_threads(int kind) { return kind == 2 ? 256 + kWsRed : kind == 1 ? 192 + kWsRed : kPlainThreads; }

// Every batched shape: the lanes-over-points family (gw_lanes.cu), the
// dials-over-threads family (gw_multi.cu), then the warp-specialised small-K
// family (gw_ws.cu).
static const ShapeEntry* shape_entry(int i) {
  const ShapeEntry* lanes;
  const ShapeEntry* multi;
  const ShapeEntry* ws;
  const int nl = lane_shapes(&lanes);
  const int nm = multi_shapes(&multi);
  const int ns = ws_shapes(&ws);
  if (i < 0 || i >= nl + nm + ns) return nullptr;
  if (i < nl) return &lanes[i];
  if (i < nl + nm) return &multi[i - nl];
  return &ws[i - nl - nm];
}

int batched_shape_count() {
  const ShapeEntry* p;
  return lane_shapes(&p) + multi_shapes(&p) + ws_shapes(&p);
}

BatchedShape batched_shape(int i) {
  const ShapeEntry& e = *shape_entry(i);
  return BatchedShape{e.kind, e.kc, e.kr, e.threads, e.stages, e.minb};
}

static const ShapeEntry* find_shape(const BatchedShape& b) {
  for (int i = 0; i < batched_shape_count(); ++i) {
    const ShapeEntry* e = shape_entry(i);
    if (e->kind == b.kind && e->kc == b.kc && e->kr == b.kr && e->threads == b.threads && e->stages == b.stages &&
        e->minb == b.minb)
      return e;
  }
  return nullptr;
}

static const void* pick_plain(const DevView& v) {
  if (v.precision == 2) return plain_fn<dfloat>(v.plain_kind);
  return v.precision ? plain_fn<float>(v.plain_kind) : plain_fn<double>(v.plain_kind);
}

// Raises the kernel's limit of dynamic shared memory on the current device to
// `smem`, and never lowers it: the limit is the kernel's, not an engine's, and set to
// the need of the engine built last it would refuse the launches of an earlier one
// with larger tiles or more parameters.
static cudaError_t open_shared(const void* fn, size_t smem) {
  static std::mutex mu;
  std::lock_guard<std::mutex> lk(mu);
  cudaFuncAttributes a;
  const cudaError_t r = cudaFuncGetAttributes(&a, fn);
  if (r != cudaSuccess || (size_t)a.maxDynamicSharedSizeBytes >= smem) return r;
  return cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
}

// Resident blocks per SM, 0 when the kernel cannot run with that much shared memory.
static int blocks_per_sm(const void* fn, int threads, size_t smem) {
  int n = 0;
  if (open_shared(fn, smem) != cudaSuccess ||
      cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, fn, threads, smem) != cudaSuccess) {
    cudaGetLastError();
    return 0;
  }
  return n;
}

int plain_blocks_per_sm(const DevView& v) {
  return blocks_per_sm(pick_plain(v), plain_threads(v.plain_kind), plain_smem_bytes(v));
}

int batched_blocks_per_sm(const DevView& v, const BatchedShape& b) {
  const ShapeEntry* e = find_shape(b);
  if (!e) return 0;
  const void* fn = e->fn[v.precision];
  if (!fn) return 0;  // not compiled for this precision
  return blocks_per_sm(fn, b.threads, batched_smem_bytes(v, b));
}

size_t params_smem_bytes(const DevView& v) { return (size_t)v.n_params * sizeof(double) * (v.n_eigen > 0 ? 2 : 1); }

cudaError_t prepare_params(const DevView& v) {
  return open_shared(v.precision == 2 ? (const void*)k_params<dfloat>
                     : v.precision   ? (const void*)k_params<float>
                                     : (const void*)k_params<double>,
                     params_smem_bytes(v));
}

cudaError_t launch_params(const DevView& v, const double* params, int K, cudaStream_t s) {
  const size_t smem = params_smem_bytes(v);
  const dim3 grid(K, 1 + v.n_pen);
  if (v.precision == 2)
    k_params<dfloat><<<grid, 256, smem, s>>>(v, params);
  else if (v.precision)
    k_params<float><<<grid, 256, smem, s>>>(v, params);
  else
    k_params<double><<<grid, 256, smem, s>>>(v, params);
  return cudaGetLastError();
}

cudaError_t launch_table_fns(const DevView& v, int K, int max_size, cudaStream_t s) {
  if (v.n_table_fns == 0) return cudaSuccess;
  const dim3 grid((max_size + 127) / 128, v.n_table_fns, (K + kTabPts - 1) / kTabPts);
  if (v.precision == 2)
    launch_dependent(k_table_fn<dfloat>, grid, 128, 0, s, v, K);
  else if (v.precision)
    launch_dependent(k_table_fn<float>, grid, 128, 0, s, v, K);
  else
    launch_dependent(k_table_fn<double>, grid, 128, 0, s, v, K);
  return cudaGetLastError();
}

// The K = 1 chain is dependent launches (gw_launch.h): parameter update, weights
// and bins are short, and the weights kernel's first tiles travel while the
// parameters are updated (100k events, FP64: 81 -> 71 us an evaluation).  The
// batched chain is not: a batched kernel fills the SMs for a millisecond, and
// launched that way it ran slower (64 points of 1M events 1.17 -> 1.26 ms, in
// FP64 2.04 -> 2.45 ms).
cudaError_t launch_plain(const DevView& v, int grid, cudaStream_t s) {
  const size_t smem = plain_smem_bytes(v);
  if (v.plain_kind == 2) {
    const int nt = plain_threads(2);
    if (v.precision == 2)
      launch_dependent(k_plain_ws<dfloat, 256>, grid, nt, smem, s, v);
    else if (v.precision)
      launch_dependent(k_plain_ws<float, 256>, grid, nt, smem, s, v);
    else
      launch_dependent(k_plain_ws<double, 256>, grid, nt, smem, s, v);
  } else if (v.plain_kind == 1) {
    const int nt = plain_threads(1);
    if (v.precision == 2)
      launch_dependent(k_plain_ws<dfloat, 192>, grid, nt, smem, s, v);
    else if (v.precision)
      launch_dependent(k_plain_ws<float, 192>, grid, nt, smem, s, v);
    else
      launch_dependent(k_plain_ws<double, 192>, grid, nt, smem, s, v);
  } else {
    if (v.precision == 2)
      launch_dependent(k_plain<dfloat>, grid, kPlainThreads, smem, s, v);
    else if (v.precision)
      launch_dependent(k_plain<float>, grid, kPlainThreads, smem, s, v);
    else
      launch_dependent(k_plain<double>, grid, kPlainThreads, smem, s, v);
  }
  return cudaGetLastError();
}

bool batched_shape_covers(const DevView& v, const BatchedShape& b, int K) {
  const int per_pass = b.kind == 0 ? b.kc * b.kr : b.kc;
  return K >= 1 && per_pass >= 1 && (int64_t)((K + per_pass - 1) / per_pass) * per_pass <= (int64_t)v.kpad;
}

cudaError_t launch_batched(const DevView& v, int K, const BatchedShape& b, int grid, cudaStream_t s) {
  const ShapeEntry* e = find_shape(b);
  if (!e || !e->launch[v.precision] || !batched_shape_covers(v, b, K)) return cudaErrorInvalidValue;
  e->launch[v.precision](v, K, grid, batched_smem_bytes(v, b), s);
  return cudaGetLastError();
}

cudaError_t launch_bins_llh(const DevView& v, int K, double* sums, double* sums2, double* llh,
                            double* llh_stat, cudaStream_t s) {
  // point tiles as wide as K allows, so that phase 2's warps are full
  auto grid = [&](int kt, int bt) { return dim3((v.n_bins + bt - 1) / bt, (K + kt - 1) / kt); };
  if (K == 1)
    return launch_dependent(k_bins_llh<1, 32>, grid(1, 32), 256, 0, s, v, K, sums, sums2, llh, llh_stat);
  if (K <= 4)  // a warp of terms per point: of three points in one tile of four, a quarter was idle
    k_bins_llh<2, 32><<<grid(2, 32), 256, 0, s>>>(v, K, sums, sums2, llh, llh_stat);
  else if (K <= 8)
    k_bins_llh<8, 16><<<grid(8, 16), 256, 0, s>>>(v, K, sums, sums2, llh, llh_stat);
  else if (K <= 16)
    k_bins_llh<16, 16><<<grid(16, 16), 256, 0, s>>>(v, K, sums, sums2, llh, llh_stat);
  else
    k_bins_llh<32, kLlhBins><<<grid(32, kLlhBins), 256, 0, s>>>(v, K, sums, sums2, llh, llh_stat);
  return cudaGetLastError();
}

cudaError_t launch_log_data(const DevView& v, cudaStream_t s) {
  k_log_data<<<(v.n_bins + 255) / 256, 256, 0, s>>>(v.data, v.log_data, v.n_bins);
  return cudaGetLastError();
}

}  // namespace gw

// ---------------------------------------------------------------------------
// Per-bin likelihood terms on the device, one thread per bin: the same device
// functions k_bins_llh sums.
// ---------------------------------------------------------------------------
namespace gw {
namespace {
__global__ void k_llh_bins(int type, const double* data, const double* pred, const double* sqrt_sum_w2, int n,
                           double* out) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  out[i] = type == GW_LLH_POISSON ? llh_poisson(data[i], pred[i]) : llh_bb_bin(data[i], log_data_of(data[i]), pred[i], sqrt_sum_w2[i]);
}
}  // namespace
}  // namespace gw

extern "C" int gw_llh_bins(int32_t llh_type, const double* data, const double* pred, const double* sqrt_sum_w2,
                           int32_t n, double* out) {
  if (!data || !pred || !sqrt_sum_w2 || !out || n < 0 ||
      (llh_type != GW_LLH_POISSON && llh_type != GW_LLH_BARLOW_BEESTON_OA2021))
    return GW_ERR_ARG;
  if (n == 0) return GW_OK;
  double* d = nullptr;
  const size_t bytes = sizeof(double) * (size_t)n;
  if (cudaMalloc(&d, 4 * bytes) != cudaSuccess) {
    cudaGetLastError();
    return GW_ERR_NOMEM;
  }
  cudaError_t e = cudaMemcpy(d, data, bytes, cudaMemcpyHostToDevice);
  if (e == cudaSuccess) e = cudaMemcpy(d + n, pred, bytes, cudaMemcpyHostToDevice);
  if (e == cudaSuccess) e = cudaMemcpy(d + 2 * (size_t)n, sqrt_sum_w2, bytes, cudaMemcpyHostToDevice);
  if (e == cudaSuccess) {
    gw::k_llh_bins<<<(n + 255) / 256, 256>>>(llh_type, d, d + n, d + 2 * (size_t)n, n, d + 3 * (size_t)n);
    e = cudaGetLastError();
  }
  if (e == cudaSuccess) e = cudaMemcpy(out, d + 3 * (size_t)n, bytes, cudaMemcpyDeviceToHost);
  cudaFree(d);
  if (e != cudaSuccess) {
    cudaGetLastError();
    return GW_ERR_CUDA;
  }
  return GW_OK;
}

// Compiled by the CUDA compiler: the device code above is in this library.
extern "C" int gw_using_cuda(int32_t* using_cuda) {
  if (!using_cuda) return GW_ERR_ARG;
#ifdef __CUDACC__
  *using_cuda = 1;
#else
  *using_cuda = 0;
#endif
  return GW_OK;
}

// ---------------------------------------------------------------------------
// Failure-path self-test: an mbarrier that expects bytes no copy will ever
// deliver (nothing is in flight).  The bounded wait must give up after
// limit_us and report it, leaving the context usable.
// ---------------------------------------------------------------------------
namespace gw {
namespace {
__global__ void k_selftest_wait(uint64_t limit_ns, uint32_t* status) {
  __shared__ uint64_t bar;
  mbar_init(&bar, 1);
  fence_mbar_init();
  mbar_expect_tx(&bar, 16u);  // arrives, but 16 bytes stay pending forever
  const bool ok = mbar_wait_bounded(&bar, 0u, limit_ns);
  *status = ok ? 0u : kStatusCopyTimeout;
}
}  // namespace
}  // namespace gw

extern "C" int gw_selftest_wait_timeout(uint32_t limit_us, int32_t* timed_out) {
  if (!timed_out || limit_us == 0 || limit_us > 1000000u) return GW_ERR_ARG;
  uint32_t* d = nullptr;
  if (cudaMalloc(&d, sizeof(uint32_t)) != cudaSuccess) {
    cudaGetLastError();
    return GW_ERR_CUDA;
  }
  cudaMemset(d, 0xFF, sizeof(uint32_t));
  gw::k_selftest_wait<<<1, 1>>>((uint64_t)limit_us * 1000ull, d);
  uint32_t h = 0;
  cudaError_t e = cudaGetLastError();
  if (e == cudaSuccess) e = cudaMemcpy(&h, d, sizeof(uint32_t), cudaMemcpyDeviceToHost);
  cudaFree(d);
  if (e != cudaSuccess) return GW_ERR_CUDA;
  *timed_out = (h == gw::kStatusCopyTimeout) ? 1 : 0;
  return GW_OK;
}

// ---------------------------------------------------------------------------
// FP32 throughput probe (the denominator of the compute roofline of the
// batched kernels): independent FMA chains in registers, no memory traffic
// in the loop.
// ---------------------------------------------------------------------------
namespace gw {
namespace {
__global__ void __launch_bounds__(256) k_fma_probe(int iters, float b, float c, float* sink) {
  float a[8];
#pragma unroll
  for (int j = 0; j < 8; ++j) a[j] = (float)(threadIdx.x + j) * 1e-3f;
  for (int i = 0; i < iters; ++i) {
#pragma unroll
    for (int j = 0; j < 8; ++j) a[j] = fmaf(a[j], b, c);
  }
  float s = 0.f;
#pragma unroll
  for (int j = 0; j < 8; ++j) s += a[j];
  if (s == 12345.678f) sink[0] = s;  // keeps the chains live
}
}  // namespace
}  // namespace gw

extern "C" int gw_measure_fp32_peak(int32_t device, double* tflops) {
  if (!tflops) return GW_ERR_ARG;
  if (cudaSetDevice(device) != cudaSuccess) {
    cudaGetLastError();
    return GW_ERR_CUDA;
  }
  int sms = 0;
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device);
  float* sink = nullptr;
  if (cudaMalloc(&sink, sizeof(float)) != cudaSuccess) {
    cudaGetLastError();
    return GW_ERR_NOMEM;
  }
  const int iters = 8192, blocks = sms * 8, threads = 256;
  cudaEvent_t a, b;
  cudaEventCreate(&a);
  cudaEventCreate(&b);
  double best = 0.0;
  for (int rep = 0; rep < 4; ++rep) {
    cudaEventRecord(a);
    gw::k_fma_probe<<<blocks, threads>>>(iters, 0.999f, 1e-4f, sink);
    cudaEventRecord(b);
    cudaEventSynchronize(b);
    float ms = 0.f;
    cudaEventElapsedTime(&ms, a, b);
    if (ms > 0.f) best = std::max(best, 2.0 * 8.0 * iters * (double)blocks * threads / (ms * 1e-3) / 1e12);
  }
  cudaEventDestroy(a);
  cudaEventDestroy(b);
  cudaFree(sink);
  const cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return GW_ERR_CUDA;
  *tflops = best;
  return GW_OK;
}
