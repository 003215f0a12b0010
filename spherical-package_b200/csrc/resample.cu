// resample_from_map (gather) and resample_to_map (adjoint, through a scatter plan).
#include <algorithm>

#include "common.cuh"
#include "plane_groups.cuh"

namespace sph {

// One thread decodes one map position once and then walks kPlanesPerThread
// (batch, channel) planes with the same taps.  Reference kernel:
// ext_modules/include/cuda/resample.cuh:50-81 (one thread per (c, position), one
// launch per image); arithmetic: common/resample.h:34-52, 85-107.
// Bound: wavefronts of the SM's path to L1, as many per load as the lines that a warp's positions lie in (89 %).  A block's positions
// are 16 x 16: a row of 256 tangent-image samples crosses many image rows (96 planes of 1024 x 2048 into 20 x 256 x 256: rows of 256
// 454 us, 32 x 8 391, 16 x 16 358, 8 x 32 411).
//
// With `quad` (UV-map gather, common/resample.h:133-159) every plane holds NT textures of H x W and position i samples
// texture quad[i]; an index outside [0, NT) yields zero.
template <typename T, int INTERP, bool WEIGHTED, int PPT>
__global__ void __launch_bounds__(256)
resample_from_map_kernel(const T *__restrict__ x, const T *__restrict__ map, const T *__restrict__ iw,
                         T *__restrict__ y, BlockTile bt, int planes, int H, int W, int P, const int64_t *__restrict__ quad,
                         int NT) {
  const int i = bt.output(), n = bt.width * bt.height;
  if (i < 0) return;
  const int p0 = blockIdx.y * PPT;
  const int np = min(PPT, planes - p0);
  size_t hw = (size_t)H * W;
  const T *xp = x + (size_t)p0 * hw;
  T *yp = y + (size_t)p0 * n + i;
  Taps<T> t;
  bool dead = false;
  if (quad) {
    const int64_t q = __ldg(quad + i);
    dead = q < 0 || q >= NT;
    xp = x + (size_t)p0 * hw * NT + (dead ? 0 : (size_t)q * hw);
    hw *= NT;
  }
  if (!WEIGHTED) {
    decode<T, INTERP>(__ldg(map + 2 * (size_t)i), __ldg(map + 2 * (size_t)i + 1), H, W, t);
    if (dead) {
#pragma unroll
      for (int k = 0; k < 4; k++) t.off[k] = -1;
    }
    if constexpr (sizeof(T) == 4) {
      if (INTERP != SPH_NEAREST && !quad && np == PPT && __all_sync(__activemask(), square_taps(t, W))) {
        const float *at = xp + t.off[0];
#pragma unroll
        for (int j = 0; j < PPT; j++, at += hw) yp[(size_t)j * n] = gather_square(at, W, t);
        return;
      }
    }
#pragma unroll
    for (int j = 0; j < PPT; j++)
      if (j < np) yp[(size_t)j * n] = gather<T, INTERP>(xp + j * hw, t);
  } else {
    T acc[PPT];
#pragma unroll
    for (int j = 0; j < PPT; j++) acc[j] = T(0);
    for (int q = 0; q < P; q++) {
      const size_t e = (size_t)i * P + q;
      decode<T, INTERP>(__ldg(map + 2 * e), __ldg(map + 2 * e + 1), H, W, t);
      const T wq = __ldg(iw + e);
#pragma unroll
      for (int j = 0; j < PPT; j++)
        if (j < np) acc[j] = RN<T>::add(acc[j], RN<T>::mul(wq, gather<T, INTERP>(xp + j * hw, t)));
    }
#pragma unroll
    for (int j = 0; j < PPT; j++)
      if (j < np) yp[(size_t)j * n] = acc[j];
  }
}

// a[j] / d for all j, rounded as a division is.  Float32: with the reciprocal r of d, rounded to nearest, q = a r is less than two units
// off, and each step q + (a - q d) r, the remainder in one fused operation, makes an approximation within a unit the nearest one (P.
// Markstein, IBM J. Res. Dev. 34, 1990); two steps of them.  It takes divisors within 2^+-60 and values that are zero or within 2^+-60:
// quotients are then normal numbers, remainders exact, and nothing over- or underflows.  (A subnormal quotient can lie half way between
// two numbers, which the last step's addition then rounds once more.)  Others are divided.  (154 planes of 974 x 1948
// pixels with plain divisions: 472 us, 145 of them the divisions.)
template <int N> __device__ __forceinline__ void divide_all(float (&a)[N], float d) {
  float least = 1.0f, most = 1.0f;
#pragma unroll
  for (int j = 0; j < N; j++) {
    least = fminf(least, a[j] == 0.0f ? 1.0f : fabsf(a[j]));
    most = fmaxf(most, fabsf(a[j]));
  }
  if (d >= 0x1p-60f && d <= 0x1p60f && least >= 0x1p-60f && most <= 0x1p60f) {
    const float r = 1.0f / d;
#pragma unroll
    for (int j = 0; j < N; j++) {
      float q = __fmul_rn(a[j], r);
      q = fmaf(fmaf(-q, d, a[j]), r, q);
      a[j] = fmaf(fmaf(-q, d, a[j]), r, q);
    }
  } else {
#pragma unroll
    for (int j = 0; j < N; j++) a[j] = a[j] / d;
  }
}
template <int N> __device__ __forceinline__ void divide_all(double (&a)[N], double d) {
#pragma unroll
  for (int j = 0; j < N; j++) a[j] = a[j] / d;
}

// Adjoint as a gather through the plan.  A thread owns one destination pixel of PL planes and walks the pixel's segment:
// an entry's source and weight are read once (the next entry's while this one's values are on their way) and serve PL
// independent loads, products and sums.  A block's pixels are 32 x 8: their entries lie in fewer lines than those of 256 pixels of
// a row (96 planes of 20 x 256 x 256 tangent samples onto 1024 x 2048 pixels, in rows 740 us, 32 x 8 586, 16 x 16 609, 64 x 4 601, 8 x 32 713;
// with 12 planes per thread 536, 16 542, 24 544, four 870;
// normalised 683, 12 planes 622, 566 with five blocks per SM and divide_all).  Sums run in plan order whatever the scheduling: deterministic, with no zero-fill
// pass and no atomics (the reference's scatter kernels use atomicAdd: ext_modules/include/cuda/resample.cuh:14-47).
//   DIV   x[s / div] / div instead of x[s]: mapped average unpooling, whose plan runs over the flattened map slots
//         s = o * K + k and whose slots all carry grad[o] / K (common/mapped_avg_pool.h:41-69, 109-143)
//   NORM  the sum is divided by (sum of the segment's weights + 1e-12), i.e. scatter(x) / (scatter(1) + 1e-12), the
//         weight-sum normalisation the reference composes in Python (layers/functional/sphere_ops.py:74-80)
// Blocks per SM that registers leave room for: six (40 registers) for plain float32 sums of eight planes, five (48) for others, four (64)
// and three for float64.  With 48, 56 and 72 registers, a block less each, 64 planes of 321 x 641 took 34.6 us instead of 30.8, in
// float64 56.8 instead of 51.1.
template <typename T, int PL, bool NORM, bool DIV>
__global__ void __launch_bounds__(256, sizeof(T) == 8 ? (DIV ? 3 : 4) : PL == 12 || NORM || DIV ? 5 : 6)
resample_to_map_kernel(const T *__restrict__ x, const void *__restrict__ plan_blob, T *__restrict__ out, BlockTile bt, int n_src,
                       int planes, int div, FastDiv fd) {
  const int q = bt.output(), n_dst = bt.width * bt.height;
  if (q < 0) return;
  bool ok;
  const PlanView<T> pv = plan_view<T>(plan_blob, n_dst, ok, DIV ? n_src * div : n_src);
  const int e0 = ok ? __ldg(pv.offsets + q) : 0, e1 = ok ? __ldg(pv.offsets + q + 1) : 0;
  const int p0 = blockIdx.y * PL, np = min(PL, planes - p0);
  const T *xp = x + (size_t)p0 * n_src;
  T acc[PL], wsum = T(0);
#pragma unroll
  for (int j = 0; j < PL; j++) acc[j] = T(0);
  int s = e0 < e1 ? __ldg(pv.src + e0) : 0;
  T w = e0 < e1 ? __ldg(pv.w + e0) : T(0);
  for (int e = e0; e < e1; e++) {
    const unsigned o = DIV ? fd.div((unsigned)s) : (unsigned)s;
    const bool fine = index_ok(s, pv.n_src);
    const T we = w;
    if (e + 1 < e1) {
      s = __ldg(pv.src + e + 1);
      w = __ldg(pv.w + e + 1);
    }
    if (!fine) continue;
    T v[PL];
    const T *src = xp + o;
    if (np == PL) {  // (the usual block: no predicates)
#pragma unroll
      for (int j = 0; j < PL; j++, src += n_src) v[j] = __ldg(src);
    } else {
#pragma unroll
      for (int j = 0; j < PL; j++, src += n_src) v[j] = j < np ? __ldg(src) : T(0);
    }
#pragma unroll
    for (int j = 0; j < PL; j++) acc[j] = RN<T>::add(acc[j], RN<T>::mul(we, DIV ? v[j] / (T)div : v[j]));
    if (NORM) wsum += we;
  }
  if (NORM && e1 > e0) {  // (an empty sum is zero already)
    divide_all(acc, wsum + T(1e-12));
  }
  T *op = out + (size_t)p0 * n_dst + q;
#pragma unroll
  for (int j = 0; j < PL; j++)
    if (j < np) __stcs(op + (size_t)j * n_dst, acc[j]);
}

// Planes walked per thread: 8 amortises the tap decode best; small problems use 2 so that enough threads are
// in flight to cover the memory latency.
static int planes_per_thread(int64_t n, int64_t planes) {
  return n * ((planes + 7) / 8) >= (int64_t)148 * 2048 * 2 ? 8 : 2;
}

template <typename T, int PPT>
static void from_map_launch(const void *x, const void *map, const void *iw, void *y, int64_t planes, int64_t H, int64_t W,
                            int64_t MH, int64_t MW, int64_t P, int interp, cudaStream_t st, const int64_t *quad, int NT) {
  const BlockTile bt = BlockTile::make(MH, MW, 4);
  dim3 grid(bt.blocks(), cdiv(planes, PPT));
  SPH_DISPATCH_INTERP(interp, {
    if (P > 0)
      resample_from_map_kernel<T, INTERP, true, PPT><<<grid, 256, 0, st>>>((const T *)x, (const T *)map, (const T *)iw, (T *)y,
                                                                           bt, (int)planes, (int)H, (int)W, (int)P, nullptr, 1);
    else
      resample_from_map_kernel<T, INTERP, false, PPT><<<grid, 256, 0, st>>>((const T *)x, (const T *)map, nullptr, (T *)y,
                                                                            bt, (int)planes, (int)H, (int)W, 0, quad, NT);
  });
}

template <typename T>
static int from_map(const void *x, const void *map, const void *iw, void *y, int64_t planes, int64_t H, int64_t W,
                    int64_t MH, int64_t MW, int64_t P, int interp, cudaStream_t st, const int64_t *quad = nullptr, int NT = 1) {
  if (planes_per_thread(MH * MW, planes) == 8) from_map_launch<T, 8>(x, map, iw, y, planes, H, W, MH, MW, P, interp, st, quad, NT);
  else from_map_launch<T, 2>(x, map, iw, y, planes, H, W, MH, MW, P, interp, st, quad, NT);
  return launch_status();
}

template <typename T, int PL>
static int to_map_launch(const void *x, const void *plan, void *out, int64_t planes, int64_t n_src, int64_t OH, int64_t OW, cudaStream_t st,
                         int src_div, bool normalize) {
  const BlockTile bt = BlockTile::make(OH, OW, 5);
  const dim3 grid(bt.blocks(), cdiv(planes, PL));
  const FastDiv fd = FastDiv::make((unsigned)src_div);
#define SPH_SCATTER(NORM, DIV)                                                                                               \
  resample_to_map_kernel<T, PL, NORM, DIV><<<grid, 256, 0, st>>>((const T *)x, plan, (T *)out, bt, (int)n_src, (int)planes, \
                                                                 src_div, fd)
  if (src_div > 1) SPH_SCATTER(false, true);  // (never normalised)
  else if (normalize) SPH_SCATTER(true, false);
  else SPH_SCATTER(false, false);
#undef SPH_SCATTER
  return launch_status();
}

// Planes per thread: 12 share an entry best (comment of the kernel), 8 in float64, where there are no more, and where groups of 12 would
// have to be filled up further.  Average unpooling, which divides each value, takes 12 only where that fills up less (3 x 3 gnomonic maps
// of stride 2, 8 and 12 planes per thread: 12 planes of 400 x 801 53 and 32 us, 36 100 and 82, 60 148 and 132; but 24 planes of 64 x 128
// 7.0 and 9.0, 24 of 400 x 801 53.4 and 56.9, 48 101 and 107, 96 195 and 207).
template <typename T>
static int to_map(const void *x, const void *plan, void *out, int64_t planes, int64_t n_src, int64_t OH, int64_t OW, cudaStream_t st,
                  int src_div = 1, bool normalize = false) {
  if constexpr (sizeof(T) == 4) {
    const int64_t by12 = (planes + 11) / 12 * 12, by8 = (planes + 7) / 8 * 8;
    if (planes > 8 && by12 < by8 + (src_div > 1 ? 0 : 1))
      return to_map_launch<T, 12>(x, plan, out, planes, n_src, OH, OW, st, src_div, normalize);
  }
  return to_map_launch<T, 8>(x, plan, out, planes, n_src, OH, OW, st, src_div, normalize);
}

// ---- over plane groups (plane_groups.cuh) ----------------------------------------------------------------------
// The scatter: a thread owns one destination pixel of all PG planes of a group; an entry is one row.  Groups of at most 16
// (96 planes of 20 x 256 x 256 positions onto 1024 x 2048 pixels, transposition apart: 8 planes 0.55 ms, 16 0.48 ms, 32 0.54 ms;
// two entries in flight 0.61 ms; the kernel above 0.74 ms).
template <int PG, bool NORM>
struct ScatterOp {
  PlaneChunks c;
  const float *x;
  const void *plan;
  float *out;
  int n_dst;
  FastDiv stage_tiles, use_tiles;

  size_t stage_smem() const { return stage_aligned(x, c.n_src) ? 0 : kStageBlock<PG>; }
  __device__ __forceinline__ void stage(int p0, char *rows, int tile) const { stage_quad<PG>(x, c.planes, c.n_src, p0, tile, rows); }
  __device__ __forceinline__ void use(int p0, const char *rows, int tile) const {
    constexpr int VP = PG < 8 ? PG : 8, NV = PG / VP;
    const int q = tile * kStageThreads + threadIdx.x;
    if (q >= n_dst) return;
    bool ok;
    const PlanView<float> pv = plan_view<float>(plan, n_dst, ok, c.n_src);
    const int e0 = ok ? __ldg(pv.offsets + q) : 0, e1 = ok ? __ldg(pv.offsets + q + 1) : 0;
    Vec<VP> acc[NV];
#pragma unroll
    for (int i = 0; i < NV; i++) acc[i] = vec_fill<VP>(0.0f);
    float wsum = 0.0f;
    if (e0 < e1) {
      const int *sp = pv.src + e0, *end = pv.src + e1;
      const float *wp = pv.w + e0;
      int s = __ldg(sp);
      float w = __ldg(wp);
      for (;;) {
        const char *row = rows + (size_t)(unsigned)s * (PG * 4);
        const bool fine = index_ok(s, pv.n_src);
        const float we = w;
        sp++;
        wp++;
        const bool more = sp < end;
        if (more) {  // the next entry's source and weight travel with this one's row
          s = __ldg(sp);
          w = __ldg(wp);
        }
        if (fine) {
          Vec<VP> v[NV];
#pragma unroll
          for (int i = 0; i < NV; i++) v[i] = row_load<VP>(row, i * (VP * 4));
#pragma unroll
          for (int i = 0; i < NV; i++) acc[i] = vec_add<VP>(acc[i], vec_scale<VP>(we, v[i]));
          if (NORM) wsum += we;
        }
        if (!more) break;
      }
      if (NORM) {
#pragma unroll
        for (int i = 0; i < NV; i++) divide_all(acc[i].f, wsum + 1e-12f);
      }
    }
#pragma unroll
    for (int i = 0; i < NV; i++) store_planes<VP>(out, n_dst, q, p0 + i * VP, c.planes, acc[i]);
  }
};

template <int PG>
static int to_map_groups(const PlaneChunks &c, const void *x, const void *plan, void *out, int64_t n_src, int64_t n_dst, bool normalize,
                         cudaStream_t st) {
  const FastDiv ts = FastDiv::make(stage_tiles<PG>(n_src)), tu = FastDiv::make(cdiv(n_dst, kStageThreads));
  if (normalize)
    return launch_plane_groups(ScatterOp<PG, true>{c, (const float *)x, plan, (float *)out, (int)n_dst, ts, tu}, 0, st);
  return launch_plane_groups(ScatterOp<PG, false>{c, (const float *)x, plan, (float *)out, (int)n_dst, ts, tu}, 0, st);
}

template <int PG, int INTERP, bool WEIGHTED>
struct GatherOp {
  PlaneChunks c;
  const float *x, *map, *iw;
  float *y;
  int n, H, W, P;
  TileGrid grid;
  FastDiv stage_tiles, use_tiles;

  size_t stage_smem() const { return stage_aligned(x, c.n_src) ? 0 : kStageBlock<PG>; }
  __device__ __forceinline__ void stage(int p0, char *rows, int tile) const { stage_quad<PG>(x, c.planes, c.n_src, p0, tile, rows); }
  __device__ __forceinline__ void use(int p0, const char *rows, int tile) const {
    constexpr int VP = Split<PG>::VP, LP = Split<PG>::LP;
    const int i = grid.output<PG>(tile, threadIdx.x / LP);
    if (i < 0) return;
    rows += threadIdx.x % LP * (VP * 4);
    Vec<VP> acc = vec_fill<VP>(0.0f);
    for (int q = 0; q < (WEIGHTED ? P : 1); q++) {
      const size_t e = (size_t)i * (WEIGHTED ? P : 1) + q;
      const RowTaps t = row_taps<INTERP>(__ldg(map + 2 * e), __ldg(map + 2 * e + 1), H, W, PG * 4);
      const Vec<VP> v = row_gather<VP, INTERP>(rows, t);
      acc = WEIGHTED ? vec_add<VP>(acc, vec_scale<VP>(__ldg(iw + e), v)) : v;
    }
    store_planes<VP>(y, n, i, p0 + threadIdx.x % LP * VP, c.planes, acc);
  }
};

template <int PG>
static int from_map_groups(const PlaneChunks &c, const void *x, const void *map, const void *iw, void *y, int64_t H, int64_t W,
                           int64_t MH, int64_t MW, int64_t P, int interp, cudaStream_t st) {
  const int64_t n = MH * MW;
  const TileGrid grid = TileGrid::make<PG>(MH, MW);
  const FastDiv ts = FastDiv::make(stage_tiles<PG>(H * W)), tu = FastDiv::make(grid.tiles<PG>());
  SPH_DISPATCH_INTERP(interp, {
    if (P > 0)
      return launch_plane_groups(GatherOp<PG, INTERP, true>{c, (const float *)x, (const float *)map, (const float *)iw, (float *)y, (int)n,
                                                            (int)H, (int)W, (int)P, grid, ts, tu}, 0, st);
    return launch_plane_groups(GatherOp<PG, INTERP, false>{c, (const float *)x, (const float *)map, nullptr, (float *)y, (int)n, (int)H,
                                                           (int)W, 0, grid, ts, tu}, 0, st);
  });
  return SPH_ERR_INVALID_ARGUMENT;
}

// Voting resample of integer labels through a nearest-neighbour plan: destination pixel o takes the label that most
// of the source pixels mapped onto it carry, the smallest such label on ties, 0 if none does (torch.argmax over a
// vote histogram in the reference: src/cpp/voting_resample_layer.cpp:8-37, core/interpolation.h:249-265).  The
// segment is walked once per entry (segments hold the few source pixels that land on one output pixel), so no
// (pixels x candidates) histogram is materialised.
__global__ void __launch_bounds__(256)
voting_resample_kernel(const int64_t *__restrict__ x, const void *__restrict__ plan_blob, int64_t *__restrict__ out, int n_dst,
                       int n_src, int planes, int64_t num_candidates, int dtype) {
  const int o = blockIdx.x * blockDim.x + threadIdx.x, p = blockIdx.y;
  if (o >= n_dst) return;
  const PlanHeader *h = (const PlanHeader *)plan_blob;
  const bool ok = h->magic == kPlanMagic && h->n_keys == n_dst && h->dtype == dtype && h->n_src == n_src;
  const int *offsets = (const int *)((const char *)plan_blob + h->off_offsets);
  const int *src = (const int *)((const char *)plan_blob + h->off_src);
  const int64_t *xp = x + (size_t)p * n_src;
  const int e0 = ok ? __ldg(offsets + o) : 0, e1 = ok ? __ldg(offsets + o + 1) : 0;
  int64_t best = 0;
  int best_votes = 0;
  for (int i = e0; i < e1; i++) {
    const int64_t li = __ldg(xp + __ldg(src + i));
    if (li < 0 || li >= num_candidates) continue;
    int votes = 0;
    bool first = true;
    for (int j = e0; j < e1; j++)
      if (__ldg(xp + __ldg(src + j)) == li) {
        votes++;
        if (j < i) first = false;
      }
    if (first && (votes > best_votes || (votes == best_votes && li < best))) {
      best = li;
      best_votes = votes;
    }
  }
  out[(size_t)p * n_dst + o] = best;
}

}  // namespace sph

using namespace sph;

SPH_TU_STATUS(resample)

extern "C" size_t sph_staging_bytes(int op, int64_t planes, int64_t n_src, int64_t reads, int dtype) {
  if (dtype != SPH_F32 || planes < 3 || n_src <= 0 || n_src >= ((int64_t)1 << 31)) return 0;
  PlaneChunks c;
  switch (op) {
    // A gather that reads a pixel less than once on average leaves whole sectors of the source untouched, which the
    // transposition would fetch; and the few taps per position of a resampling map do not pay for rows that go through HBM.
    case SPH_STAGE_GATHER:
      c = stage_chunks(planes, n_src, 4);
      if (reads < n_src || c.group_bytes > kStageGroup) return 0;
      break;
    case SPH_STAGE_SCATTER: c = stage_chunks(planes, n_src, 4, kScatterGroup); break;
    case SPH_STAGE_POOL:
      c = stage_chunks(planes, n_src, 4);
      if (reads < n_src) return 0;
      break;
    case SPH_STAGE_ARGMAX: c = stage_chunks(planes, n_src, 5); break;
    default: return 0;
  }
  return stage_fits(c) ? stage_bytes(c) : 0;
}

extern "C" int sph_resample_from_map(const void *x, const void *map, const void *iw, void *y, int64_t B, int64_t C,
                                     int64_t H, int64_t W, int64_t MH, int64_t MW, int64_t P, int dtype, int interp,
                                     void *stream) {
  return sph_resample_from_map_ws(x, map, iw, y, B, C, H, W, MH, MW, P, dtype, interp, nullptr, 0, stream);
}

extern "C" int sph_resample_from_map_ws(const void *x, const void *map, const void *iw, void *y, int64_t B, int64_t C,
                                        int64_t H, int64_t W, int64_t MH, int64_t MW, int64_t P, int dtype, int interp,
                                        void *ws, size_t ws_bytes, void *stream) {
  SPH_RANGE("sph_resample_from_map");
  if (!x || !map || !y || B < 0 || C < 0 || H <= 0 || W <= 0 || MH < 0 || MW < 0 || P < 0 || (P > 0 && !iw))
    return SPH_ERR_INVALID_ARGUMENT;
  if (dtype != SPH_F32 && dtype != SPH_F64) return SPH_ERR_UNSUPPORTED;
  if (interp < 0 || interp > 2) return SPH_ERR_INVALID_ARGUMENT;
  const int64_t n = MH * MW, planes = B * C, lim = (int64_t)1 << 31;
  if (H * W >= lim || n * (P > 0 ? P : 1) * 2 >= lim || planes / 2 >= 65535) return SPH_ERR_TOO_LARGE;
  if (n == 0 || planes == 0) return SPH_OK;
  cudaStream_t st = (cudaStream_t)stream;
  if (dtype == SPH_F32 && planes >= 3 && scratch_ok(ws)) {
    PlaneChunks c = stage_chunks(planes, H * W, 4);
    if (ws_bytes >= stage_bytes(c) && stage_fits(c)) {
      c.buf = (char *)ws;
      SPH_DISPATCH_GROUP(c.group_planes, return from_map_groups<PG>(c, x, map, iw, y, H, W, MH, MW, P, interp, st));
    }
  }
  return dtype == SPH_F32 ? from_map<float>(x, map, iw, y, planes, H, W, MH, MW, P, interp, st)
                          : from_map<double>(x, map, iw, y, planes, H, W, MH, MW, P, interp, st);
}

namespace {
int resample_to_map(const void *x, const void *plan, void *out, int64_t B, int64_t C, int64_t MH, int64_t MW, int64_t OH, int64_t OW,
                    int64_t K, bool normalize, int dtype, void *ws, size_t ws_bytes, void *stream) {
  if (!x || !plan || !out || B < 0 || C < 0 || MH <= 0 || MW <= 0 || OH <= 0 || OW <= 0 || K <= 0) return SPH_ERR_INVALID_ARGUMENT;
  if (dtype != SPH_F32 && dtype != SPH_F64) return SPH_ERR_UNSUPPORTED;
  const int64_t planes = B * C, lim = (int64_t)1 << 31;
  if (OH * OW >= lim || MH * MW * K >= lim || planes / 2 >= 65535) return SPH_ERR_TOO_LARGE;
  if (planes == 0) return SPH_OK;
  cudaStream_t st = (cudaStream_t)stream;
  if (dtype == SPH_F32 && planes >= 3 && K == 1 && scratch_ok(ws)) {
    PlaneChunks c = stage_chunks(planes, MH * MW, 4, kScatterGroup);
    if (ws_bytes >= stage_bytes(c) && stage_fits(c)) {
      c.buf = (char *)ws;
      SPH_DISPATCH_GROUP(c.group_planes, return to_map_groups<PG>(c, x, plan, out, MH * MW, OH * OW, normalize, st));
    }
  }
  return dtype == SPH_F32 ? to_map<float>(x, plan, out, planes, MH * MW, OH, OW, st, (int)K, normalize)
                          : to_map<double>(x, plan, out, planes, MH * MW, OH, OW, st, (int)K, normalize);
}
}  // namespace

extern "C" int sph_resample_to_map_ws(const void *x, const void *plan, void *out, int64_t B, int64_t C, int64_t MH, int64_t MW,
                                      int64_t OH, int64_t OW, int normalize, int dtype, void *ws, size_t ws_bytes, void *stream) {
  SPH_RANGE("sph_resample_to_map");
  return resample_to_map(x, plan, out, B, C, MH, MW, OH, OW, 1, normalize != 0, dtype, ws, ws_bytes, stream);
}

extern "C" int sph_resample_to_map(const void *x, const void *plan, void *out, int64_t B, int64_t C, int64_t MH,
                                   int64_t MW, int64_t OH, int64_t OW, int dtype, void *stream) {
  SPH_RANGE("sph_resample_to_map");
  return resample_to_map(x, plan, out, B, C, MH, MW, OH, OW, 1, false, dtype, nullptr, 0, stream);
}

extern "C" int sph_resample_to_map_normalized(const void *x, const void *plan, void *out, int64_t B, int64_t C, int64_t MH,
                                              int64_t MW, int64_t OH, int64_t OW, int dtype, void *stream) {
  SPH_RANGE("sph_resample_to_map_normalized");
  return resample_to_map(x, plan, out, B, C, MH, MW, OH, OW, 1, true, dtype, nullptr, 0, stream);
}

extern "C" int sph_mapped_avg_unpool(const void *g, const void *plan, void *grad_in, int64_t B, int64_t C, int64_t IH,
                                     int64_t IW, int64_t OH, int64_t OW, int64_t K, int dtype, void *stream) {
  SPH_RANGE("sph_mapped_avg_unpool");
  return resample_to_map(g, plan, grad_in, B, C, OH, OW, IH, IW, K, false, dtype, nullptr, 0, stream);
}

extern "C" int sph_resample_from_uv_maps(const void *tex, const int64_t *quad_idx, const void *tex_uv, void *out, int64_t B,
                                         int64_t C, int64_t NT, int64_t TH, int64_t TW, int64_t IH, int64_t IW, int dtype,
                                         int interp, void *stream) {
  SPH_RANGE("sph_resample_from_uv_maps");
  if (!tex || !quad_idx || !tex_uv || !out || B < 0 || C < 0 || NT <= 0 || TH <= 0 || TW <= 0 || IH < 0 || IW < 0 ||
      interp < 0 || interp > 2)
    return SPH_ERR_INVALID_ARGUMENT;
  if (dtype != SPH_F32 && dtype != SPH_F64) return SPH_ERR_UNSUPPORTED;
  const int64_t n = IH * IW, planes = B * C, lim = (int64_t)1 << 31;
  if (NT * TH * TW >= lim || n * 2 >= lim || planes / 2 >= 65535) return SPH_ERR_TOO_LARGE;
  if (n == 0 || planes == 0) return SPH_OK;
  cudaStream_t st = (cudaStream_t)stream;
  return dtype == SPH_F32 ? from_map<float>(tex, tex_uv, nullptr, out, planes, TH, TW, IH, IW, 0, interp, st, quad_idx, (int)NT)
                          : from_map<double>(tex, tex_uv, nullptr, out, planes, TH, TW, IH, IW, 0, interp, st, quad_idx, (int)NT);
}

extern "C" int sph_voting_resample_to_map(const int64_t *labels, const void *plan, int plan_dtype, int64_t *out, int64_t B,
                                          int64_t C, int64_t IH, int64_t IW, int64_t OH, int64_t OW, int64_t num_candidates,
                                          void *stream) {
  SPH_RANGE("sph_voting_resample_to_map");
  if (!labels || !plan || !out || B < 0 || C < 0 || IH <= 0 || IW <= 0 || OH <= 0 || OW <= 0 || num_candidates <= 0)
    return SPH_ERR_INVALID_ARGUMENT;
  if (plan_dtype != SPH_F32 && plan_dtype != SPH_F64) return SPH_ERR_UNSUPPORTED;
  const int64_t planes = B * C, lim = (int64_t)1 << 31;
  if (OH * OW >= lim || IH * IW >= lim || planes >= 65535) return SPH_ERR_TOO_LARGE;
  if (planes == 0) return SPH_OK;
  voting_resample_kernel<<<dim3(cdiv(OH * OW, 256), (unsigned)planes), 256, 0, (cudaStream_t)stream>>>(
      labels, plan, out, (int)(OH * OW), (int)(IH * IW), (int)planes, num_candidates, plan_dtype);
  return launch_status();
}
