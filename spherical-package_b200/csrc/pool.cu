// Mapped max pooling (forward: value + argmax index; argmax backward) and mapped average pooling (forward).
#include <float.h>

#include "common.cuh"
#include "plan_walk.cuh"
#include "plane_groups.cuh"

namespace sph {

// out[p,o] = max over the K map slots of output position o, first strict
// maximum, starting from -FLT_MAX as the reference's CUDA build does
// (ext_modules/include/common/mapped_max_pool.h:27-51).  idx is the offset of
// the winning slot's x coordinate in the flattened map (line 49).  One thread
// per output position walks kPlanesPerThread planes; the whole batch is one
// launch (the reference launches once per image:
// src/cuda/mapped_max_pooling_layer.cu:11-36).
//
// AVG = true turns the same walk into mapped average pooling: the K slot values are added in slot order and the sum
// is divided by K (ext_modules/include/common/mapped_avg_pool.h:12-39, 71-107); idx is not written.
//
// Bound: latency and issue.  A block's outputs are 256 in a row: in tiles of 64 x 4, which suit the kernel below, average pooling of 64
// planes of 320 x 641 takes 63.9 us instead of 54.6, weighted max pooling of 8 planes of 256 x 512 73 instead of 46, float64 max pooling
// of 256 planes of 130 x 261 95 instead of 72.
template <typename T, int INTERP, bool WEIGHTED, bool AVG>
__global__ void __launch_bounds__(256)
max_pool_kernel(const T *__restrict__ x, const T *__restrict__ map, const T *__restrict__ iw, T *__restrict__ out,
                int64_t *__restrict__ idx, int n, int planes, int H, int W, int K, int P) {
  const int o = blockIdx.x * blockDim.x + threadIdx.x;
  if (o >= n) return;
  const int p0 = blockIdx.y * kPlanesPerThread;
  const int np = min(kPlanesPerThread, planes - p0);
  const size_t hw = (size_t)H * W;
  const T *xp = x + (size_t)p0 * hw;
  const int PP = WEIGHTED ? P : 1;
  T best[kPlanesPerThread];
  int bk[kPlanesPerThread];
#pragma unroll
  for (int j = 0; j < kPlanesPerThread; j++) { best[j] = AVG ? T(0) : (T)(-FLT_MAX); bk[j] = -1; }
  for (int k = 0; k < K; k++) {
    const size_t e = ((size_t)o * K + k) * PP;
    if (!WEIGHTED) {
      Taps<T> t;
      decode<T, INTERP>(__ldg(map + 2 * e), __ldg(map + 2 * e + 1), H, W, t);
#pragma unroll
      for (int j = 0; j < kPlanesPerThread; j++)
        if (j < np) {
          const T v = gather<T, INTERP>(xp + j * hw, t);
          if (AVG) best[j] = RN<T>::add(best[j], v);
          else if (v > best[j]) { best[j] = v; bk[j] = k; }
        }
    } else {
#pragma unroll
      for (int j = 0; j < kPlanesPerThread; j++)
        if (j < np) {
          const T v = gather_slot<T, INTERP, true>(xp + j * hw, map + 2 * e, iw + e, P, H, W);
          if (AVG) best[j] = RN<T>::add(best[j], v);
          else if (v > best[j]) { best[j] = v; bk[j] = k; }
        }
    }
  }
#pragma unroll
  for (int j = 0; j < kPlanesPerThread; j++)
    if (j < np) {
      if (AVG) {
        out[(size_t)(p0 + j) * n + o] = best[j] / (T)K;
      } else {
        out[(size_t)(p0 + j) * n + o] = best[j];
        idx[(size_t)(p0 + j) * n + o] = bk[j] < 0 ? (int64_t)-1 : ((int64_t)o * K + bk[j]) * PP * 2;
      }
    }
}

// Max pooling of unweighted float32 maps of four taps, the planes read where they lie: the kernel above with fewer instructions per
// value where the taps of a warp are squares of pixels, which they are but at the image's edges, and the next slot's coordinates
// fetched with this one's pixels.  Bound: the SM's path to L1 (two to three wavefronts per load of 32 taps two pixels apart, and what
// it fetches from L2, 87 %) and issue (73 %).  3 x 3 gnomonic map of stride 2, 1024 planes of 256 x 512: the kernel above on blocks of
// 256 outputs of a row 547 us, over plane groups 568; on blocks of 32 x 8 447; so 407, on blocks of 64 x 4 385.  (Five blocks per SM
// 421, six 433; sixteen planes per thread 466, four 453; three slots at a time, so that their lines are fetched once, 434: it fetches
// a third and holds 80 registers; pairs as eight-byte loads where a warp's are aligned: 405, odd widths 463.)
template <int INTERP>
__global__ void __launch_bounds__(256, 4)
max_pool_square_kernel(const float *__restrict__ x, const float *__restrict__ map, float *__restrict__ out, int64_t *__restrict__ idx,
                       BlockTile bt, int planes, int H, int W, int K) {
  constexpr int PPT = kPlanesPerThread;
  const int o = bt.output(), n = bt.width * bt.height;
  if (o < 0) return;
  const int p0 = blockIdx.y * PPT, np = min(PPT, planes - p0);
  const size_t hw = (size_t)H * W;
  const float *xp = x + (size_t)p0 * hw, *m = map + 2 * (size_t)o * K;
  const bool pairs = ((uintptr_t)map & 7) == 0;
  const unsigned active = __activemask();
  float best[PPT];
  int bk[PPT];
#pragma unroll
  for (int j = 0; j < PPT; j++) { best[j] = -FLT_MAX; bk[j] = -1; }
  float2 next = pairs ? __ldg((const float2 *)m) : make_float2(__ldg(m), __ldg(m + 1));
#pragma unroll 1
  for (int k = 0; k < K; k++) {
    const float2 xy = next;
    m += 2;
    if (k + 1 < K) next = pairs ? __ldg((const float2 *)m) : make_float2(__ldg(m), __ldg(m + 1));
    Taps<float> t;
    decode<float, INTERP>(xy.x, xy.y, H, W, t);
    if (__all_sync(active, np == PPT && square_taps(t, W))) {
      const float *at = xp + t.off[0];
#pragma unroll
      for (int j = 0; j < PPT; j++, at += hw) {
        const float v = gather_square(at, W, t);
        if (v > best[j]) { best[j] = v; bk[j] = k; }
      }
    } else {
#pragma unroll
      for (int j = 0; j < PPT; j++)
        if (j < np) {
          const float v = gather<float, INTERP>(xp + j * hw, t);
          if (v > best[j]) { best[j] = v; bk[j] = k; }
        }
    }
  }
#pragma unroll
  for (int j = 0; j < PPT; j++)
    if (j < np) {
      __stcs(out + (size_t)(p0 + j) * n + o, best[j]);
      __stcs((long long *)idx + (size_t)(p0 + j) * n + o, bk[j] < 0 ? -1ll : ((long long)o * K + bk[j]) * 2);
    }
}

// Whether neighbouring positions of a map read neighbouring pixels: 256 pairs spread over it, slot 0; *flag = 1 if three quarters
// of the pairs are at most 8 pixels apart in both directions, else 2.  (Multiples of the golden section of 2^32: positions at equal
// distances would all lie in one column, and be pairs across the end of a row, where that distance is a multiple of the width.)
__global__ void __launch_bounds__(256) map_locality_kernel(const float *__restrict__ map, long long n, int K, int *flag) {
  const long long o = (long long)__umul64hi((unsigned long long)(threadIdx.x * 0x9e3779b9u) << 32, (unsigned long long)n);
  const float *a = map + 2 * (size_t)(o * K), *b = a + 2 * (o + 1 < n ? K : 0);
  const bool near = fabsf(__ldg(b) - __ldg(a)) <= 8.0f && fabsf(__ldg(b + 1) - __ldg(a + 1)) <= 8.0f;
  const int c = __syncthreads_count(near);
  if (threadIdx.x == 0) *(volatile int *)flag = c >= 192 ? 1 : 2;
}

// Nearest-neighbour, unweighted pooling with at most kPoolMaxK slots: the K tap offsets of the output position are
// decoded first and kept in registers, then every plane issues its K loads back to back (no load depends on
// another), which is what lets the kernel run at memory speed instead of at K round-trip latencies per plane.
constexpr int kPoolMaxK = 16;

template <typename T, int PPT, int KMAX>
__global__ void __launch_bounds__(256)
max_pool_nearest_kernel(const T *__restrict__ x, const T *__restrict__ map, T *__restrict__ out, int64_t *__restrict__ idx,
                        int n, int planes, int H, int W, int K) {
  const int o = blockIdx.x * blockDim.x + threadIdx.x;
  if (o >= n) return;
  const int p0 = blockIdx.y * PPT;
  const int np = min(PPT, planes - p0);
  const size_t hw = (size_t)H * W;
  int off[KMAX];
#pragma unroll
  for (int k = 0; k < KMAX; k++) {
    off[k] = -1;
    if (k < K) {
      Taps<T> t;
      const size_t e = (size_t)o * K + k;
      decode<T, SPH_NEAREST>(__ldg(map + 2 * e), __ldg(map + 2 * e + 1), H, W, t);
      off[k] = t.off[0];
    }
  }
  T v[PPT][KMAX];
#pragma unroll
  for (int j = 0; j < PPT; j++) {
    const T *plane = x + (size_t)(p0 + (j < np ? j : 0)) * hw;
#pragma unroll
    for (int k = 0; k < KMAX; k++) v[j][k] = (k < K && off[k] >= 0) ? __ldg(plane + off[k]) : T(0);
  }
#pragma unroll
  for (int j = 0; j < PPT; j++) {
    if (j >= np) break;
    T best = (T)(-FLT_MAX);
    int bk = -1;
#pragma unroll
    for (int k = 0; k < KMAX; k++)
      if (k < K && v[j][k] > best) { best = v[j][k]; bk = k; }
    out[(size_t)(p0 + j) * n + o] = best;
    idx[(size_t)(p0 + j) * n + o] = bk < 0 ? (int64_t)-1 : ((int64_t)o * K + bk) * 2;
  }
}

// Argmax backward: the gradient of output (p,o) goes back through the one
// map slot idx names (common/mapped_max_pool.h:60-78, 136-171).  grad_in is
// zeroed first; contributions are added with red.global.add as in the
// reference's CUDA kernel (cuda/mapped_max_pool.cuh:57-95).
template <typename T, int INTERP, bool WEIGHTED>
__global__ void __launch_bounds__(256)
max_unpool_kernel(const T *__restrict__ g, const int64_t *__restrict__ idx, const T *__restrict__ map,
                  const T *__restrict__ iw, T *__restrict__ gin, int n, int planes, int H, int W, int P,
                  int64_t map_elems) {
  const int o = blockIdx.x * blockDim.x + threadIdx.x;
  if (o >= n) return;
  const int p0 = blockIdx.y * kPlanesPerThread;
  const int np = min(kPlanesPerThread, planes - p0);
  const size_t hw = (size_t)H * W;
  const int PP = WEIGHTED ? P : 1;
  for (int j = 0; j < np; j++) {
    const size_t at = (size_t)(p0 + j) * n + o;
    const int64_t s = idx[at];
    if (s < 0 || s + 2 * PP > map_elems) continue;
    const T v = g[at];
    T *plane = gin + (size_t)(p0 + j) * hw;
    Taps<T> t;
    for (int q = 0; q < PP; q++) {
      decode<T, INTERP>(__ldg(map + s + 2 * q), __ldg(map + s + 2 * q + 1), H, W, t);
      const T vq = WEIGHTED ? __ldg(iw + s / 2 + q) * v : v;
#pragma unroll
      for (int i = 0; i < TapCount<INTERP>::value; i++)
        if (t.off[i] >= 0) atomicAdd(plane + t.off[i], INTERP == SPH_NEAREST ? vq : t.w[i] * vq);
    }
  }
}

// Deterministic argmax backward.  `plan_blob` is a scatter plan built over the FLATTENED map slots
// (sph_plan_build with n_src = OH*OW*K positions and K = 1), so the segment of input pixel q lists every
// (output position o, slot k) whose taps touch q, as s = o*K + k, in map order, with the tap weight.  The pixel sums,
// in that fixed order, the entries whose slot is the one the forward pass selected: idx[p,o] == s * 2 * PP.  No
// zero-fill, no atomics, results independent of scheduling (the reference scatters with atomicAdd:
// ext_modules/include/cuda/mapped_max_pool.cuh:57-95).  The plan is walked warp-cooperatively (plan_walk.cuh).
// STAGED: the winning slot of every output of the CTA's PL planes is first decoded into shared memory as one byte
// (255 = none), so the per-entry test reads a byte of shared memory instead of 8 random bytes of idx.
template <typename T, int PL, bool STAGED>
__global__ void __launch_bounds__(1024)
max_unpool_plan_kernel(const T *__restrict__ g, const int64_t *__restrict__ idx, const void *__restrict__ plan_blob,
                       T *__restrict__ gin, int n, int n_dst, int planes, int K, int PP, int chunk, FastDiv divK) {
  extern __shared__ unsigned char unpool_smem[];
  T *cbuf = (T *)unpool_smem;
  uint8_t *ksm = unpool_smem + (size_t)(blockDim.x >> 5) * walk_smem_per_warp<T, PL>();  // [PL][n]
  const int p0 = blockIdx.y * PL;
  const int np = min(PL, planes - p0);
  if (STAGED) {
    for (int j = 0; j < PL; j++)
      for (int o = threadIdx.x; o < n; o += blockDim.x) {
        int k = -1;
        if (j < np) {
          const int64_t s = __ldg(idx + (size_t)(p0 + j) * n + o);
          if (s >= 0) {
            const int64_t slot = s / (2 * PP), kk = slot - (int64_t)o * K;
            if (kk >= 0 && kk < K && slot * 2 * PP == s) k = (int)kk;
          }
        }
        ksm[(size_t)j * n + o] = k < 0 ? (uint8_t)255 : (uint8_t)k;
      }
    __syncthreads();
  }
  bool ok;
  const PlanView<T> plan = plan_view<T>(plan_blob, n_dst, ok, n * K);
  const int q_begin = blockIdx.x * chunk, q_end = min(q_begin + chunk, n_dst);
  const T *gp = g + (size_t)p0 * n;
  const int64_t *ip = idx + (size_t)p0 * n;
  struct Slot { int o, k, s; };
  plan_walk<T, PL>(plan, ok, n_dst, q_begin, q_end, cbuf,
                          [&](int s) {
                            const int o = (int)divK.div((unsigned)s);
                            return Slot{o, s - o * K, s};
                          },
                          [&](const Slot &e, T w, int j) {
                            const bool hit = STAGED ? ksm[j * n + e.o] == (uint8_t)e.k
                                                    : __ldg(ip + (size_t)j * n + e.o) == (int64_t)e.s * 2 * PP;
                            return hit ? w * __ldg(gp + (size_t)j * n + e.o) : T(0);
                          },
                          gin + (size_t)p0 * n_dst, np);
}

// ---- over plane groups (plane_groups.cuh) ----------------------------------------------------------------------
// Max / average pooling.  TABLE: the taps of the tile's outputs are decoded once into shared memory for the PG / 4 threads
// of every output (groups of 16 or 32 planes); else every thread decodes its own.
template <int PG, int INTERP, bool WEIGHTED, bool AVG>
struct PoolOp {
  static constexpr int VP = Split<PG>::VP, LP = Split<PG>::LP, TO = Split<PG>::TO;
  static constexpr bool TABLE = LP > 1 && !WEIGHTED;
  PlaneChunks c;
  const float *x, *map, *iw;
  float *out;
  int64_t *idx;
  int n, H, W, K, P;
  TileGrid grid;
  FastDiv stage_tiles, use_tiles;

  bool table;  // the tap table fits the shared memory a block has without opting in

  static size_t table_bytes(int64_t K) {
    const size_t b = TABLE ? (size_t)K * TO * (INTERP == SPH_NEAREST ? 4 : 32) : 0;
    return b <= 48 * 1024 ? b : 0;
  }

  size_t stage_smem() const { return stage_aligned(x, c.n_src) ? 0 : kStageBlock<PG>; }
  __device__ __forceinline__ void stage(int p0, char *rows, int tile) const { stage_quad<PG>(x, c.planes, c.n_src, p0, tile, rows); }
  __device__ __forceinline__ void use(int p0, const char *rows, int tile) const {
    extern __shared__ __align__(16) unsigned char pool_table[];
    unsigned *near_off = (unsigned *)pool_table;                       // nearest: [K][TO] offsets
    uint4 *tab_off = (uint4 *)pool_table;                              // else [K][TO] offsets, then [K][TO] weights
    float4 *tab_w = (float4 *)pool_table + (size_t)K * TO;
    const int ol = threadIdx.x / LP, o = grid.output<PG>(tile, ol);
    if (TABLE && table) {
      for (int e = threadIdx.x; e < K * TO; e += kStageThreads) {
        const int k = e / TO, oo = grid.output<PG>(tile, e % TO);
        const float *m = map + 2 * ((size_t)max(oo, 0) * K + k);
        const RowTaps t = row_taps<INTERP>(__ldg(m), __ldg(m + 1), H, W, PG * 4);
        if (INTERP == SPH_NEAREST) {
          near_off[e] = t.off.x;
        } else {
          tab_off[e] = t.off;
          tab_w[e] = t.w;
        }
      }
      __syncthreads();
    }
    if (o < 0) return;
    const int PP = WEIGHTED ? P : 1;
    const float *m = map + 2 * (size_t)o * K * PP;
    const float *wgt = WEIGHTED ? iw + (size_t)o * K * PP : nullptr;
    rows += threadIdx.x % LP * (VP * 4);
    p0 += threadIdx.x % LP * VP;
    Vec<VP> best = vec_fill<VP>(AVG ? 0.0f : -FLT_MAX);
    int bk[VP];
#pragma unroll
    for (int j = 0; j < VP; j++) bk[j] = -1;
    constexpr int UNROLL = INTERP == SPH_NEAREST && !WEIGHTED ? 3 : 1;
#pragma unroll UNROLL
    for (int k = 0; k < K; k++) {
      Vec<VP> v;
      if (WEIGHTED) {
        v = vec_fill<VP>(0.0f);
        for (int q = 0; q < P; q++) {
          const int e = k * P + q;
          const RowTaps t = row_taps<INTERP>(__ldg(m + 2 * e), __ldg(m + 2 * e + 1), H, W, PG * 4);
          v = vec_add<VP>(v, vec_scale<VP>(__ldg(wgt + e), row_gather<VP, INTERP>(rows, t)));
        }
      } else {
        RowTaps t;
        if (!TABLE || !table) {
          t = row_taps<INTERP>(__ldg(m + 2 * k), __ldg(m + 2 * k + 1), H, W, PG * 4);
        } else if (INTERP == SPH_NEAREST) {
          t.off.x = near_off[k * TO + ol];
        } else {
          t.off = tab_off[k * TO + ol];
          t.w = tab_w[k * TO + ol];
        }
        v = row_gather<VP, INTERP>(rows, t);
      }
      if (AVG) {
        best = vec_add<VP>(best, v);
      } else {
#pragma unroll
        for (int j = 0; j < VP; j++)
          if (v.f[j] > best.f[j]) { best.f[j] = v.f[j]; bk[j] = k; }
      }
    }
    if (AVG) {
#pragma unroll
      for (int j = 0; j < VP; j++) best.f[j] = best.f[j] / (float)K;
    }
    store_planes<VP>(out, n, o, p0, c.planes, best);
    if (!AVG) {
      const long long first = (long long)o * K;
      long long *ip = (long long *)idx + (size_t)p0 * n + o;
#pragma unroll
      for (int j = 0; j < VP; j++)
        if (p0 + j < c.planes) __stcs(ip + (size_t)j * n, bk[j] < 0 ? -1ll : (first + bk[j]) * (2 * PP));
    }
  }
};

// Deterministic argmax backward.  Behind a group's gradient rows lie the PG winning slots of every output as bytes
// (kNoSlot: none).  With all slots below 128, a byte b of (winners ^ slot in every byte) + 0x7f.. keeps its top bit clear
// exactly where the slots are equal: two instructions test four planes, and only threads with a winner read the gradient.
constexpr unsigned kNoSlot = 127u;
template <int PG>
struct UnpoolOp {
  PlaneChunks c;
  const float *g;
  const int64_t *idx;
  const void *plan;
  float *gin;
  int n_dst, K, PP;
  TileGrid grid;
  FastDiv divK, div2P, stage_tiles, use_tiles;

  __device__ __forceinline__ size_t winners_at() const { return (size_t)(c.n_src + 1) * PG * 4; }
  size_t stage_smem() const { return stage_aligned(g, c.n_src) ? 0 : kStageBlock<PG>; }
  __device__ __forceinline__ void stage(int p0, char *rows, int tile) const {
    constexpr int LP = PG / 4;
    stage_quad<PG>(g, c.planes, c.n_src, p0, tile, rows);
    const int q = threadIdx.x % LP, o = tile * kStagePixels<PG> + threadIdx.x / LP * 4;
    const int slots = K * 2 * PP;
    p0 += q * 4;
    const long long *ip = (const long long *)idx + (size_t)p0 * c.n_src + o;
    unsigned *w = (unsigned *)(rows + winners_at()) + (size_t)o * LP + q;
    const bool vec = (c.n_src & 3) == 0 && (((uintptr_t)idx) & 15) == 0;
    unsigned win[4] = {0u, 0u, 0u, 0u};
#pragma unroll
    for (int j = 0; j < 4; j++) {
      long long s[4] = {-1, -1, -1, -1};
      if (p0 + j < c.planes && o < c.n_src) {
        if (vec) {
          const longlong2 a = __ldcs((const longlong2 *)(ip + (size_t)j * c.n_src)), b = __ldcs((const longlong2 *)(ip + (size_t)j * c.n_src) + 1);
          s[0] = a.x; s[1] = a.y; s[2] = b.x; s[3] = b.y;
        } else {
#pragma unroll
          for (int i = 0; i < 4; i++)
            if (o + i < c.n_src) s[i] = __ldcs(ip + (size_t)j * c.n_src + i);
        }
      }
#pragma unroll
      for (int i = 0; i < 4; i++) {
        const long long d = s[i] - (long long)(o + i) * slots;  // from this output's slot 0
        unsigned k = kNoSlot;
        if (s[i] >= 0 && d >= 0 && d < slots) {
          const unsigned slot = div2P.div((unsigned)d);
          if (slot * (2 * PP) == (unsigned)d) k = slot;
        }
        win[i] |= k << (8 * j);
      }
    }
#pragma unroll
    for (int i = 0; i < 4; i++)
      if (o + i < c.n_src) w[(size_t)i * LP] = win[i];
  }
  __device__ __forceinline__ void use(int p0, const char *rows, int tile) const {
    constexpr int VP = Split<PG>::VP, LP = Split<PG>::LP, W4 = VP / 4;
    const int q = grid.output<PG>(tile, threadIdx.x / LP);
    if (q < 0) return;
    bool ok;
    const PlanView<float> pv = plan_view<float>(plan, n_dst, ok, c.n_src * K);
    const char *wins = rows + winners_at() + threadIdx.x % LP * VP;
    rows += threadIdx.x % LP * (VP * 4);
    const int e0 = ok ? __ldg(pv.offsets + q) : 0, e1 = ok ? __ldg(pv.offsets + q + 1) : 0;
    Vec<VP> acc = vec_fill<VP>(0.0f);
#pragma unroll 2
    for (int e = e0; e < e1; e++) {
      const int s = __ldg(pv.src + e);
      if (!index_ok(s, pv.n_src)) continue;
      const unsigned o = divK.div((unsigned)s), k4 = ((unsigned)s - o * K) * 0x01010101u;
      unsigned miss[W4], all = 0x80808080u;
      if constexpr (W4 == 2) {
        const uint2 w2 = __ldg((const uint2 *)(wins + o * PG));
        miss[0] = w2.x;
        miss[1] = w2.y;
      } else {
        miss[0] = __ldg((const unsigned *)(wins + o * PG));
      }
#pragma unroll
      for (int i = 0; i < W4; i++) {
        miss[i] = (miss[i] ^ k4) + 0x7f7f7f7fu;
        all &= miss[i];
      }
      if (all != 0x80808080u) {
        const float w = __ldg(pv.w + e);
        const Vec<VP> v = vec_scale<VP>(w, row_load<VP>(rows, o * (PG * 4u)));
#pragma unroll
        for (int j = 0; j < VP; j++)
          if (!(miss[j >> 2] & (0x80u << (8 * (j & 3))))) acc.f[j] = __fadd_rn(acc.f[j], v.f[j]);
      }
    }
    store_planes<VP>(gin, n_dst, q, p0 + threadIdx.x % LP * VP, c.planes, acc);
  }
};

template <int PG>
static int pool_groups(const PlaneChunks &c, const void *x, const void *map, const void *iw, void *out, int64_t *idx, int64_t H, int64_t W,
                       int64_t OH, int64_t OW, int64_t K, int64_t P, int interp, cudaStream_t st, bool avg) {
  const int64_t n = OH * OW;
  const TileGrid grid = TileGrid::make<PG>(OH, OW);
  const FastDiv ts = FastDiv::make(stage_tiles<PG>(H * W)), tu = FastDiv::make(grid.tiles<PG>());
#define SPH_POOL_GROUPS(WEIGHTED, AVG)                                                                                                     \
  do {                                                                                                                                  \
    using Op = PoolOp<PG, INTERP, WEIGHTED, AVG>;                                                                                       \
    const size_t tb = Op::table_bytes(K);                                                                                               \
    return launch_plane_groups(Op{c, (const float *)x, (const float *)map, (const float *)iw, (float *)out, idx, (int)n, (int)H, (int)W, \
                                  (int)K, (int)P, grid, ts, tu, tb > 0}, tb, st);                                                             \
  } while (0)
  SPH_DISPATCH_INTERP(interp, {
    if (P > 0) {
      if (avg) SPH_POOL_GROUPS(true, true);
      SPH_POOL_GROUPS(true, false);
    }
    if (avg) SPH_POOL_GROUPS(false, true);
    SPH_POOL_GROUPS(false, false);
  });
#undef SPH_POOL_GROUPS
  return SPH_ERR_INVALID_ARGUMENT;
}

template <int PG>
static int unpool_groups(const PlaneChunks &c, const void *g, const int64_t *idx, const void *plan, void *gin, int64_t IH, int64_t IW,
                         int64_t K, int64_t P, cudaStream_t st) {
  const int64_t n_dst = IH * IW;
  const TileGrid grid = TileGrid::make<PG>(IH, IW);
  const int PP = (int)(P > 0 ? P : 1);
  return launch_plane_groups(UnpoolOp<PG>{c, (const float *)g, idx, plan, (float *)gin, (int)n_dst, (int)K, PP, grid, FastDiv::make((unsigned)K),
                                          FastDiv::make((unsigned)(2 * PP)), FastDiv::make(stage_tiles<PG>(c.n_src)),
                                          FastDiv::make(grid.tiles<PG>())}, 0, st);
}

template <typename T>
static int unpool_planned(const void *g, const int64_t *idx, const void *plan, void *gin, int64_t planes, int64_t n_dst,
                          int64_t n, int64_t K, int64_t P, cudaStream_t st) {
  const int PP = (int)(P > 0 ? P : 1);
  constexpr int PL = 4;
  const int groups = cdiv(planes, PL);
  const size_t stage = (size_t)PL * n;
  if (K <= 254 && stage + 32 * (size_t)walk_smem_per_warp<T, PL>() <= 200 * 1024) {
    // one CTA of 32 warps per SM (the staged slots fill its shared memory); CTAs = plane groups x pixel chunks
    int chunks = cdiv((int64_t)148 * 2, groups);
    if (chunks > cdiv(n_dst, 1024)) chunks = cdiv(n_dst, 1024);
    const int chunk = cdiv(cdiv(n_dst, chunks), 1024) * 1024;
    const size_t smem = stage + 32 * (size_t)walk_smem_per_warp<T, PL>();
    cudaFuncSetAttribute(max_unpool_plan_kernel<T, PL, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    max_unpool_plan_kernel<T, PL, true><<<dim3(cdiv(n_dst, chunk), groups), 1024, smem, st>>>(
        (const T *)g, idx, plan, (T *)gin, (int)n, (int)n_dst, (int)planes, (int)K, PP, chunk, FastDiv::make((unsigned)K));
  } else {
    int64_t chunks = ((int64_t)148 * 16 + groups - 1) / groups;
    if (chunks > (n_dst + 255) / 256) chunks = (n_dst + 255) / 256;
    const int chunk = (int)(((n_dst + chunks - 1) / chunks + 255) / 256 * 256);
    const size_t smem = 8 * (size_t)walk_smem_per_warp<T, PL>();
    max_unpool_plan_kernel<T, PL, false><<<dim3(cdiv(n_dst, chunk), groups), 256, smem, st>>>(
        (const T *)g, idx, plan, (T *)gin, (int)n, (int)n_dst, (int)planes, (int)K, PP, chunk, FastDiv::make((unsigned)K));
  }
  return launch_status();
}

template <typename T>
static int pool(const void *x, const void *map, const void *iw, void *out, int64_t *idx, int64_t planes, int64_t H,
                int64_t W, int64_t OH, int64_t OW, int64_t K, int64_t P, int interp, cudaStream_t st, bool avg = false) {
  const int n = (int)(OH * OW);
  if (avg) {
    dim3 grid(cdiv(n, 256), cdiv(planes, kPlanesPerThread));
    SPH_DISPATCH_INTERP(interp, {
      if (P > 0)
        max_pool_kernel<T, INTERP, true, true><<<grid, 256, 0, st>>>((const T *)x, (const T *)map, (const T *)iw, (T *)out,
                                                                     nullptr, n, (int)planes, (int)H, (int)W, (int)K, (int)P);
      else
        max_pool_kernel<T, INTERP, false, true><<<grid, 256, 0, st>>>((const T *)x, (const T *)map, nullptr, (T *)out, nullptr,
                                                                      n, (int)planes, (int)H, (int)W, (int)K, 0);
    });
    return launch_status();
  }
  if (interp == SPH_NEAREST && P == 0 && K <= kPoolMaxK) {
    constexpr int PPT = 4;
    dim3 grid(cdiv(n, 256), cdiv(planes, PPT));
#define SPH_POOL_NEAREST(KMAX) \
    max_pool_nearest_kernel<T, PPT, KMAX><<<grid, 256, 0, st>>>((const T *)x, (const T *)map, (T *)out, idx, n, (int)planes, (int)H, (int)W, (int)K)
    if (K <= 4) SPH_POOL_NEAREST(4);
    else if (K <= 9) SPH_POOL_NEAREST(9);
    else SPH_POOL_NEAREST(16);
#undef SPH_POOL_NEAREST
    return launch_status();
  }
  dim3 grid(cdiv(n, 256), cdiv(planes, kPlanesPerThread));
  SPH_DISPATCH_INTERP(interp, {
    if (P > 0)
      max_pool_kernel<T, INTERP, true, false><<<grid, 256, 0, st>>>((const T *)x, (const T *)map, (const T *)iw, (T *)out, idx,
                                                             n, (int)planes, (int)H, (int)W, (int)K, (int)P);
    else if constexpr (sizeof(T) == 4 && INTERP != SPH_NEAREST) {
      const BlockTile sq = BlockTile::make(OH, OW, 6);
      grid.x = sq.blocks();
      max_pool_square_kernel<INTERP><<<grid, 256, 0, st>>>((const float *)x, (const float *)map, (float *)out, idx, sq, (int)planes, (int)H, (int)W,
                                                        (int)K);
    } else
      max_pool_kernel<T, INTERP, false, false><<<grid, 256, 0, st>>>((const T *)x, (const T *)map, nullptr, (T *)out, idx, n,
                                                              (int)planes, (int)H, (int)W, (int)K, 0);
  });
  return launch_status();
}

template <typename T>
static int unpool(const void *g, const int64_t *idx, const void *map, const void *iw, void *gin, int64_t planes,
                  int64_t H, int64_t W, int64_t n, int64_t K, int64_t P, int interp, cudaStream_t st) {
  if (cudaMemsetAsync(gin, 0, sizeof(T) * (size_t)(planes * H * W), st) != cudaSuccess) return SPH_ERR_CUDA;
  dim3 grid(cdiv(n, 256), cdiv(planes, kPlanesPerThread));
  const int64_t map_elems = n * K * (P > 0 ? P : 1) * 2;
  SPH_DISPATCH_INTERP(interp, {
    if (P > 0)
      max_unpool_kernel<T, INTERP, true><<<grid, 256, 0, st>>>((const T *)g, idx, (const T *)map, (const T *)iw, (T *)gin,
                                                               (int)n, (int)planes, (int)H, (int)W, (int)P, map_elems);
    else
      max_unpool_kernel<T, INTERP, false><<<grid, 256, 0, st>>>((const T *)g, idx, (const T *)map, nullptr, (T *)gin, (int)n,
                                                                (int)planes, (int)H, (int)W, 0, map_elems);
  });
  return launch_status();
}

static int check(const void *a, const void *b, const void *c, const void *d, const void *iw, int64_t B, int64_t C,
                 int64_t IH, int64_t IW, int64_t OH, int64_t OW, int64_t K, int64_t P, int dtype, int interp) {
  if (!a || !b || !c || !d || B < 0 || C < 0 || IH <= 0 || IW <= 0 || OH < 0 || OW < 0 || K <= 0 || P < 0 ||
      (P > 0 && !iw) || interp < 0 || interp > 2)
    return SPH_ERR_INVALID_ARGUMENT;
  if (dtype != SPH_F32 && dtype != SPH_F64) return SPH_ERR_UNSUPPORTED;
  const int64_t lim = (int64_t)1 << 31;
  if (IH * IW >= lim || OH * OW * K * (P > 0 ? P : 1) * 2 >= lim || B * C / 4 >= 65535)
    return SPH_ERR_TOO_LARGE;
  return SPH_OK;
}

}  // namespace sph

using namespace sph;

SPH_TU_STATUS(pool)

extern "C" int sph_mapped_pool_ws(const void *x, const void *map, const void *iw, void *out, int64_t *idx, int64_t B, int64_t C,
                                  int64_t IH, int64_t IW, int64_t OH, int64_t OW, int64_t K, int64_t P, int average, int dtype,
                                  int interp, void *ws, size_t ws_bytes, void *stream) {
  SPH_RANGE(average ? "sph_mapped_avg_pool" : "sph_mapped_max_pool");
  const int rc = check(x, map, out, average ? out : (const void *)idx, iw, B, C, IH, IW, OH, OW, K, P, dtype, interp);
  if (rc != SPH_OK) return rc;
  if (B * C == 0 || OH * OW == 0) return SPH_OK;
  cudaStream_t st = (cudaStream_t)stream;
  if (dtype == SPH_F32 && B * C >= 3 && scratch_ok(ws)) {
    PlaneChunks c = stage_chunks(B * C, IH * IW, 4);
    if (ws_bytes >= stage_bytes(c) && stage_fits(c)) {
      c.buf = (char *)ws;
      SPH_DISPATCH_GROUP(c.group_planes, return pool_groups<PG>(c, x, map, iw, out, idx, IH, IW, OH, OW, K, P, interp, st, average != 0));
    }
  }
  return dtype == SPH_F32 ? pool<float>(x, map, iw, out, idx, B * C, IH, IW, OH, OW, K, P, interp, st, average != 0)
                          : pool<double>(x, map, iw, out, idx, B * C, IH, IW, OH, OW, K, P, interp, st, average != 0);
}

extern "C" int sph_map_locality(const void *map, int64_t n, int64_t K, int *flag, void *stream) {
  if (!map || !flag || n <= 0 || K <= 0 || K >= ((int64_t)1 << 31)) return SPH_ERR_INVALID_ARGUMENT;
  map_locality_kernel<<<1, 256, 0, (cudaStream_t)stream>>>((const float *)map, (long long)n, (int)K, flag);
  return launch_status();
}

extern "C" int sph_mapped_max_pool(const void *x, const void *map, const void *iw, void *out, int64_t *idx, int64_t B,
                                   int64_t C, int64_t IH, int64_t IW, int64_t OH, int64_t OW, int64_t K, int64_t P,
                                   int dtype, int interp, void *stream) {
  return sph_mapped_pool_ws(x, map, iw, out, idx, B, C, IH, IW, OH, OW, K, P, 0, dtype, interp, nullptr, 0, stream);
}

extern "C" int sph_mapped_max_unpool(const void *g, const int64_t *idx, const void *map, const void *iw, void *grad_in,
                                     int64_t B, int64_t C, int64_t IH, int64_t IW, int64_t OH, int64_t OW, int64_t K,
                                     int64_t P, int dtype, int interp, void *stream) {
  SPH_RANGE("sph_mapped_max_unpool");
  const int rc = check(g, map, grad_in, idx, iw, B, C, IH, IW, OH, OW, K, P, dtype, interp);
  if (rc != SPH_OK) return rc;
  if (B * C == 0) return SPH_OK;
  cudaStream_t st = (cudaStream_t)stream;
  if (OH * OW == 0)
    return cudaMemsetAsync(grad_in, 0, (dtype == SPH_F64 ? 8 : 4) * (size_t)(B * C * IH * IW), st) == cudaSuccess
               ? SPH_OK : SPH_ERR_CUDA;
  return dtype == SPH_F32 ? unpool<float>(g, idx, map, iw, grad_in, B * C, IH, IW, OH * OW, K, P, interp, st)
                          : unpool<double>(g, idx, map, iw, grad_in, B * C, IH, IW, OH * OW, K, P, interp, st);
}

extern "C" int sph_mapped_max_unpool_planned(const void *g, const int64_t *idx, const void *plan, void *grad_in, int64_t B,
                                             int64_t C, int64_t IH, int64_t IW, int64_t OH, int64_t OW, int64_t K, int64_t P,
                                             int dtype, void *stream) {
  return sph_mapped_max_unpool_ws(g, idx, plan, grad_in, B, C, IH, IW, OH, OW, K, P, dtype, nullptr, 0, stream);
}

extern "C" int sph_mapped_max_unpool_ws(const void *g, const int64_t *idx, const void *plan, void *grad_in, int64_t B, int64_t C,
                                        int64_t IH, int64_t IW, int64_t OH, int64_t OW, int64_t K, int64_t P, int dtype, void *ws,
                                        size_t ws_bytes, void *stream) {
  SPH_RANGE("sph_mapped_max_unpool_planned");
  const int rc = check(g, plan, grad_in, idx, nullptr, B, C, IH, IW, OH, OW, K, 0, dtype, 0);
  if (rc != SPH_OK) return rc;
  if (P < 0 || OH * OW * K >= ((int64_t)1 << 31) / (2 * (P > 0 ? P : 1))) return P < 0 ? SPH_ERR_INVALID_ARGUMENT : SPH_ERR_TOO_LARGE;
  if (B * C == 0) return SPH_OK;
  cudaStream_t st = (cudaStream_t)stream;
  if (OH * OW == 0)
    return cudaMemsetAsync(grad_in, 0, (dtype == SPH_F64 ? 8 : 4) * (size_t)(B * C * IH * IW), st) == cudaSuccess
               ? SPH_OK : SPH_ERR_CUDA;
  if (dtype == SPH_F32 && B * C >= 3 && K < kNoSlot && scratch_ok(ws)) {
    PlaneChunks c = stage_chunks(B * C, OH * OW, 5);
    if (ws_bytes >= stage_bytes(c) && stage_fits(c)) {
      c.buf = (char *)ws;
      SPH_DISPATCH_GROUP(c.group_planes, return unpool_groups<PG>(c, g, idx, plan, grad_in, IH, IW, K, P, st));
    }
  }
  return dtype == SPH_F32 ? unpool_planned<float>(g, idx, plan, grad_in, B * C, IH * IW, OH * OW, K, P, st)
                          : unpool_planned<double>(g, idx, plan, grad_in, B * C, IH * IW, OH * OW, K, P, st);
}

extern "C" int sph_mapped_avg_pool(const void *x, const void *map, const void *iw, void *out, int64_t B, int64_t C, int64_t IH,
                                   int64_t IW, int64_t OH, int64_t OW, int64_t K, int64_t P, int dtype, int interp,
                                   void *stream) {
  return sph_mapped_pool_ws(x, map, iw, out, nullptr, B, C, IH, IW, OH, OW, K, P, 1, dtype, interp, nullptr, 0, stream);
}
