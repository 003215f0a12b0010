// float32 mapped convolutions on the tensor cores, without giving up float32.
//
// A float32 operand is the exact sum of three bf16 parts, x = h + m + l (8 + 8 + 8 significand bits, by truncation), so a
// float32 product is nine bf16 products, of which l*l, m*l and l*m lie below 2^-23 of it.  The other six run on tcgen05
// with float32 accumulation in tensor memory.  What remains to be guarded is the accumulation: the tensor core cuts
// every addition off toward zero (measured on B200: 144 additions of one sign lose 6.6e-6 of the sum, where a chain of
// float32 multiply-adds is off by 7e-7).  So
//   - the large products h*h go to an accumulator of their own, which takes at most kSeg chunks (64 columns, four additions)
//     before the epilogue warps add it, round to nearest, to float32 sums (kept in tensor memory); two such accumulators
//     alternate;
//   - the five small ones go to a second accumulator, whose losses are 2^-7 of the large one's: it takes kRun segments (800
//     additions, ten per chunk: 4e-7) before it is added to the sums too.  (One accumulator for a whole weight gradient of 768 tiles
//     was off by 1.6e-5, so 7e-7, the CUDA cores' sums 1.4e-6; it cost a weight gradient of 70 tiles per block 1.6 %.)
// (Tiles of one segment need no sums: their columns are the small products' second buffer, and the next tile's products run
// while this one's results are stored.)
// The result is at least as close to the exact sum as the SIMT kernels' (conv_simt.cu; tests/test_conv_x3_gpu.py compares
// both with float64).  Infinities and NaNs come out as from float32 arithmetic: see add_small().
//
// The two kernels mirror conv_tc.cu (tiles of 128 pixels, producer warps that gather, weights or gradient tile images by
// bulk copies, one MMA thread, epilogue warps), but gather float32 values from a channels-last float32 copy of the source
// and interpolate in float32, each tap after the first in one fused operation, before the values are split:
//   x3_gemm_kernel   Out[b, n, pix] = sum_j Col[b, pix, j] * Wt[n, j]  (+ bias[n])     through a map, a plan, or the identity
//   x3_dw_kernel     dW[n, j] = sum_{b, pix} G[b, n, pix] * Col[b, pix, j]
//
// Why the tiles are what they are: per chunk of 128 pixels x 32 columns the six products take 768 tensor cycles (N = 128) and
// the SM's 128-byte data path carries 512 wavefronts of gathered taps, 192 + 192 of operand stores and 768 of operand
// reads; 32-column chunks (64-byte swizzled rows, 48 KB a stage for both operands in three parts) leave the L1 room for
// the tile's neighbourhood, which 64-column chunks (96 KB a stage) do not.
#include <float.h>
#include <string.h>

#include <algorithm>

#include "common.cuh"
#include "conv_internal.h"
#include "tc_common.cuh"

namespace sph {
namespace {

using namespace tc;

constexpr int kCols = 32;                               // GEMM columns per chunk
constexpr int kPix = 128, kTileW = 16, kTileH = 8;      // pixels of a tile: 8 rows of 16
constexpr int kEpi = 4, kProd = 16;                     // epilogue and producer warps
constexpr int kThreads3 = 32 * (kEpi + 1 + kProd);
constexpr int kProd0 = 32 * (kEpi + 1);                 // first producer thread
constexpr int kSeg = 2;                                 // chunks per segment of large products; tiles of at most kOneSeg chunks
constexpr int kOneSeg = 4;                              // (the multiply-first product) are one segment
constexpr int kRun = 40;                                // segments that share an accumulator of small products
constexpr int kPartA = kPix * 64;                       // bytes of one part of a 128-row x 32-column operand tile
constexpr int kNMax = 128;
constexpr size_t kSmemMax = 227 * 1024;
// tensor memory columns: large products of a segment (two buffers of 128), small products, float32 sums of finished segments
constexpr uint32_t kHh = 0, kCorr = 256, kSum = 384;

enum { SRC_MAP1 = 0, SRC_MAP4 = 1, SRC_PLAN = 2, SRC_SELF = 3 };

__device__ int g_wait_status3;

int padded3(int64_t CH) {
  if (CH <= 8) return 8;
  if (CH <= 16) return 16;
  return (int)align_up((size_t)CH, 32);
}

// Descriptor of a K-major operand tile stored as rows of 64 bytes (32 bf16) with the 64-byte swizzle (16-byte unit index XOR
// (row >> 1) & 3): 8-row groups 512 bytes apart, layout code 4.
__device__ __forceinline__ uint64_t smem_desc_sw64(uint32_t saddr) {
  return (uint64_t)((saddr >> 4) & 0x3FFFu) | (1ull << 16) | ((uint64_t)(512 >> 4) << 32) | (1ull << 46) | (4ull << 61);
}

struct Src3 {
  const char *xl;            // (B, SH*SW + 1, Cp) channels-last float32; the last pixel of every image is zero
  const float *map, *iw;
  const void *plan;
  int Cp, SH, SW, K, P, GH, GW, interp;
};

struct Ring3 {
  int s = 0;
  uint32_t ph = 0;
  __device__ __forceinline__ void next(int stages) {
    if (++s == stages) { s = 0; ph ^= 1u; }
  }
};

// ---- taps of a tile in shared memory, for slots [s0, s0 + ns): offsets [slot][pixel] (4 or 1), weights [slot][pixel] (4), and in
// plan mode the range of entries beyond the fourth
template <int SRC> struct TapTable {
  static constexpr int NT = SRC == SRC_MAP1 || SRC == SRC_SELF ? 1 : 4;
  static size_t bytes(int ns) { return SRC == SRC_SELF ? 0 : (size_t)ns * kPix * (NT == 1 ? 4 : SRC == SRC_PLAN ? 40 : 32); }
  uint32_t off, w, rest;  // shared-space addresses
  __device__ __forceinline__ TapTable(uint32_t base, int ns) {
    off = base;
    w = off + ns * kPix * (NT * 4);
    rest = w + ns * kPix * 16;
  }
};

__device__ __forceinline__ int tile_pixel3(int l, int ty, int tx, int GH, int GW) {
  const int y = ty * kTileH + (l >> 4), x = tx * kTileW + (l & 15);
  return (y < GH && x < GW) ? y * GW + x : -1;
}

// Two entries at a time: nobody computes meanwhile, and an entry's reads are two round trips to L2 (input gradient of 64 -> 128 channels,
// 8 x 128 x 256: one at a time 555 us, two 531, three, which spill, 561; the map modes, one round trip per entry, lose by it: 330, 349
// and 352).
template <int SRC>
__device__ __forceinline__ void fill_plan3(const Src3 &g, const TapTable<SRC> &t, const PlanView<float> &pv, bool plan_ok, int s0, int ns,
                                           int ty, int tx, int pt) {
  constexpr int U = 2, STEP = 32 * kProd;
  const uint32_t pitch = (uint32_t)g.Cp * 4u, zero = (uint32_t)(g.SH * g.SW) * pitch;
  const auto key = [&](int idx, bool &in) {  // (pixel, slot) of an entry as an index, 0 where there is none
    const int slot = s0 + idx / kPix, pix = tile_pixel3(idx % kPix, ty, tx, g.GH, g.GW);
    in = idx < ns * kPix && pix >= 0 && slot < g.K;
    return in ? (size_t)pix * g.K + slot : (size_t)0;
  };
  const int total = ns * kPix;
#pragma unroll 1
  for (int i0 = pt; i0 < total; i0 += U * STEP) {
    int e0[U], e1[U], sp[U][4];
    float w[U][4];
#pragma unroll
    for (int u = 0; u < U; u++) {
      bool in;
      const int *off = pv.offsets + key(i0 + u * STEP, in);
      in = in && plan_ok;
      e0[u] = in ? __ldg(off) : 0;
      e1[u] = in ? __ldg(off + 1) : 0;
    }
#pragma unroll
    for (int u = 0; u < U; u++)
#pragma unroll
      for (int i = 0; i < 4; i++) {
        const bool in = e0[u] + i < e1[u];
        sp[u][i] = in ? __ldg(pv.src + e0[u] + i) : -1;
        w[u][i] = in ? __ldg(pv.w + e0[u] + i) : 0.0f;
      }
#pragma unroll
    for (int u = 0; u < U; u++) {
      const int idx = i0 + u * STEP;
      if (idx >= ns * kPix) break;
      uint32_t o[4];
#pragma unroll
      for (int i = 0; i < 4; i++) {
        const bool ok = sp[u][i] >= 0 && index_ok(sp[u][i], pv.n_src);
        o[i] = ok ? (uint32_t)sp[u][i] * pitch : zero;
        w[u][i] = ok ? w[u][i] : 0.0f;
      }
      asm volatile("st.shared.v2.u32 [%0], {%1, %2};" ::"r"(t.rest + idx * 8), "r"(min(e0[u] + 4, e1[u])), "r"(e1[u]) : "memory");
      sts128(t.off + idx * 16, make_uint4(o[0], o[1], o[2], o[3]));
      sts128(t.w + idx * 16, make_uint4(__float_as_uint(w[u][0]), __float_as_uint(w[u][1]), __float_as_uint(w[u][2]), __float_as_uint(w[u][3])));
    }
  }
}

template <int SRC>
__device__ __forceinline__ void fill_taps3(const Src3 &g, const TapTable<SRC> &t, const PlanView<float> &pv, bool plan_ok, int s0, int ns,
                                           int ty, int tx, int pt) {
  if (SRC == SRC_SELF) return;
  if (SRC == SRC_PLAN) return fill_plan3<SRC>(g, t, pv, plan_ok, s0, ns, ty, tx, pt);
  const uint32_t pitch = (uint32_t)g.Cp * 4u, zero = (uint32_t)(g.SH * g.SW) * pitch;
  for (int idx = pt; idx < ns * kPix; idx += 32 * kProd) {
    const int slot = s0 + idx / kPix, pix = tile_pixel3(idx % kPix, ty, tx, g.GH, g.GW);
    const bool in = pix >= 0 && slot < g.K;
    if constexpr (SRC == SRC_MAP1) {
      uint32_t o = zero;
      if (in) {
        const float *m = g.map + 2 * ((size_t)pix * g.K + slot);
        Taps<float> q;
        decode<float, SPH_NEAREST>(__ldg(m), __ldg(m + 1), g.SH, g.SW, q);
        if (q.off[0] >= 0 && index_ok(q.off[0], q.limit)) o = (uint32_t)q.off[0] * pitch;
      }
      sts32(t.off + idx * 4, o);
    } else {
      uint32_t o[4] = {zero, zero, zero, zero};
      float w[4] = {0.f, 0.f, 0.f, 0.f};
      if constexpr (SRC == SRC_MAP4) {
        if (in) {
          const size_t e = ((size_t)pix * g.K + slot) * (g.P > 0 ? g.P : 1);
          Taps<float> q;
          if (g.P > 0) {  // weighted nearest, at most four points: the points take the taps' places
#pragma unroll
            for (int i = 0; i < 4; i++)
              if (i < g.P) {
                decode<float, SPH_NEAREST>(__ldg(g.map + 2 * (e + i)), __ldg(g.map + 2 * (e + i) + 1), g.SH, g.SW, q);
                if (q.off[0] >= 0 && index_ok(q.off[0], q.limit)) o[i] = (uint32_t)q.off[0] * pitch;
                w[i] = __ldg(g.iw + e + i);
              }
          } else {
            const float x = __ldg(g.map + 2 * e), y = __ldg(g.map + 2 * e + 1);
            if (g.interp == SPH_BISPHERICAL) decode<float, SPH_BISPHERICAL>(x, y, g.SH, g.SW, q);
            else decode<float, SPH_BILINEAR>(x, y, g.SH, g.SW, q);
#pragma unroll
            for (int i = 0; i < 4; i++) {
              if (q.off[i] >= 0 && index_ok(q.off[i], q.limit)) o[i] = (uint32_t)q.off[i] * pitch;
              w[i] = q.w[i];
            }
          }
        }
      }
      sts128(t.off + idx * 16, make_uint4(o[0], o[1], o[2], o[3]));
      sts128(t.w + idx * 16, make_uint4(__float_as_uint(w[0]), __float_as_uint(w[1]), __float_as_uint(w[2]), __float_as_uint(w[3])));
    }
  }
}

// Eight channels of one source pixel.
struct V8 {
  float f[8];
};
// Two values per instruction: four producer warps per scheduler wait for each other's and their own instructions as long as for their
// reads (a chunk was 240 instructions per warp, issue 48 % busy).  64 -> 128 channels, 8 x 128 x 256, one value per instruction and so:
// forward 330 and 310 us, input gradient 547 and 520, weight gradient 316 and 295.
__device__ __forceinline__ uint64_t pack2(float lo, float hi) {
  uint64_t r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
  return r;
}
__device__ __forceinline__ void unpack2(uint64_t v, float &lo, float &hi) { asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v)); }
__device__ __forceinline__ uint64_t mul2(uint64_t a, uint64_t b) {
  uint64_t r;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ uint64_t fma2(uint64_t a, uint64_t b, uint64_t c) {
  uint64_t r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
  return r;
}
__device__ __forceinline__ uint64_t add2(uint64_t a, uint64_t b) {
  uint64_t r;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ uint64_t sub2(uint64_t a, uint64_t b) {
  uint64_t r;
  asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ V8 load8(const char *p) {
  V8 v;
  asm volatile("ld.global.nc.v8.f32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
               : "=f"(v.f[0]), "=f"(v.f[1]), "=f"(v.f[2]), "=f"(v.f[3]), "=f"(v.f[4]), "=f"(v.f[5]), "=f"(v.f[6]), "=f"(v.f[7])
               : "l"(p));
  return v;
}

// The loads of one (pixel, slot, 8 channels) item, issued ahead of their use.
template <int SRC> struct Item {
  static constexpr int NT = TapTable<SRC>::NT;
  V8 q[NT];
  float w[NT];
};
template <int SRC>
__device__ __forceinline__ void item_load(Item<SRC> &it, const TapTable<SRC> &t, const char *img, int entry, uint32_t self_off) {
  if constexpr (SRC == SRC_SELF) {
    it.q[0] = load8(img + self_off);
  } else if constexpr (SRC == SRC_MAP1) {
    uint32_t o;
    asm volatile("ld.shared.u32 %0, [%1];" : "=r"(o) : "r"(t.off + entry * 4));
    it.q[0] = load8(img + o);
  } else {
    const uint4 o = lds128(t.off + entry * 16), w = lds128(t.w + entry * 16);
    it.q[0] = load8(img + o.x);
    it.q[1] = load8(img + o.y);
    it.q[2] = load8(img + o.z);
    it.q[3] = load8(img + o.w);
    it.w[0] = __uint_as_float(w.x);
    it.w[1] = __uint_as_float(w.y);
    it.w[2] = __uint_as_float(w.z);
    it.w[3] = __uint_as_float(w.w);
  }
}
template <int SRC>
__device__ __forceinline__ V8 item_value(const Item<SRC> &it, const TapTable<SRC> &t, const PlanView<float> &pv, const char *img, int entry,
                                         uint32_t pitch) {
  V8 v;
  if constexpr (Item<SRC>::NT == 1) {
    v = it.q[0];
  } else {
    uint64_t w[4];
#pragma unroll
    for (int i = 0; i < 4; i++) w[i] = pack2(it.w[i], it.w[i]);
#pragma unroll
    for (int j = 0; j < 8; j += 2) {
      uint64_t a = mul2(w[0], pack2(it.q[0].f[j], it.q[0].f[j + 1]));
#pragma unroll
      for (int i = 1; i < 4; i++) a = fma2(w[i], pack2(it.q[i].f[j], it.q[i].f[j + 1]), a);
      unpack2(a, v.f[j], v.f[j + 1]);
    }
  }
  if constexpr (SRC == SRC_PLAN) {
    const uint2 r = lds64(t.rest + entry * 8);
    if (r.x < r.y) {
      // Segments longer than the table: the next entry's index and weight are on their way with this one's row.  (Each entry's
      // loads in turn: 691 us for the input gradient of 64 -> 128 channels, 8 x 128 x 256; so 565 us; four rows in flight
      // spill, 975 us.)
      int s = __ldg(pv.src + r.x);
      float w = __ldg(pv.w + r.x);
      for (int e = (int)r.x + 1;; e++) {
        const bool ok = index_ok(s, pv.n_src);
        const V8 x = load8(img + (size_t)(ok ? s : 0) * pitch);
        const float we = ok ? w : 0.0f;
        const bool more = e < (int)r.y;
        if (more) {
          s = __ldg(pv.src + e);
          w = __ldg(pv.w + e);
        }
        const uint64_t w2 = pack2(we, we);
#pragma unroll
        for (int j = 0; j < 8; j += 2)
          unpack2(fma2(w2, pack2(x.f[j], x.f[j + 1]), pack2(v.f[j], v.f[j + 1])), v.f[j], v.f[j + 1]);
        if (!more) break;
      }
    }
  }
  return v;
}

__device__ __forceinline__ float upper(float x) { return __uint_as_float(__float_as_uint(x) & 0xffff0000u); }
// x = h + m + l by truncation; the parts of eight values as three 16-byte vectors, stored `part` bytes apart.
__device__ __forceinline__ void store_parts(uint32_t dst, uint32_t part, const V8 &v) {
  uint32_t h[4], m[4], l[4];
#pragma unroll
  for (int i = 0; i < 4; i++) {
    const float a = v.f[2 * i], b = v.f[2 * i + 1];
    float ra, rb, la, lb;
    const uint64_t rest = sub2(pack2(a, b), pack2(upper(a), upper(b)));
    unpack2(rest, ra, rb);
    unpack2(sub2(rest, pack2(upper(ra), upper(rb))), la, lb);
    h[i] = __byte_perm(__float_as_uint(a), __float_as_uint(b), 0x7632);
    m[i] = __byte_perm(__float_as_uint(ra), __float_as_uint(rb), 0x7632);
    l[i] = __byte_perm(__float_as_uint(la), __float_as_uint(lb), 0x7632);
  }
  sts128(dst, make_uint4(h[0], h[1], h[2], h[3]));
  sts128(dst + part, make_uint4(m[0], m[1], m[2], m[3]));
  sts128(dst + 2 * part, make_uint4(l[0], l[1], l[2], l[3]));
}

__device__ __forceinline__ void producer_bar3() { asm volatile("bar.sync 1, %0;" ::"n"(32 * kProd) : "memory"); }

struct Bars {
  uint64_t *full, *empty, *seg_full, *seg_empty, *corr_empty;
  uint32_t *tmem_ptr;
  volatile int *abort_flag;
};
inline size_t bars_bytes(int stages) { return 8 * (2 * stages + 6) + 16; }
__device__ __forceinline__ Bars carve_bars(uint8_t *q, int stages) {
  Bars b;
  b.full = (uint64_t *)q;
  b.empty = b.full + stages;
  b.seg_full = b.empty + stages;
  b.seg_empty = b.seg_full + 2;
  b.corr_empty = b.seg_empty + 2;
  b.tmem_ptr = (uint32_t *)(b.corr_empty + 2);
  b.abort_flag = (volatile int *)(b.tmem_ptr + 1);
  return b;
}
__device__ __forceinline__ uint32_t start_block(const Bars &b, int stages, int tid) {
  if (tid == 0) {
    for (int s = 0; s < stages; s++) {
      mbar_init(b.full + s, kProd + 1);
      mbar_init(b.empty + s, 1);
    }
    for (int i = 0; i < 2; i++) {
      mbar_init(b.seg_full + i, 1);
      mbar_init(b.seg_empty + i, kEpi);
      mbar_init(b.corr_empty + i, kEpi);
    }
    *b.abort_flag = 0;
    fence_barrier_init();
  }
  if ((tid >> 5) == kEpi) {
    tmem_alloc(b.tmem_ptr, 512);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  return *b.tmem_ptr;
}

// The twelve MMAs of one 32-deep step: h*h into `hh`, the five smaller products into `corr`.  Descriptors of part 0; `pa` / `pb` =
// distance between parts, `ka` / `kb` = advance per 16 of depth, all in 16-byte units.
__device__ __forceinline__ void issue_step(uint32_t hh, uint32_t corr, uint64_t a, uint64_t b, uint32_t pa, uint32_t pb, uint32_t ka,
                                           uint32_t kb, uint32_t idesc, bool first_hh, bool first_corr) {
#pragma unroll
  for (int k = 0; k < 2; k++) {
    const uint64_t a0 = a + k * ka, b0 = b + k * kb;
    umma_bf16(hh, a0, b0, idesc, !(first_hh && k == 0));
    umma_bf16(corr, a0, b0 + pb, idesc, !(first_corr && k == 0));  // h * m
    umma_bf16(corr, a0 + pa, b0, idesc, 1);                        // m * h
    umma_bf16(corr, a0 + pa, b0 + pb, idesc, 1);                   // m * m
    umma_bf16(corr, a0, b0 + 2 * pb, idesc, 1);                    // h * l
    umma_bf16(corr, a0 + 2 * pa, b0, idesc, 1);                    // l * h
  }
}

// The small products join.  An operand that is infinite has parts (inf, NaN, NaN): the large products then carry the sum, infinite
// or NaN as in float32 arithmetic, and the small ones are NaN.  fmaxf() makes a number of a NaN, which changes neither an infinity
// nor a NaN, and leaves numbers as they are.  (One instruction per value: a comparison and a selection cost the forward product
// 1.4 %, one test for 16 values its registers.)
__device__ __forceinline__ uint32_t add_small(uint32_t large, uint32_t small) {
  return __float_as_uint(__fadd_rn(__uint_as_float(large), fmaxf(__uint_as_float(small), -FLT_MAX)));
}

// r[j] += t[j], r[j + 1] += t[j + 1]
__device__ __forceinline__ void add_pair(uint32_t (&r)[16], const uint32_t (&t)[16], int j) {
  float a, b;
  unpack2(add2(pack2(__uint_as_float(t[j]), __uint_as_float(t[j + 1])), pack2(__uint_as_float(r[j]), __uint_as_float(r[j + 1]))), a, b);
  r[j] = __float_as_uint(a);
  r[j + 1] = __float_as_uint(b);
}

// One tile's sums in an epilogue warp (lanes 32 * warp ..): every finished segment of large products is added to the running
// sums in tensor memory; with the last one the small products join and the 16-column blocks go to `put(first column, values)`.
// `sg` and `rn` count segments and runs over all tiles; `nc`: buffers of the small products.  False if a wait gave up.
template <class Put>
__device__ __forceinline__ bool drain_tile(const Bars &b, uint32_t lane_addr, int ncols, int nseg, int &sg, int &rn, int nc, int lane,
                                           Put put) {
  const int cb = nc == 2 ? rn & 1 : 0;
  for (int s = 0; s < nseg; s++, sg++) {
    const int buf = sg & 1;
    if (!mbar_wait(b.seg_full + buf, (sg >> 1) & 1, b.abort_flag)) return false;
    tc_fence_after();
    const bool last = s + 1 == nseg;
    for (int c = 0; c < ncols; c += 16) {
      uint32_t r[16], t[16], u[16];
      tmem_ld_32x16(lane_addr + kHh + buf * 128 + c, r);
      if (s > 0) tmem_ld_32x16(lane_addr + kSum + c, t);
      if (last) tmem_ld_32x16(lane_addr + kCorr + cb * 128 + c, u);
      tmem_ld_wait();
      if (s > 0) {
#pragma unroll
        for (int j = 0; j < 16; j += 2) add_pair(r, t, j);
      }
      if (last) {  // (the small products' last one was committed with this segment)
        float v[16];
#pragma unroll
        for (int j = 0; j < 16; j++) v[j] = __uint_as_float(add_small(r[j], u[j]));
        put(c, v);
      } else {
        tmem_st_32x16(lane_addr + kSum + c, r);
      }
    }
    if (!last) tmem_st_wait();
    tc_fence_before();
    __syncwarp();
    if (lane == 0) {
      mbar_arrive(b.seg_empty + buf);
      if (last) mbar_arrive(b.corr_empty + cb);
    }
  }
  rn++;
  return true;
}

// The same for tiles of more than one run: a finished run of small products is added like a segment of large ones, and the sums go
// to `put` after the last buffers were given back.  (A kernel of its own, because the forward product of tiles of one run lost 5 %
// to the registers of this form.)
template <class Put>
__device__ __forceinline__ bool drain_long_tile(const Bars &b, uint32_t lane_addr, int ncols, int nseg, int &sg, int &rn, int lane, Put put) {
  for (int s = 0; s < nseg; s++, sg++) {
    const int buf = sg & 1;
    if (!mbar_wait(b.seg_full + buf, (sg >> 1) & 1, b.abort_flag)) return false;
    tc_fence_after();
    const bool flush = s + 1 == nseg || s % kRun == kRun - 1;  // (the run's last small product was committed with this segment)
    for (int pass = 0; pass < (flush ? 2 : 1); pass++) {
      for (int c = 0; c < ncols; c += 16) {
        uint32_t r[16], t[16];
        tmem_ld_32x16(lane_addr + (pass ? kCorr : kHh + buf * 128) + c, r);
        if (s + pass > 0) tmem_ld_32x16(lane_addr + kSum + c, t);
        tmem_ld_wait();
        if (pass) {
#pragma unroll
          for (int j = 0; j < 16; j++) r[j] = add_small(t[j], r[j]);
        } else if (s > 0) {
#pragma unroll
          for (int j = 0; j < 16; j += 2) add_pair(r, t, j);
        }
        tmem_st_32x16(lane_addr + kSum + c, r);
      }
      tmem_st_wait();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(pass ? b.corr_empty : b.seg_empty + buf);
    }
    if (flush) rn++;
  }
#pragma unroll 1
  for (int c = 0; c < ncols; c += 16) {
    uint32_t r[16];
    tmem_ld_32x16(lane_addr + kSum + c, r);
    tmem_ld_wait();
    float v[16];
#pragma unroll
    for (int j = 0; j < 16; j++) v[j] = __uint_as_float(r[j]);
    put(c, v);
  }
  return true;
}

// The MMA thread's wait for the buffer of a new run of small products; its index in `cb`.
__device__ __forceinline__ bool start_run(const Bars &b, int &rn, int nc, int &cb) {
  cb = nc == 2 ? rn & 1 : 0;
  const int use = nc == 2 ? rn >> 1 : rn;  // this buffer's use count
  rn++;
  return mbar_wait(b.corr_empty + cb, (use & 1) ^ 1, b.abort_flag);
}

struct Gemm3 {
  Src3 g;
  const __nv_bfloat16 *wp;  // weight tile images [nblk][chunk][part][Npb rows][32 columns], 64-byte swizzled
  const float *bias;        // (Nout) or null
  float *out;               // (B, Nout, GH*GW); SRC_SELF: rows (B, GH*GW, Nout), Nout a multiple of 8
  int *status;
  int B, Nout, Npb, nblk, nchunks, tiles_x, tiles_y, stages;
};

__host__ __device__ inline int chunks3(int Cp, int K) { return Cp >= kCols ? Cp / kCols * K : (K * Cp + kCols - 1) / kCols; }
// (slot, first channel) of vector v (8 columns) of a chunk: channel blocks outermost, so that consecutive chunks read the same
// neighbourhood; slots packed into a chunk where a slot has fewer than 32 channels (slot >= K: padding)
__host__ __device__ inline void chunk_item3(int Cp, int K, int chunk, int v, int &slot, int &c0) {
  if (Cp >= kCols) {
    const int cc = chunk / K;
    slot = chunk - cc * K;
    c0 = cc * kCols + v * 8;
  } else {
    const int q = chunk * kCols + v * 8;
    slot = q / Cp;
    c0 = q - slot * Cp;
  }
}

template <int SRC> inline size_t gemm3_smem(int stages, int Npb, int K) {
  return 1024 + (size_t)stages * (3 * kPartA + 3 * Npb * 64) + align_up(TapTable<SRC>::bytes(K), 16) + bars_bytes(stages);
}

// LONG: the small products of a tile take more than one run
template <int SRC, bool LONG>
__global__ void __launch_bounds__(kThreads3, 1) x3_gemm_kernel(const Gemm3 p) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t *base = (uint8_t *)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, S = p.stages;
  const Src3 &g = p.g;
  const uint32_t bbytes = 3u * (uint32_t)p.Npb * 64u, stage_bytes = 3u * kPartA + bbytes;
  const uint32_t stage0 = smem_u32(base);
  const TapTable<SRC> taps(stage0 + S * stage_bytes, g.K);
  const Bars bars = carve_bars(base + (size_t)S * stage_bytes + ((TapTable<SRC>::NT == 1 ? (SRC == SRC_SELF ? 0 : g.K * kPix * 4)
                                                                                     : g.K * kPix * (SRC == SRC_PLAN ? 40 : 32)) + 15) / 16 * 16, S);
  const uint32_t tmem = start_block(bars, S, tid);
  const int tiles_per_image = p.tiles_x * p.tiles_y, total = p.B * tiles_per_image * p.nblk, npix = g.GH * g.GW;
  const int seg = p.nchunks <= kOneSeg ? kOneSeg : kSeg, nseg = (p.nchunks + seg - 1) / seg;
  const int nc = nseg == 1 ? 2 : 1;  // buffers of the small products

  // (The producers of map modes wait after their first tile's taps; in plan mode, a wait inside the tile loop cost its gather 6 %.)
  if (SRC == SRC_PLAN || warp <= kEpi) wait_for_launcher();
  if (warp < kEpi) {
    int sg = 0, rn = 0;
    for (int tile = blockIdx.x; tile < total; tile += gridDim.x) {
      const int nb = tile % p.nblk, rest = tile / p.nblk, b = rest / tiles_per_image, t2 = rest % tiles_per_image;
      const int pix = tile_pixel3(warp * 32 + lane, t2 / p.tiles_x, t2 % p.tiles_x, g.GH, g.GW);
      const int n0 = nb * p.Npb;
      float *out = p.out + ((size_t)b * p.Nout + n0) * npix + pix;
      const auto put = [&](int c, float (&v)[16]) {
        if (pix < 0) return;
        const int left = p.Nout - n0 - c;
        if constexpr (SRC == SRC_SELF) {  // the column buffer of the multiply-first adjoint: this pixel's 16 columns are one 64-byte run
          float *o = p.out + ((size_t)b * npix + pix) * p.Nout + n0 + c;
#pragma unroll
          for (int j = 0; j < 16; j += 8)
            if (j < left)
              asm volatile("st.global.v8.f32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"l"(o + j), "f"(v[j]), "f"(v[j + 1]), "f"(v[j + 2]),
                           "f"(v[j + 3]), "f"(v[j + 4]), "f"(v[j + 5]), "f"(v[j + 6]), "f"(v[j + 7]) : "memory");
          return;
        }
        if (p.bias) {
#pragma unroll
          for (int j = 0; j < 16; j++)
            if (j < left) v[j] += __ldg(p.bias + n0 + c + j);
        }
        float *o = out + (size_t)c * npix;
        if (left >= 16) {
#pragma unroll
          for (int j = 0; j < 16; j++, o += npix) *o = v[j];
        } else {
#pragma unroll
          for (int j = 0; j < 16; j++, o += npix)
            if (j < left) *o = v[j];
        }
      };
      const uint32_t lane_addr = tmem + ((uint32_t)(warp * 32) << 16);
      bool ok;
      if constexpr (LONG) ok = drain_long_tile(bars, lane_addr, p.Npb, nseg, sg, rn, lane, put);
      else ok = drain_tile(bars, lane_addr, p.Npb, nseg, sg, rn, nc, lane, put);
      if (!ok) break;
    }
  } else if (warp == kEpi) {
    if (lane == 0) {
      const uint32_t idesc = idesc_bf16(kPix, p.Npb, 0, 0);
      int sg = 0, rn = 0, cb = 0;
      Ring3 ring;
      bool alive = true;
      for (int tile = blockIdx.x; alive && tile < total; tile += gridDim.x) {
        if (!start_run(bars, rn, nc, cb)) break;
        for (int chunk = 0; chunk < p.nchunks; chunk++, ring.next(S)) {
          const bool first = chunk % seg == 0, first_corr = LONG ? chunk % (kSeg * kRun) == 0 : chunk == 0;
          const int buf = sg & 1;
          if (LONG && first_corr && chunk > 0 && !start_run(bars, rn, nc, cb)) { alive = false; break; }
          if (first && !mbar_wait(bars.seg_empty + buf, ((sg >> 1) & 1) ^ 1, bars.abort_flag)) { alive = false; break; }
          if (!mbar_wait(bars.full + ring.s, ring.ph, bars.abort_flag)) { alive = false; break; }
          tc_fence_after();
          const uint32_t a = stage0 + ring.s * stage_bytes, bw = a + 3 * kPartA;
          issue_step(tmem + kHh + buf * 128, tmem + kCorr + cb * 128, smem_desc_sw64(a), smem_desc_sw64(bw), kPartA >> 4,
                     (uint32_t)p.Npb * 4u, 2, 2, idesc, first, first_corr);
          umma_commit(bars.empty + ring.s);
          if (chunk % seg == seg - 1 || chunk + 1 == p.nchunks) {
            umma_commit(bars.seg_full + buf);
            sg++;
          }
        }
      }
    }
  } else {
    // producers: thread = vector v (8 columns) of pixel px
    const int pt = tid - kProd0, v = pt & 3, px = pt >> 2;
    const uint32_t pitch = (uint32_t)g.Cp * 4u;
    const size_t image = (size_t)(g.SH * g.SW + 1) * pitch;
    const uint32_t dst = stage0 + px * 64 + ((v ^ ((px >> 1) & 3)) << 4);
    PlanView<float> pv{};
    bool plan_ok = true;
    if (SRC == SRC_PLAN) pv = plan_view<float>(g.plan, npix * g.K, plan_ok);
    Ring3 ring;
    bool alive = true;
    for (int tile = blockIdx.x; tile < total; tile += gridDim.x) {
      const int nb = tile % p.nblk, rest = tile / p.nblk, b = rest / tiles_per_image, t2 = rest % tiles_per_image;
      const int ty = t2 / p.tiles_x, tx = t2 % p.tiles_x;
      const char *img = g.xl + (size_t)b * image;
      if constexpr (SRC != SRC_SELF) {
        producer_bar3();  // the previous tile's taps have been read
        fill_taps3<SRC>(g, taps, pv, plan_ok, 0, g.K, ty, tx, pt);
        if (SRC != SRC_PLAN && tile == (int)blockIdx.x) wait_for_launcher();
        producer_bar3();
        if (!alive) continue;
      } else {
        if (!alive) break;
        if (tile == (int)blockIdx.x) wait_for_launcher();
      }
      uint32_t self = 0u;
      if (SRC == SRC_SELF) {
        const int q = tile_pixel3(px, ty, tx, g.GH, g.GW);
        self = (uint32_t)(q >= 0 ? q : g.SH * g.SW) * pitch;
      }
      Item<SRC> it;
      int slot, c0;
      chunk_item3(g.Cp, g.K, 0, v, slot, c0);
      if (slot < g.K) item_load<SRC>(it, taps, img + c0 * 4, slot * kPix + px, self);
      for (int chunk = 0; chunk < p.nchunks; chunk++, ring.next(S)) {
        V8 val;
        if (slot < g.K) {
          val = item_value<SRC>(it, taps, pv, img + c0 * 4, slot * kPix + px, pitch);
        } else {
#pragma unroll
          for (int j = 0; j < 8; j++) val.f[j] = 0.0f;
        }
        if (chunk + 1 < p.nchunks) {  // the next chunk's loads are in flight while this one is split, stored and handed over
          if (g.Cp >= kCols) {        // (chunk_item3 without its division)
            if (++slot == g.K) {
              slot = 0;
              c0 += kCols;
            }
          } else {
            chunk_item3(g.Cp, g.K, chunk + 1, v, slot, c0);
          }
          if (slot < g.K) item_load<SRC>(it, taps, img + c0 * 4, slot * kPix + px, self);
        }
        if (!mbar_wait(bars.empty + ring.s, ring.ph ^ 1u, bars.abort_flag)) { alive = false; break; }
        if (pt == 0) {
          mbar_arrive_expect_tx(bars.full + ring.s, bbytes);
          bulk_copy_g2s(base + (size_t)ring.s * stage_bytes + 3 * kPartA, (const char *)p.wp + ((size_t)nb * p.nchunks + chunk) * bbytes,
                        bbytes, bars.full + ring.s);
        }
        store_parts(dst + ring.s * stage_bytes, kPartA, val);
        fence_proxy_async();
        __syncwarp();
        if (lane == 0) mbar_arrive(bars.full + ring.s);
      }
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == kEpi) tmem_dealloc(tmem, 512);
  if (tid == 0 && *bars.abort_flag) {
    *p.status = 1;
    g_wait_status3 = 1;
  }
}

// ---- weight gradient ---------------------------------------------------------------------------------------------------
// A block owns 128 gradient rows x 128 columns (a column group) and a range of pixel tiles; a tile is four steps of 32 pixels.
// A operand: the gradient's tile image, K-major (64-byte rows); B operand: gathered columns, MN-major (rows of 64 columns of one
// pixel, 128-byte swizzle).  The tap table is double buffered: the next tile's taps are decoded while this one is gathered.
constexpr int kDwN = 128, kDwPix3 = 32;
constexpr int kPartB3 = 2 * kDwPix3 * 128;  // one part of a step's columns: two groups of 64 columns
constexpr int kStepA = 3 * kPartA, kStepB = 3 * kPartB3;

struct Dw3 {
  Src3 g;
  const __nv_bfloat16 *gt;  // gradient tile images [tile][row block][step][part][128 rows][32 pixels]
  float *partial;           // [split][mbs * 128][groups * 128]
  int *status;
  int B, mbs, groups, slots, tiles_x, tiles_y, splits, stages;  // slots: most slots of a column group
};

template <int SRC> inline size_t dw3_smem(int stages, int slots) {
  return 1024 + (size_t)stages * (kStepA + kStepB) + 2 * align_up(TapTable<SRC>::bytes(slots), 16) + bars_bytes(stages);
}

template <int SRC>
__global__ void __launch_bounds__(kThreads3, 1) x3_dw_kernel(const Dw3 p) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t *base = (uint8_t *)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, S = p.stages;
  const Src3 &g = p.g;
  constexpr uint32_t stage_bytes = kStepA + kStepB;
  const uint32_t stage0 = smem_u32(base), table_bytes = (uint32_t)p.slots * kPix * (TapTable<SRC>::NT == 1 ? 4 : 32);
  const Bars bars = carve_bars(base + (size_t)S * stage_bytes + 2 * ((table_bytes + 15) / 16 * 16), S);
  const uint32_t tmem = start_block(bars, S, tid);
  const int grp = blockIdx.x, split = blockIdx.y, mb = blockIdx.z;
  const int tiles_per_image = p.tiles_x * p.tiles_y;
  const int64_t total = (int64_t)p.B * tiles_per_image;
  const int lo = (int)(total * split / p.splits), hi = (int)(total * (split + 1) / p.splits);
  const int nseg = (hi - lo) * 4 / kSeg;

  if (warp <= kEpi) wait_for_launcher();  // (the producers: after their first tile's taps)
  if (warp < kEpi) {
    int sg = 0, rn = 0;
    float *o = p.partial + ((size_t)split * p.mbs * 128 + mb * 128 + warp * 32 + lane) * (p.groups * kDwN) + grp * kDwN;
    const auto put = [&](int c, const float (&v)[16]) {
#pragma unroll
      for (int j = 0; j < 16; j += 4) *(float4 *)(o + c + j) = make_float4(v[j], v[j + 1], v[j + 2], v[j + 3]);
    };
    drain_long_tile(bars, tmem + ((uint32_t)(warp * 32) << 16), kDwN, nseg, sg, rn, lane, put);
  } else if (warp == kEpi) {
    if (lane == 0) {
      const uint32_t idesc = idesc_bf16(128, kDwN, 0, 1);
      Ring3 ring;
      const int steps = (hi - lo) * 4;
      int rn = 0, cb = 0;
      for (int st = 0; st < steps; st++, ring.next(S)) {
        const int sg = st / kSeg, buf = sg & 1;
        const bool first = st % kSeg == 0, first_corr = st % (kSeg * kRun) == 0;
        if (first_corr && !start_run(bars, rn, 1, cb)) break;
        if (first && !mbar_wait(bars.seg_empty + buf, ((sg >> 1) & 1) ^ 1, bars.abort_flag)) break;
        if (!mbar_wait(bars.full + ring.s, ring.ph, bars.abort_flag)) break;
        tc_fence_after();
        const uint32_t a = stage0 + ring.s * stage_bytes;
        issue_step(tmem + kHh + buf * 128, tmem + kCorr, smem_desc_sw64(a), smem_desc_sw128(a + kStepA, kDwPix3 * 128, 1024), kPartA >> 4,
                   kPartB3 >> 4, 2, 16 * 128 >> 4, idesc, first, first_corr);
        umma_commit(bars.empty + ring.s);
        if (st % kSeg == kSeg - 1) umma_commit(bars.seg_full + buf);
      }
    }
  } else {
    // producers: thread = vector v (8 of the group's 128 columns) of pixel px of the step
    const int pt = tid - kProd0, v = pt & 15, px = pt >> 4;
    const uint32_t pitch = (uint32_t)g.Cp * 4u;
    const size_t image = (size_t)(g.SH * g.SW + 1) * pitch;
    const int s0 = grp * kDwN / g.Cp, col = grp * kDwN + v * 8, slot = col / g.Cp, c0 = col - slot * g.Cp;
    const bool have = slot < g.K;
    const int row0 = have ? (slot - s0) * kPix + px : 0;
    const uint32_t dst = stage0 + kStepA + (v >> 3) * (kDwPix3 * 128) + px * 128 + (((v & 7) ^ (px & 7)) << 4);
    const uint32_t table0 = stage0 + S * stage_bytes, table_pitch = (table_bytes + 15) / 16 * 16;
    const PlanView<float> none{};
    const auto fill = [&](int t2, int buf) {
      fill_taps3<SRC>(g, TapTable<SRC>(table0 + buf * table_pitch, p.slots), none, true, s0, p.slots, t2 / p.tiles_x, t2 % p.tiles_x, pt);
    };
    int image_of = lo / tiles_per_image, t2 = lo - image_of * tiles_per_image;  // image and tile of `tile`
    if (lo < hi) fill(t2, 0);
    wait_for_launcher();
    Ring3 ring;
    bool alive = true;
    for (int tile = lo; tile < hi; tile++) {
      const TapTable<SRC> taps(table0 + ((tile - lo) & 1) * table_pitch, p.slots);
      const char *img = g.xl + (size_t)image_of * image + c0 * 4;
      if (++t2 == tiles_per_image) {
        t2 = 0;
        image_of++;
      }
      producer_bar3();  // this tile's table is complete, the other one no longer read
      Item<SRC> it;
      if (alive && have) item_load<SRC>(it, taps, img, row0, 0u);
      if (tile + 1 < hi) fill(t2, (tile + 1 - lo) & 1);
      for (int q = 0; alive && q < 4; q++, ring.next(S)) {
        V8 val;
        if (have) {
          val = item_value<SRC>(it, taps, none, img, 0, pitch);
        } else {
#pragma unroll
          for (int j = 0; j < 8; j++) val.f[j] = 0.0f;
        }
        if (q < 3 && have) item_load<SRC>(it, taps, img, row0 + (q + 1) * kDwPix3, 0u);
        if (!mbar_wait(bars.empty + ring.s, ring.ph ^ 1u, bars.abort_flag)) { alive = false; break; }
        if (pt == 0) {
          mbar_arrive_expect_tx(bars.full + ring.s, kStepA);
          bulk_copy_g2s(base + (size_t)ring.s * stage_bytes, (const char *)p.gt + (((size_t)tile * p.mbs + mb) * 4 + q) * kStepA, kStepA,
                        bars.full + ring.s);
        }
        store_parts(dst + ring.s * stage_bytes, kPartB3, val);
        fence_proxy_async();
        __syncwarp();
        if (lane == 0) mbar_arrive(bars.full + ring.s);
      }
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == kEpi) tmem_dealloc(tmem, 512);
  if (tid == 0 && *bars.abort_flag) {
    *p.status = 1;
    g_wait_status3 = 1;
  }
}

// A NaN whose payload lies in the lower half alone would have an infinity for its upper part: NaNs become the canonical one.
__device__ __forceinline__ float quiet(float x) { return x != x ? __int_as_float(0x7fffffff) : x; }

// ---- layout pre-passes ---------------------------------------------------------------------------------------------------
// (B, C, HW) -> (B, HW + 1, Cp) float32; padding channels and the extra pixel are zero.  128 pixels x 32 channels per block,
// through shared memory (blocks of 32 x 32 spent half their instructions on finding their place: 41 -> 27 us per 67 MB).  With
// `sums` every block also leaves its channels' sums over its pixels, sums[(b * px_blocks + block) * Cp + c]: the bias gradient
// where the gathered side is the output's gradient.
constexpr int kNhwcPix = 128;
struct Nhwc3 {
  const float *x;
  float *y, *sums;
  int C, Cp, HW, px_blocks, ch_blocks, blocks;
};
using NhwcTile = float[32][kNhwcPix + 1];
__device__ __forceinline__ void nhwc_block(const Nhwc3 &q, int block, NhwcTile &tile) {
  const int bp = block % q.px_blocks, bc = block / q.px_blocks % q.ch_blocks, b = block / (q.px_blocks * q.ch_blocks);
  const int c0 = bc * 32, p0 = bp * kNhwcPix, tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
#pragma unroll
  for (int i = 0; i < 4; i++) {
    const int c = c0 + ty + 8 * i;
    const float *x = q.x + ((size_t)b * q.C + c) * q.HW + p0 + tx;
    float v[4];
#pragma unroll
    for (int j = 0; j < 4; j++) v[j] = c < q.C && p0 + tx + 32 * j < q.HW ? __ldg(x + 32 * j) : 0.0f;
#pragma unroll
    for (int j = 0; j < 4; j++) tile[ty + 8 * i][tx + 32 * j] = v[j];
    if (q.sums) {
      float s = (v[0] + v[1]) + (v[2] + v[3]);
#pragma unroll
      for (int d = 16; d > 0; d >>= 1) s += __shfl_xor_sync(0xffffffffu, s, d);
      if (tx == 0 && c < q.Cp) q.sums[((size_t)b * q.px_blocks + bp) * q.Cp + c] = s;
    }
  }
  __syncthreads();
  const int c = c0 + tx, np = min(kNhwcPix, q.HW + 1 - p0);
  if (c >= q.Cp) return;
  float *y = q.y + ((size_t)b * (q.HW + 1) + p0) * q.Cp + c;
#pragma unroll 4
  for (int i = ty; i < np; i += 8) y[(size_t)i * q.Cp] = quiet(tile[tx][i]);
}

__device__ __forceinline__ void split3(float x, uint16_t &h, uint16_t &m, uint16_t &l) {
  x = quiet(x);
  const float r = x - __uint_as_float(__float_as_uint(x) & 0xffff0000u), s = r - __uint_as_float(__float_as_uint(r) & 0xffff0000u);
  h = (uint16_t)(__float_as_uint(x) >> 16);
  m = (uint16_t)(__float_as_uint(r) >> 16);
  l = (uint16_t)(__float_as_uint(s) >> 16);
}

// Weights -> three-part tile images.  Rows n = nb * Npb + row; `premul`: rows are n = k * premul + m of the multiply-first adjoint
// (columns: source channels), else rows are output channels and columns (slot, channel) items.  W[m * sm + ch * sc + k * sk].
struct Weight3 {
  const float *w;
  uint16_t *wp;
  int M, CH, Cp, K, Npb, nblk, nchunks, premul, blocks;  // premul: padded M, or 0
  int64_t sm, sc, sk;
};
__device__ __forceinline__ void weight_block(const Weight3 &q, int block) {
  const int i = block * 256 + threadIdx.x;
  if (i >= q.nblk * q.nchunks * q.Npb * kCols) return;
  const int col = i % kCols, r = i / kCols % q.Npb, chunk = i / (kCols * q.Npb) % q.nchunks, nb = i / (kCols * q.Npb * q.nchunks);
  const int n = nb * q.Npb + r;
  float v = 0.0f;
  if (q.premul) {
    const int k = n / q.premul, m = n - k * q.premul, ch = chunk * kCols + col;
    if (k < q.K && m < q.M && ch < q.CH) v = __ldg(q.w + m * q.sm + ch * q.sc + k * q.sk);
  } else {
    int slot, c0;
    chunk_item3(q.Cp, q.K, chunk, col >> 3, slot, c0);
    const int ch = c0 + (col & 7);
    if (n < q.M && slot < q.K && ch < q.CH) v = __ldg(q.w + n * q.sm + ch * q.sc + slot * q.sk);
  }
  uint16_t h, m, l;
  split3(v, h, m, l);
  uint16_t *t = q.wp + ((int64_t)nb * q.nchunks + chunk) * 3 * q.Npb * kCols + r * kCols + ((((col >> 3) ^ ((r >> 1) & 3)) << 3) | (col & 7));
  t[0] = h;
  t[(int64_t)q.Npb * kCols] = m;
  t[(int64_t)2 * q.Npb * kCols] = l;
}

// The pre-pass of x3_gemm in one launch: source, weights, the call's status word.
__global__ void __launch_bounds__(256) gemm_prepare3_kernel(const Nhwc3 src, const Weight3 wgt, int *status) {
  __shared__ NhwcTile tile;
  launch_dependents();
  if (blockIdx.x == 0 && threadIdx.x == 0) *status = 0;
  if ((int)blockIdx.x < wgt.blocks) weight_block(wgt, blockIdx.x);
  else nhwc_block(src, blockIdx.x - wgt.blocks, tile);
}

// Gradient (B, N, GH*GW) -> tile images [tile][row block][step][part][128 rows][32 pixels] and, with `sums`, the sum of every
// row over the tile's pixels: sums[(tile * mbs + row block) * 128 + row].  One block = one tile and row block.
struct Grad3 {
  const float *g;
  uint8_t *gt;
  float *sums;
  int N, GH, GW, tiles_x, tiles_y, mbs, blocks;
};
__device__ __forceinline__ void grad_block(const Grad3 &q, int block) {
  const int N = q.N, GH = q.GH, GW = q.GW, tiles_x = q.tiles_x, tiles_y = q.tiles_y, mbs = q.mbs;
  const int mb = block % mbs, t2 = block / mbs % (tiles_x * tiles_y), b = block / (mbs * tiles_x * tiles_y);
  const int ty = t2 / tiles_x, tx = t2 % tiles_x;
  const float *gsrc = q.g;
  uint8_t *gt = q.gt;
  float *sums = q.sums;
  const size_t npix = (size_t)GH * GW, tile = (size_t)b * tiles_x * tiles_y + t2;
  uint8_t *dst = gt + (tile * mbs + mb) * 4 * kStepA;
  const bool vec = (GW & 3) == 0 && (((uintptr_t)gsrc) & 15) == 0;
  for (int i = threadIdx.x; i < 128 * 16; i += 256) {
    const int r = i >> 4, u = i & 15, n = mb * 128 + r;  // u: 8 pixels of the tile, row u >> 1, columns (u & 1) * 8 ..
    const int y = ty * kTileH + (u >> 1), x0 = tx * kTileW + (u & 1) * 8;
    const float *src = gsrc + ((size_t)b * N + n) * npix + (size_t)y * GW + x0;
    V8 v;
    if (n < N && y < GH && x0 + 8 <= GW && vec) {
      const float4 a = __ldg((const float4 *)src), c = __ldg((const float4 *)src + 1);
      v.f[0] = a.x; v.f[1] = a.y; v.f[2] = a.z; v.f[3] = a.w;
      v.f[4] = c.x; v.f[5] = c.y; v.f[6] = c.z; v.f[7] = c.w;
    } else {
#pragma unroll
      for (int e = 0; e < 8; e++) v.f[e] = n < N && y < GH && x0 + e < GW ? __ldg(src + e) : 0.0f;
    }
    uint16_t h[8], m[8], l[8];
#pragma unroll
    for (int e = 0; e < 8; e++) split3(v.f[e], h[e], m[e], l[e]);
    const auto pack = [](const uint16_t (&q)[8]) {
      return make_uint4(q[0] | (uint32_t)q[1] << 16, q[2] | (uint32_t)q[3] << 16, q[4] | (uint32_t)q[5] << 16, q[6] | (uint32_t)q[7] << 16);
    };
    uint8_t *d = dst + (size_t)(u >> 2) * kStepA + r * 64 + (((u & 3) ^ ((r >> 1) & 3)) << 4);
    *(uint4 *)d = pack(h);
    *(uint4 *)(d + kPartA) = pack(m);
    *(uint4 *)(d + 2 * kPartA) = pack(l);
    if (sums) {
      float s = ((v.f[0] + v.f[1]) + (v.f[2] + v.f[3])) + ((v.f[4] + v.f[5]) + (v.f[6] + v.f[7]));
#pragma unroll
      for (int d2 = 1; d2 < 16; d2 <<= 1) s += __shfl_xor_sync(0xffffffffu, s, d2);
      if (u == 0) sums[(tile * mbs + mb) * 128 + r] = s;
    }
  }
}

// The pre-pass of x3_dw in one launch: gathered side, gradient tile images, the call's status word.
__global__ void __launch_bounds__(256) dw_prepare3_kernel(const Nhwc3 src, const Grad3 grad, int *status) {
  __shared__ NhwcTile tile;
  launch_dependents();
  if (blockIdx.x == 0 && threadIdx.x == 0) *status = 0;
  if ((int)blockIdx.x < grad.blocks) grad_block(grad, blockIdx.x);
  else nhwc_block(src, blockIdx.x - grad.blocks, tile);
}

// The pre-pass of both in one launch (x3_backward): two gathered sides, the second one empty where both products gather from the same.
// A convolution's products share the output's gradient, one as the gathered side, the other as tile images: their blocks take turns, in
// proportion, so that the second read comes from L2 (8 x 128 planes of 128 x 256: 119 us one after the other, so 102; a transposed
// convolution, which makes its images of another tensor, 41 and 45).
__global__ void __launch_bounds__(256) backward_prepare3_kernel(const Nhwc3 src, const Nhwc3 src2, const Weight3 wgt, const Grad3 grad,
                                                                int *status, int *status2) {
  __shared__ NhwcTile tile;
  launch_dependents();
  if (blockIdx.x == 0 && threadIdx.x == 0) *status = *status2 = 0;
  const int both = grad.blocks + src.blocks;
  int block = blockIdx.x;
  if (block < both) {
    int s = max(block - grad.blocks, 0), next = max(block + 1 - grad.blocks, 0);  // blocks of `src` before this one and the next
    if (src.x == grad.g) {
      s = (int)((int64_t)block * src.blocks / both);
      next = (int)((int64_t)(block + 1) * src.blocks / both);
    }
    if (next > s) nhwc_block(src, s, tile);
    else grad_block(grad, block - s);
    return;
  }
  if ((block -= both) < wgt.blocks) return weight_block(wgt, block);
  nhwc_block(src2, block - wgt.blocks, tile);
}

// The post-pass of x3_dw in one launch: gw[m, ch, k] = sum over splits, in order, of the partial sums (256 values per block, columns
// fastest), and gb[c] = sum over `parts` of sums[part * pitch + c], one block per channel, in a fixed order.
struct Reduce3 {
  const float *partial, *sums;
  float *gw, *gb;
  int splits, rows, cols, M, CH, Cp, K, blocks, parts, pitch;
  int64_t sm, sc, sk;
};
__global__ void __launch_bounds__(256) dw_reduce3_kernel(const Reduce3 q) {
  __shared__ float red[256];
  if ((int)blockIdx.x < q.blocks) {
    const int i = blockIdx.x * 256 + threadIdx.x;
    if (i >= q.M * q.CH * q.K) return;
    const int ch = i % q.CH, k = (i / q.CH) % q.K, m = i / (q.CH * q.K);
    const float *s = q.partial + (size_t)m * q.cols + k * q.Cp + ch;
    const size_t step = (size_t)q.rows * q.cols;
    float a = 0.0f;
    int z = 0;
    for (; z + 4 <= q.splits; z += 4) {  // (four loads in flight, added in order)
      const float v0 = __ldg(s + z * step), v1 = __ldg(s + (z + 1) * step), v2 = __ldg(s + (z + 2) * step), v3 = __ldg(s + (z + 3) * step);
      a = (((a + v0) + v1) + v2) + v3;
    }
    for (; z < q.splits; z++) a += __ldg(s + z * step);
    q.gw[m * q.sm + ch * q.sc + k * q.sk] = a;
    return;
  }
  const int c = blockIdx.x - q.blocks;
  float s = 0.0f;
  for (int t = threadIdx.x; t < q.parts; t += 256) s += __ldg(q.sums + (size_t)t * q.pitch + c);
  red[threadIdx.x] = s;
  __syncthreads();
  for (int d = 128; d > 0; d >>= 1) {
    if (threadIdx.x < d) red[threadIdx.x] += red[threadIdx.x + d];
    __syncthreads();
  }
  if (threadIdx.x == 0) q.gb[c] = red[0];
}

// Second half of the multiply-first adjoint: out[b][m][q] (+bias) = sum over the plan entries (p, k, w) of destination pixel q, in
// plan order, of w * T[b][p][k * Mp + m].  L neighbouring threads share a destination pixel; each adds NV vectors of eight channels,
// L apart, so that an instruction reads whole lines of a row.  The next entry's index and weight are on their way with this
// one's row.  (Transposed 128 -> 64 channels, 8 x 128 x 256: one thread per pixel and 16 channels 92 us; so 69 us.)
template <int NV, int L>
__global__ void __launch_bounds__(256) plan_gather_rows3_kernel(const float *__restrict__ T, const void *__restrict__ plan_blob,
                                                                const float *__restrict__ bias, float *__restrict__ out, int K, int M, int Mp,
                                                                int n_src, int n_dst) {
  const int q = blockIdx.x * (256 / L) + threadIdx.x / L, m0 = (blockIdx.y * NV * L + threadIdx.x % L) * 8, b = blockIdx.z;
  if (q >= n_dst || m0 >= Mp) return;
  bool ok;
  const PlanView<float> pv = plan_view<float>(plan_blob, n_dst * K, ok);
  const uint32_t pitch = (uint32_t)(K * Mp) * 4u;
  const char *rows = (const char *)(T + (size_t)b * n_src * (K * Mp) + m0);
  V8 acc[NV];
#pragma unroll
  for (int i = 0; i < NV; i++)
#pragma unroll
    for (int j = 0; j < 8; j++) acc[i].f[j] = 0.0f;
  if (ok) {
    const int *off = pv.offsets + (size_t)q * K;
    int e = __ldg(off), e1 = __ldg(off + 1);
    const int end = __ldg(off + K);
    int s = 0;
    float w = 0.0f;
    if (e < end) {
      s = __ldg(pv.src + e);
      w = __ldg(pv.w + e);
    }
    while (e < end) {
      while (e >= e1) {
        off++;
        e1 = __ldg(off + 1);
        rows += Mp * 4;
      }
      const bool in = index_ok(s, n_src);
      const float we = in ? w : 0.0f;
      const char *row = rows + (size_t)(unsigned)(in ? s : 0) * pitch;
      V8 v[NV];
#pragma unroll
      for (int i = 0; i < NV; i++)
        if (i == 0 || m0 + i * L * 8 < Mp) v[i] = load8(row + i * L * 32);
      if (++e < end) {
        s = __ldg(pv.src + e);
        w = __ldg(pv.w + e);
      }
#pragma unroll
      for (int i = 0; i < NV; i++)
        if (i == 0 || m0 + i * L * 8 < Mp)
#pragma unroll
          for (int j = 0; j < 8; j++) acc[i].f[j] = fmaf(we, v[i].f[j], acc[i].f[j]);
    }
  }
#pragma unroll
  for (int i = 0; i < NV; i++)
#pragma unroll
    for (int j = 0; j < 8; j++) {
      const int m = m0 + i * L * 8 + j;
      if (m < M) out[((size_t)b * M + m) * n_dst + q] = acc[i].f[j] + (bias ? __ldg(bias + m) : 0.0f);
    }
}

// ---- host side -------------------------------------------------------------------------------------------------------------
constexpr int kMaxDev3 = 64;
int device3() {
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kMaxDev3) dev = 0;
  return dev;
}
int sms3() {
  static int n[kMaxDev3];
  const int dev = device3();
  int v = __atomic_load_n(&n[dev], __ATOMIC_RELAXED);
  if (v == 0) {
    if (cudaDeviceGetAttribute(&v, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || v <= 0) v = 148;
    __atomic_store_n(&n[dev], v, __ATOMIC_RELAXED);
  }
  return v;
}
template <typename Kernel> void allow_smem3(Kernel kernel, int *granted, size_t smem) {
  const int dev = device3();
  if (__atomic_load_n(&granted[dev], __ATOMIC_RELAXED) >= (int)smem) return;
  cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  __atomic_store_n(&granted[dev], (int)smem, __ATOMIC_RELAXED);
}

// Source kind of a gather, or -1 where the kernels here do not cover it (more than four taps per slot).
int source3(bool use_plan, int64_t P, int interp) {
  if (use_plan) return SRC_PLAN;
  if (P == 0) return interp == SPH_NEAREST ? SRC_MAP1 : SRC_MAP4;
  return P <= 4 && interp == SPH_NEAREST ? SRC_MAP4 : -1;
}
size_t table3(int src, int ns) {
  return src == SRC_SELF ? 0 : (size_t)ns * kPix * (src == SRC_MAP1 ? 4 : src == SRC_PLAN ? 40 : 32);
}
// Three stages where they leave the L1 about 70 KB, else two (64 -> 128 channels, 8 x 128 x 256: bilinear forward 348 us with two
// stages of 48 KB and 36 KB of taps, 355 with three; its input gradient, 36 KB stages, 681 with two, 662 with three).  The
// weight gradient, whose tap tables are small, takes three (350 -> 310 us).
constexpr size_t kSmemSoft = 160 * 1024;

struct GemmPlan3 {
  int Cp, nchunks, Npb, nblk, stages;
  size_t xl_bytes, wp_bytes, smem;
  bool ok;
};
GemmPlan3 gemm_plan3(int src, int64_t B, int64_t CH, int64_t SHW, int64_t K, int64_t Nout) {
  GemmPlan3 q{};
  q.Cp = padded3(CH);
  q.nchunks = chunks3(q.Cp, (int)K);
  const int np = (int)align_up((size_t)Nout, 16);
  q.nblk = (np + kNMax - 1) / kNMax;
  q.Npb = (int)align_up((size_t)((np + q.nblk - 1) / q.nblk), 16);  // blocks of equal width
  q.xl_bytes = align_up((size_t)(B * (SHW + 1)) * q.Cp * 4, 256);
  q.wp_bytes = align_up((size_t)q.nblk * q.nchunks * 3 * q.Npb * kCols * 2, 256);
  const auto smem = [&](int s) { return 1024 + (size_t)s * (3 * kPartA + 3 * q.Npb * 64) + align_up(table3(src, (int)K), 16) + bars_bytes(s); };
  q.stages = smem(3) <= kSmemSoft ? 3 : 2;
  q.smem = smem(q.stages);
  q.ok = src >= 0 && q.smem <= kSmemMax && (SHW + 1) * q.Cp * 4 < ((int64_t)1 << 32) &&
         (int64_t)q.nblk * q.nchunks * q.Npb * kCols < ((int64_t)1 << 31);
  return q;
}

// Multiply first (conv_simt.cu says when and why): a dense product over the source grid with N = K * M rows.
struct Premul3 {
  GemmPlan3 q;
  int Mp;  // output channels padded to 8: a thread of the plan gather reads 8 (or 16) of a row at once
  size_t t_bytes;
  bool use;
};
Premul3 premul3(int64_t B, int64_t CH, int64_t SHW, int64_t K, int64_t M, int64_t n_dst) {
  Premul3 r{};
  r.Mp = (int)align_up((size_t)M, 8);
  r.q = gemm_plan3(SRC_SELF, B, CH, SHW, 1, K * r.Mp);
  r.t_bytes = align_up((size_t)(B * K * r.Mp * SHW) * 4, 256);
  r.use = r.q.ok && n_dst >= 3 * SHW && CH >= 16 && r.t_bytes <= ((size_t)8 << 30);
  return r;
}

struct DwPlan3 {
  int Cp, groups, mbs, slots, splits, stages, tiles_x, tiles_y;
  size_t xl_bytes, gt_bytes, partial_bytes, sums_bytes, smem;
  bool ok;
};
DwPlan3 dw_plan3(int src, int64_t B, int64_t CH, int64_t SHW, int64_t K, int64_t M, int64_t GH, int64_t GW) {
  DwPlan3 d{};
  d.Cp = padded3(CH);
  d.groups = (int)((K * d.Cp + kDwN - 1) / kDwN);
  d.mbs = (int)((M + 127) / 128);
  // (the position of a group's first column within its slot repeats after at most Cp / 32 groups)
  for (int g = 0; g < d.groups && g < std::max(d.Cp / 32, 1); g++)
    d.slots = std::max(d.slots, (g * kDwN + kDwN - 1) / d.Cp - g * kDwN / d.Cp + 1);
  d.tiles_x = cdiv(GW, kTileW);
  d.tiles_y = cdiv(GH, kTileH);
  const int64_t tiles = B * d.tiles_x * d.tiles_y;
  int64_t s = sms3() / ((int64_t)d.groups * d.mbs);
  d.splits = (int)(s < 1 ? 1 : s > tiles ? tiles : s);
  const auto dw_smem = [&](int s) { return 1024 + (size_t)s * (kStepA + kStepB) + 2 * align_up(table3(src, d.slots), 16) + bars_bytes(s); };
  d.stages = dw_smem(3) <= kSmemMax ? 3 : 2;
  d.smem = dw_smem(d.stages);
  d.xl_bytes = align_up((size_t)(B * (SHW + 1)) * d.Cp * 4, 256);
  d.gt_bytes = align_up((size_t)tiles * d.mbs * 4 * kStepA, 256);
  d.partial_bytes = align_up((size_t)d.splits * d.mbs * 128 * d.groups * kDwN * 4, 256);
  // (row sums of the gradient's tiles, or channel sums of the gathered side's blocks)
  d.sums_bytes = align_up((size_t)std::max<int64_t>(tiles * d.mbs * 128, B * cdiv(SHW + 1, kNhwcPix) * d.Cp) * 4, 256);
  d.ok = src >= 0 && src != SRC_PLAN && d.smem <= kSmemMax && (SHW + 1) * d.Cp * 4 < ((int64_t)1 << 32) && tiles < ((int64_t)1 << 28);
  return d;
}

Nhwc3 nhwc3(const void *x, float *y, int64_t B, int64_t C, int Cp, int64_t HW, float *sums = nullptr) {
  Nhwc3 q{(const float *)x, y, sums, (int)C, Cp, (int)HW, cdiv(HW + 1, kNhwcPix), cdiv(Cp, 32), 0};
  q.blocks = q.px_blocks * q.ch_blocks * (int)B;
  return q;
}

template <int SRC, bool LONG> void launch_gemm3_as(const Gemm3 &p, int64_t tiles, size_t smem, cudaStream_t st) {
  static int granted[kMaxDev3];
  allow_smem3(x3_gemm_kernel<SRC, LONG>, granted, smem);
  launch_after(x3_gemm_kernel<SRC, LONG>, dim3((unsigned)std::min<int64_t>(tiles, sms3())), kThreads3, smem, st, p);
}
template <int SRC> void launch_gemm3(const Gemm3 &p, int64_t tiles, size_t smem, cudaStream_t st) {
  if (p.nchunks > kSeg * kRun) launch_gemm3_as<SRC, true>(p, tiles, smem, st);
  else launch_gemm3_as<SRC, false>(p, tiles, smem, st);
}
template <int SRC> void launch_dw3(const Dw3 &p, size_t smem, cudaStream_t st) {
  static int granted[kMaxDev3];
  allow_smem3(x3_dw_kernel<SRC>, granted, smem);
  launch_after(x3_dw_kernel<SRC>, dim3(p.groups, p.splits, p.mbs), kThreads3, smem, st, p);
}

}  // namespace

// Scratch of x3_gemm; 0: not covered.
size_t x3_gemm_workspace(bool use_plan, int64_t B, int64_t CH, int64_t SHW, int64_t K, int64_t P, int interp, int64_t Nout, int64_t n_dst) {
  if (use_plan) {
    const Premul3 r = premul3(B, CH, SHW, K, Nout, n_dst);
    if (r.use) return 256 + r.q.xl_bytes + r.q.wp_bytes + r.t_bytes;
  }
  const GemmPlan3 q = gemm_plan3(source3(use_plan, P, interp), B, CH, SHW, K, Nout);
  return q.ok ? 256 + q.xl_bytes + q.wp_bytes : 0;
}

namespace {

// What x3_gemm launches: the pre-pass's operands, the product, the row gather of the multiply-first form.
struct GemmCall3 {
  Premul3 r;
  GemmPlan3 q;
  int kind;
  Nhwc3 pre;
  Weight3 wt;
  Gemm3 p;
  const void *plan, *bias;
  void *out;
  int64_t Nout, K, B, n_src, n_dst;
};
GemmCall3 gemm_call3(bool use_plan, const void *src, const void *map, const void *iw, const void *plan, int64_t CH, int64_t SH, int64_t SW,
                     int64_t K, int64_t P, int64_t GH, int64_t GW, int interp, const void *wgt, int64_t sm, int64_t sc, int64_t sk,
                     const void *bias, void *out, int64_t Nout, int64_t B, void *ws) {
  GemmCall3 c{};
  c.r = use_plan ? premul3(B, CH, SH * SW, K, Nout, GH * GW) : Premul3{};
  c.kind = c.r.use ? (int)SRC_SELF : source3(use_plan, P, interp);
  c.q = c.r.use ? c.r.q : gemm_plan3(c.kind, B, CH, SH * SW, K, Nout);
  const Premul3 &r = c.r;
  const GemmPlan3 &q = c.q;
  char *w = (char *)ws;
  float *xl = (float *)(w + 256);
  uint16_t *wp = (uint16_t *)(w + 256 + q.xl_bytes);
  float *T = (float *)(w + 256 + q.xl_bytes + q.wp_bytes);
  c.pre = nhwc3(src, xl, B, CH, q.Cp, SH * SW);
  c.wt = Weight3{(const float *)wgt, wp, (int)Nout, (int)CH, q.Cp, (int)K, q.Npb, q.nblk, q.nchunks, r.use ? r.Mp : 0,
                 cdiv((int64_t)q.nblk * q.nchunks * q.Npb * kCols, 256), sm, sc, sk};
  Gemm3 &p = c.p;
  p.g = Src3{(const char *)xl, (const float *)map, (const float *)iw, plan, q.Cp, (int)SH, (int)SW, r.use ? 1 : (int)K, (int)P,
             (int)(r.use ? SH : GH), (int)(r.use ? SW : GW), interp};
  p.wp = (const __nv_bfloat16 *)wp;
  p.bias = r.use ? nullptr : (const float *)bias;
  p.out = r.use ? T : (float *)out;
  p.status = (int *)w;
  p.B = (int)B; p.Nout = (int)(r.use ? K * r.Mp : Nout); p.Npb = q.Npb; p.nblk = q.nblk; p.nchunks = q.nchunks;
  p.tiles_x = cdiv(p.g.GW, kTileW); p.tiles_y = cdiv(p.g.GH, kTileH); p.stages = q.stages;
  c.plan = plan; c.bias = bias; c.out = out;
  c.Nout = Nout; c.K = K; c.B = B; c.n_src = SH * SW; c.n_dst = GH * GW;
  return c;
}
// The product; `prepared`: launches of the pre-pass.
int run_gemm3(const GemmCall3 &c, int prepared, cudaStream_t st) {
  const int64_t tiles = c.B * c.p.tiles_x * c.p.tiles_y * c.q.nblk;
  switch (c.kind) {
    case SRC_MAP1: launch_gemm3<SRC_MAP1>(c.p, tiles, c.q.smem, st); break;
    case SRC_MAP4: launch_gemm3<SRC_MAP4>(c.p, tiles, c.q.smem, st); break;
    case SRC_PLAN: launch_gemm3<SRC_PLAN>(c.p, tiles, c.q.smem, st); break;
    default: launch_gemm3<SRC_SELF>(c.p, tiles, c.q.smem, st); break;
  }
  const int rc = launch_status(1 + prepared);
  if (rc != SPH_OK || !c.r.use) return rc;
  const int vecs = c.r.Mp / 8, lanes = vecs >= 4 ? 4 : vecs >= 2 ? 2 : 1, nv = vecs > 4 ? 2 : 1;
  const dim3 grid(cdiv(c.n_dst, 256 / lanes), cdiv(vecs, nv * lanes), (unsigned)c.B);
  const auto rows = nv == 2 ? plan_gather_rows3_kernel<2, 4>
                            : (lanes == 4 ? plan_gather_rows3_kernel<1, 4> : lanes == 2 ? plan_gather_rows3_kernel<1, 2> : plan_gather_rows3_kernel<1, 1>);
  rows<<<grid, 256, 0, st>>>(c.p.out, c.plan, (const float *)c.bias, (float *)c.out, (int)c.K, (int)c.Nout, c.r.Mp, (int)c.n_src, (int)c.n_dst);
  return launch_status();
}

}  // namespace

int x3_gemm(bool use_plan, const void *src, const void *map, const void *iw, const void *plan, int64_t CH, int64_t SH, int64_t SW, int64_t K,
            int64_t P, int64_t GH, int64_t GW, int interp, const void *wgt, int64_t sm, int64_t sc, int64_t sk, const void *bias, void *out,
            int64_t Nout, int64_t B, void *ws, cudaStream_t st) {
  const GemmCall3 c = gemm_call3(use_plan, src, map, iw, plan, CH, SH, SW, K, P, GH, GW, interp, wgt, sm, sc, sk, bias, out, Nout, B, ws);
  gemm_prepare3_kernel<<<(unsigned)(c.wt.blocks + c.pre.blocks), 256, 0, st>>>(c.pre, c.wt, c.p.status);
  return run_gemm3(c, 1, st);
}

size_t x3_dw_workspace(int64_t B, int64_t CH, int64_t SHW, int64_t K, int64_t P, int interp, int64_t M, int64_t GH, int64_t GW) {
  const DwPlan3 d = dw_plan3(source3(false, P, interp), B, CH, SHW, K, M, GH, GW);
  return d.ok ? 256 + d.xl_bytes + d.gt_bytes + d.partial_bytes + d.sums_bytes : 0;
}

namespace {

// What x3_dw launches.  `copy`: the gathered side's channels-last copy, if another product's pre-pass makes it.
struct DwCall3 {
  DwPlan3 d;
  int kind;
  Nhwc3 pre;
  Grad3 grad;
  Dw3 p;
  Reduce3 red;
  int channels;  // of the bias gradient
};
DwCall3 dw_call3(const void *A, const void *src, const void *map, const void *iw, int64_t CH, int64_t SH, int64_t SW, int64_t K, int64_t P,
                 int64_t GH, int64_t GW, int interp, int64_t M, int64_t B, void *gw, int64_t sm, int64_t sc, int64_t sk, void *gb,
                 bool bias_of_src, void *ws, const char *copy = nullptr) {
  DwCall3 c{};
  c.kind = source3(false, P, interp);
  c.d = dw_plan3(c.kind, B, CH, SH * SW, K, M, GH, GW);
  const DwPlan3 &d = c.d;
  char *w = (char *)ws + 256;
  float *xl = (float *)w;
  if (!copy) w += d.xl_bytes;
  uint8_t *gt = (uint8_t *)w;
  float *partial = (float *)(w + d.gt_bytes), *sums = (float *)((char *)partial + d.partial_bytes);
  c.pre = nhwc3(src, xl, B, CH, d.Cp, SH * SW, bias_of_src ? sums : nullptr);
  const int tiles = (int)(B * d.tiles_x * d.tiles_y);
  c.grad = Grad3{(const float *)A, gt, bias_of_src ? nullptr : sums, (int)M, (int)GH, (int)GW, d.tiles_x, d.tiles_y, d.mbs, tiles * d.mbs};
  Dw3 &p = c.p;
  p.g = Src3{copy ? copy : (const char *)xl, (const float *)map, (const float *)iw, nullptr, d.Cp, (int)SH, (int)SW, (int)K, (int)P, (int)GH,
             (int)GW, interp};
  p.gt = (const __nv_bfloat16 *)gt; p.partial = partial; p.status = (int *)ws;
  p.B = (int)B; p.mbs = d.mbs; p.groups = d.groups; p.slots = d.slots; p.tiles_x = d.tiles_x; p.tiles_y = d.tiles_y;
  p.splits = d.splits; p.stages = d.stages;
  c.red = Reduce3{partial, sums, (float *)gw, (float *)gb, d.splits, d.mbs * 128, d.groups * kDwN, (int)M, (int)CH, d.Cp, (int)K,
                  cdiv(M * CH * K, 256), bias_of_src ? (int)B * c.pre.px_blocks : tiles, bias_of_src ? d.Cp : d.mbs * 128, sm, sc, sk};
  c.channels = (int)(bias_of_src ? CH : M);
  return c;
}
int run_dw3(const DwCall3 &c, int prepared, cudaStream_t st) {
  if (c.kind == SRC_MAP1) launch_dw3<SRC_MAP1>(c.p, c.d.smem, st);
  else launch_dw3<SRC_MAP4>(c.p, c.d.smem, st);
  dw_reduce3_kernel<<<(unsigned)(c.red.blocks + c.channels), 256, 0, st>>>(c.red);
  return launch_status(2 + prepared);
}

}  // namespace

// gw[m, ch, k] = sum A[b, m, pix] * Col[b, pix, (ch, k)], and the bias gradient gb: the sums of A's rows or (bias_of_src: a
// transposed convolution, whose gathered side is the output's gradient) of the source's channels.
int x3_dw(const void *A, const void *src, const void *map, const void *iw, int64_t CH, int64_t SH, int64_t SW, int64_t K, int64_t P,
          int64_t GH, int64_t GW, int interp, int64_t M, int64_t B, void *gw, int64_t sm, int64_t sc, int64_t sk, void *gb, bool bias_of_src,
          void *ws, cudaStream_t st) {
  const DwCall3 c = dw_call3(A, src, map, iw, CH, SH, SW, K, P, GH, GW, interp, M, B, gw, sm, sc, sk, gb, bias_of_src, ws);
  dw_prepare3_kernel<<<(unsigned)(c.grad.blocks + c.pre.blocks), 256, 0, st>>>(c.pre, c.grad, c.p.status);
  return run_dw3(c, 1, st);
}

// All gradients of a convolution, or of a transposed one, with one pre-pass.  Both products of a transposed convolution gather from the
// output's gradient: its copy is made once.
size_t x3_backward_workspace(bool transposed, int64_t B, int64_t Cin, int64_t Cout, int64_t IH, int64_t IW, int64_t OH, int64_t OW, int64_t K,
                             int64_t P, int interp) {
  const size_t dx = transposed ? x3_gemm_workspace(false, B, Cout, OH * OW, K, P, interp, Cin, 0)
                               : x3_gemm_workspace(true, B, Cout, OH * OW, K, 0, 0, Cin, IH * IW);
  const size_t dw = transposed ? x3_dw_workspace(B, Cout, OH * OW, K, P, interp, Cin, IH, IW)
                               : x3_dw_workspace(B, Cin, IH * IW, K, P, interp, Cout, OH, OW);
  if (dx == 0 || dw == 0) return 0;
  const size_t shared = transposed ? dw_plan3(source3(false, P, interp), B, Cout, OH * OW, K, Cin, IH, IW).xl_bytes : 0;
  return align_up(dx, 256) + dw - shared;
}

int x3_backward(bool transposed, const void *gout, const void *x, const void *plan, const void *map, const void *iw, const void *weight,
                void *gx, void *gw, void *gb, int64_t B, int64_t Cin, int64_t Cout, int64_t IH, int64_t IW, int64_t OH, int64_t OW, int64_t K,
                int64_t P, int interp, void *ws, cudaStream_t st) {
  GemmCall3 dx = transposed ? gemm_call3(false, gout, map, iw, nullptr, Cout, OH, OW, K, P, IH, IW, interp, weight, Cout * K, K, 1, nullptr,
                                         gx, Cin, B, ws)
                            : gemm_call3(true, gout, nullptr, nullptr, plan, Cout, OH, OW, K, 0, IH, IW, 0, weight, K, Cin * K, 1, nullptr, gx,
                                         Cin, B, ws);
  void *ws2 = (char *)ws + align_up(transposed ? x3_gemm_workspace(false, B, Cout, OH * OW, K, P, interp, Cin, 0)
                                               : x3_gemm_workspace(true, B, Cout, OH * OW, K, 0, 0, Cin, IH * IW), 256);
  DwCall3 dw = transposed ? dw_call3(x, gout, map, iw, Cout, OH, OW, K, P, IH, IW, interp, Cin, B, gw, Cout * K, K, 1, gb, true, ws2,
                                     dx.p.g.xl)
                          : dw_call3(gout, x, map, iw, Cin, IH, IW, K, P, OH, OW, interp, Cout, B, gw, Cin * K, K, 1, gb, false, ws2);
  if (transposed) {
    dx.pre.sums = dw.pre.sums;
    dw.pre.blocks = 0;
  }
  mark_phase(0, st);
  backward_prepare3_kernel<<<(unsigned)(dw.grad.blocks + dx.wt.blocks + dx.pre.blocks + dw.pre.blocks), 256, 0, st>>>(
      dx.pre, dw.pre, dx.wt, dw.grad, dx.p.status, dw.p.status);
  mark_phase(1, st);
  int rc = run_gemm3(dx, 1, st);
  if (rc != SPH_OK) return rc;
  mark_phase(2, st);
  rc = run_dw3(dw, 0, st);
  mark_phase(3, st);
  return rc;
}

int x3_wait_status(int reset) {
  int v = 0;
  if (cudaMemcpyFromSymbol(&v, g_wait_status3, sizeof(int)) != cudaSuccess) return -1;
  if (reset && v) {
    const int zero = 0;
    if (cudaMemcpyToSymbol(g_wait_status3, &zero, sizeof(int)) != cudaSuccess) return -1;
  }
  return v;
}

}  // namespace sph

SPH_TU_STATUS(conv_x3)
