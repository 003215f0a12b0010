// Gathers over plane groups: the float32 path of resampling and pooling when the caller supplies scratch.
//
// The operators of resample.cu and pool.cu apply ONE sparse pattern (a sample map or its inverse, a scatter plan) to
// many independent (batch, channel) planes.  Read straight from NCHW, every tap costs one 4-byte load per plane: a warp
// load of 32 neighbouring taps touches two to seven 128-byte lines for 128 bytes of data, a random tap moves a 32-byte
// sector for 4 useful bytes, and the pattern itself is decoded or read again for every few planes.  Here groups of PG
// planes (32, fewer where there are fewer) are first transposed into rows of PG floats per pixel.  A thread owns one
// output pixel and VP = 8 planes of its group (4 in groups of four); the PG / VP threads of a pixel read a tap as one
// contiguous row, so the L1 serves whole 128-byte lines whatever the map's stride or locality, and a plan entry or a
// decoded tap costs its instructions once per eight planes.
//
// The transposition is a launch of its own per chunk of planes (chunks bound the scratch; keeping them small enough for the
// rows to stay in L2, or overlapping one chunk's transposition with the previous one's gathers, was measured and changes
// nothing: the gathers are bound by instruction issue, L1 and latency).
//
// Sums are taken in the same order with the same roundings as in the direct kernels: results are bit-identical.
#pragma once

#include "common.cuh"

namespace sph {

// ---- four planes of one pixel -----------------------------------------------------------------------------------
__device__ __forceinline__ unsigned long long pack_f32x2(float lo, float hi) {
  unsigned long long r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
  return r;
}
__device__ __forceinline__ void unpack_f32x2(unsigned long long v, float &lo, float &hi) {
  asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v));
}
__device__ __forceinline__ unsigned long long add_f32x2(unsigned long long a, unsigned long long b) {
  unsigned long long r;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
// VP planes of one pixel.
template <int VP> struct Vec {
  float f[VP];
};
template <int VP> __device__ __forceinline__ Vec<VP> vec_fill(float v) {
  Vec<VP> r;
#pragma unroll
  for (int i = 0; i < VP; i++) r.f[i] = v;
  return r;
}
// w * v and a + b, separately rounded (as RN<float>); the sums go two at a time.  The products are scalar multiplies: the
// assembler contracts a packed multiply followed by a packed add into one fused operation even though both carry .rn
// (measured: the last bit of a quarter of the interpolated values).
template <int VP> __device__ __forceinline__ Vec<VP> vec_scale(float w, const Vec<VP> &v) {
  Vec<VP> r;
#pragma unroll
  for (int i = 0; i < VP; i++) r.f[i] = __fmul_rn(w, v.f[i]);
  return r;
}
template <int VP> __device__ __forceinline__ Vec<VP> vec_add(const Vec<VP> &a, const Vec<VP> &b) {
  Vec<VP> r;
#pragma unroll
  for (int i = 0; i < VP; i += 2)
    unpack_f32x2(add_f32x2(pack_f32x2(a.f[i], a.f[i + 1]), pack_f32x2(b.f[i], b.f[i + 1])), r.f[i], r.f[i + 1]);
  return r;
}
// One tap: a thread's part of a row of the scratch (written by an earlier launch, so the read-only path is safe).
template <int VP> __device__ __forceinline__ Vec<VP> row_load(const char *rows, unsigned off) {
  Vec<VP> v;
  if constexpr (VP == 8)
    asm("ld.global.nc.v8.f32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
        : "=f"(v.f[0]), "=f"(v.f[1]), "=f"(v.f[2]), "=f"(v.f[3]), "=f"(v.f[4]), "=f"(v.f[5]), "=f"(v.f[6]), "=f"(v.f[7])
        : "l"(rows + off));
  else
    asm("ld.global.nc.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.f[0]), "=f"(v.f[1]), "=f"(v.f[2]), "=f"(v.f[3]) : "l"(rows + off));
  return v;
}

// Decoded taps of one coordinate as byte offsets of rows of `pitch` bytes; a tap outside the image reads the zero row
// behind the last pixel.
struct RowTaps {
  uint4 off;
  float4 w;
};
template <int INTERP> __device__ __forceinline__ RowTaps row_taps(float x, float y, int H, int W, unsigned pitch) {
  Taps<float> t;
  decode<float, INTERP>(x, y, H, W, t);
  const unsigned zero = (unsigned)t.limit * pitch;
  unsigned o[4];
#pragma unroll
  for (int i = 0; i < 4; i++)
    o[i] = i < TapCount<INTERP>::value && t.off[i] >= 0 && index_ok(t.off[i], t.limit) ? (unsigned)t.off[i] * pitch : zero;
  RowTaps r;
  r.off = make_uint4(o[0], o[1], o[2], o[3]);
  r.w = INTERP == SPH_NEAREST ? make_float4(1.f, 0.f, 0.f, 0.f) : make_float4(t.w[0], t.w[1], t.w[2], t.w[3]);
  return r;
}

// Interpolated value: ((w0 v0 + w1 v1) + w2 v2) + w3 v3 (common.cuh: gather()).
template <int VP, int INTERP> __device__ __forceinline__ Vec<VP> row_gather(const char *rows, const RowTaps &t) {
  const Vec<VP> v0 = row_load<VP>(rows, t.off.x);
  if constexpr (INTERP == SPH_NEAREST) {
    return v0;
  } else {
    const Vec<VP> v1 = row_load<VP>(rows, t.off.y), v2 = row_load<VP>(rows, t.off.z), v3 = row_load<VP>(rows, t.off.w);
    return vec_add<VP>(vec_add<VP>(vec_add<VP>(vec_scale<VP>(t.w.x, v0), vec_scale<VP>(t.w.y, v1)), vec_scale<VP>(t.w.z, v2)),
                       vec_scale<VP>(t.w.w, v3));
  }
}

// ---- chunks ----------------------------------------------------------------------------------------------------
constexpr int kStageThreads = 256;
constexpr size_t kStageScratch = (size_t)256 << 20;
// Largest group of an unpooled gather (resample_from_map), well inside what pays at the nine reads a pixel that were measured: 32
// planes, smooth and random map, direct and in groups, by group: 4 MB 15 and 20 us, 27 and 19; 16 MB 27 and 26, 98 and 28; 32 MB 53
// and 42, 188 and 46; 64 MB 102 and 87, 376 and 99; 128 MB 198 and 179, 748 and 242; 256 MB 385 and 423, 1494 and 533.
constexpr size_t kStageGroup = (size_t)34 << 20;
constexpr int kScatterGroup = 16;                 // largest group of a scatter (resample_to_map)

struct PlaneChunks {
  int planes, group_planes, groups, per_chunk, n_src;  // n_src: pixels of one source plane
  size_t group_bytes;
  char *buf;
};

// plane_bytes: scratch per pixel and plane: 4, or 5 with a winning slot.  Groups as large as possible (32 planes fill a
// 128-byte line) that do not pad the planes by more than a quarter over groups of four; `most`: the operator's largest.
inline PlaneChunks stage_chunks(int64_t planes, int64_t n_src, int plane_bytes, int most = 32) {
  int pg = most;
  while (pg > 4 && (planes + pg - 1) / pg * pg * 4 > (planes + 3) / 4 * 4 * 5) pg /= 2;
  PlaneChunks c{};
  c.planes = (int)planes;
  c.group_planes = pg;
  c.n_src = (int)n_src;
  c.groups = (int)((planes + pg - 1) / pg);
  c.group_bytes = align_up((size_t)(n_src + 1) * pg * plane_bytes, 256);
  int64_t per = (int64_t)(kStageScratch / c.group_bytes);
  if (per < 1) per = 1;
  const int64_t chunks = (c.groups + per - 1) / per;
  c.per_chunk = (int)((c.groups + chunks - 1) / chunks);
  return c;
}
inline size_t stage_bytes(const PlaneChunks &c) { return (size_t)c.per_chunk * c.group_bytes; }
// Row offsets are 32-bit.
inline bool stage_fits(const PlaneChunks &c) { return c.group_bytes < ((size_t)1 << 32); }
inline bool scratch_ok(const void *ws) { return ws != nullptr && ((uintptr_t)ws & 31) == 0; }

// Transposition: a thread reads four pixels of four planes as 16-byte vectors and stores its 16 bytes of four rows; the PG / 4
// threads of a pixel complete the row.  Planes whose rows do not all start 16-byte aligned go through shared memory instead, read
// pixel by pixel in whole segments (four scattered reads in place of a vector took up to 1.3 times as long).
template <int PG> constexpr int kStagePixels = 4 * kStageThreads / (PG / 4);  // pixels of one block
template <int PG> inline int stage_tiles(int64_t n_src) { return cdiv(n_src + 1, kStagePixels<PG>); }

__host__ __device__ inline bool stage_aligned(const float *x, int n_src) { return (n_src & 3) == 0 && (((uintptr_t)x) & 15) == 0; }
template <int PG> constexpr size_t kStageBlock = (size_t)PG * (kStagePixels<PG> + 1) * 4;
template <int PG>
__device__ __forceinline__ void stage_scalar(const float *__restrict__ x, int planes, int n_src, int p0, int tile, char *buf) {
  constexpr int LP = PG / 4, PX = kStagePixels<PG>, LOADS = PG * PX / kStageThreads;
  extern __shared__ __align__(16) unsigned char stage_block[];  // (dynamic: the aligned case keeps it for L1)
  float(*block)[PX + 1] = (float(*)[PX + 1])stage_block;
  const int i0 = tile * PX;
  const float *src = x + (size_t)p0 * n_src + i0;
#pragma unroll 1
  for (int l0 = 0; l0 < LOADS; l0 += 8) {  // eight loads in flight
    float f[8];
#pragma unroll
    for (int l = 0; l < 8; l++) {
      const int e = threadIdx.x + (l0 + l) * kStageThreads, p = e / PX, i = e % PX;
      f[l] = p0 + p < planes && i0 + i < n_src ? __ldcs(src + (size_t)p * n_src + i) : 0.0f;  // (pixel n_src: the zero row)
    }
#pragma unroll
    for (int l = 0; l < 8; l++) {
      const int e = threadIdx.x + (l0 + l) * kStageThreads;
      block[e / PX][e % PX] = f[l];
    }
  }
  __syncthreads();
  const int q = threadIdx.x % LP * 4;
#pragma unroll
  for (int i = threadIdx.x / LP; i < PX; i += kStageThreads / LP)
    if (i0 + i <= n_src)
      ((float4 *)buf)[(size_t)(i0 + i) * LP + q / 4] = make_float4(block[q][i], block[q + 1][i], block[q + 2][i], block[q + 3][i]);
}

// p0: first plane of the group; buf: the group's rows
template <int PG>
__device__ __forceinline__ void stage_quad(const float *__restrict__ x, int planes, int n_src, int p0, int tile, char *buf) {
  constexpr int LP = PG / 4;
  if (!stage_aligned(x, n_src)) return stage_scalar<PG>(x, planes, n_src, p0, tile, buf);
  const int q = threadIdx.x % LP, i = tile * kStagePixels<PG> + threadIdx.x / LP * 4;
  if (i > n_src) return;
  const int np = planes - p0 - q * 4, n = n_src - i;
  const float *src = x + (size_t)(p0 + q * 4) * n_src + i;
  float f[4][4];  // [plane][pixel]
#pragma unroll
  for (int j = 0; j < 4; j++) {
    const float4 v = j < np && n > 0 ? __ldcs((const float4 *)(src + (size_t)j * n_src)) : make_float4(0.f, 0.f, 0.f, 0.f);
    f[j][0] = v.x; f[j][1] = v.y; f[j][2] = v.z; f[j][3] = v.w;
  }
  float4 *row = (float4 *)buf + (size_t)i * LP + q;
#pragma unroll
  for (int k = 0; k < 4; k++)
    if (k <= n) row[(size_t)k * LP] = make_float4(f[0][k], f[1][k], f[2][k], f[3][k]);  // (k == n: the zero row)
}

// Op: c, stage_tiles and use_tiles (blocks of one group); stage(first plane, rows, tile) transposes,
// use(first plane, rows, tile) works.
template <class Op, bool STAGE>
__global__ void __launch_bounds__(kStageThreads) plane_group_kernel(const Op op, int first_group) {
  const FastDiv &tiles = STAGE ? op.stage_tiles : op.use_tiles;
  const unsigned g = tiles.div(blockIdx.x), tile = blockIdx.x - g * tiles.d;
  const int p0 = (first_group + (int)g) * op.c.group_planes;
  char *rows = op.c.buf + (size_t)g * op.c.group_bytes;
  if (STAGE) op.stage(p0, rows, (int)tile);
  else op.use(p0, rows, (int)tile);
}

template <class Op>
int launch_plane_groups(const Op &op, size_t smem, cudaStream_t st) {
  int n = 0;
  for (int g = 0; g < op.c.groups; g += op.c.per_chunk, n += 2) {
    const unsigned groups = (unsigned)(op.c.groups - g < op.c.per_chunk ? op.c.groups - g : op.c.per_chunk);
    plane_group_kernel<Op, true><<<groups * op.stage_tiles.d, kStageThreads, op.stage_smem(), st>>>(op, g);
    plane_group_kernel<Op, false><<<groups * op.use_tiles.d, kStageThreads, smem, st>>>(op, g);
  }
  return launch_status(n);
}

// Work split of the using blocks: VP planes of one output per thread.  The threads of a warp are the LP threads of a row
// times 32 / LP outputs: eight consecutive ones (a store of one plane then writes whole 32-byte sectors) of each of 4 / LP
// rows.  A block's TO outputs are eight columns of 32 / LP rows, so that the taps of neighbouring outputs meet in L1: one
// image row of 64 outputs needs the rows of 8 pixels per output where the 8 x 8 block needs 5 (3 x 3 bilinear map of stride
// 2), and four such blocks no longer overflow the L1 (B200: L1 hit rate 40 % before).
template <int PG> struct Split {
  static constexpr int VP = PG < 8 ? PG : 8, LP = PG / VP, TO = kStageThreads / LP;
  static constexpr int TX = 8, TY = TO / TX;
};
// Outputs as a (height, width) image cut into TX x TY blocks.
struct TileGrid {
  int width, height;
  FastDiv across;
  template <int PG> static TileGrid make(int64_t height, int64_t width) {
    return TileGrid{(int)width, (int)height, FastDiv::make(cdiv(width, Split<PG>::TX))};
  }
  template <int PG> unsigned tiles() const { return across.d * (unsigned)cdiv(height, Split<PG>::TY); }
  // Output of this block's local index `l`, or -1 outside the image.
  template <int PG> __device__ __forceinline__ int output(int tile, int l) const {
    const int ty = (int)across.div((unsigned)tile), tx = tile - ty * (int)across.d;
    const int x = tx * Split<PG>::TX + l % Split<PG>::TX, y = ty * Split<PG>::TY + l / Split<PG>::TX;
    return x < width && y < height ? y * width + x : -1;
  }
};

// A thread's planes [p, p + VP) of output i.
template <int VP>
__device__ __forceinline__ void store_planes(float *__restrict__ out, int n, int i, int p, int planes, const Vec<VP> &v) {
  float *o = out + (size_t)p * n + i;
  if (p + VP <= planes) {
#pragma unroll
    for (int j = 0; j < VP; j++) __stcs(o + (size_t)j * n, v.f[j]);
  } else {
#pragma unroll
    for (int j = 0; j < VP; j++)
      if (p + j < planes) __stcs(o + (size_t)j * n, v.f[j]);
  }
}

#define SPH_DISPATCH_GROUP(pg, ...)                            \
  switch (pg) {                                                \
    case 32: { constexpr int PG = 32; __VA_ARGS__; break; }    \
    case 16: { constexpr int PG = 16; __VA_ARGS__; break; }    \
    case 8: { constexpr int PG = 8; __VA_ARGS__; break; }      \
    default: { constexpr int PG = 4; __VA_ARGS__; break; }     \
  }

}  // namespace sph
