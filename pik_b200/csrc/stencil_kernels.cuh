// The full-frame 3x3 stencil passes:
//  * k_gaborish_tile: ConvolveGaborish (pik/gaborish.cc:137-159) of the
//    planes, for the stage export (the EPF recomputes the smoothed values
//    that it needs);
//  * k_gaborish_minmax: the min/max of its output (MinMax,
//    pik/epf_target.cc:980-1006), for the EPF guide, without storing it;
//  * k_final_direct: gaborish #2 (or a copy), ShrinkTo(xsize, ysize),
//    XybToRgb (pik/opsin_inverse.cc:38-123) and optional sRGB-8
//    (pik/color_management.cc:323-345, pik/external_image.cc:1205).
//
// k_gaborish_tile stages a 128 x TH output tile with its 1-pixel halo (rows
// y0 - 1 .. y0 + TH, columns x0 - 4 .. x0 + 131, widened to 16-byte
// boundaries) in shared memory: interior tiles with independent 128-bit loads
// (many in flight per thread), border tiles with mirrored scalar loads. Each
// thread then computes 4 adjacent columns of TH / 8 rows, reading 128-bit row
// segments and taking the left/right neighbours from the adjacent lanes.
// The arithmetic of each output is Sym3's, in the same order, so results are
// bit-identical to it. The padded plane width must be a multiple of 4 (it is
// 8 Bx).
// Included by recon_kernels.cu.
#pragma once

namespace pikgpu {

constexpr int kTileW = 128, kTileThreads = 256;
constexpr int kTileSW = kTileW + 8;  // staged columns x0 - 4 .. x0 + 131
constexpr int kGabTileH = 64;        // rows per CTA

// Symmetric 3x3 stencil of output column i (0..3) from three 6-value rows
// (columns x - 1 .. x + 4), in Sym3's operation order.
__device__ __forceinline__ float Sym3Rows(const float* t, const float* m,
                                          const float* b, int i, float w0,
                                          float w1, float w2) {
  const float sum_tb = t[i + 1] + b[i + 1];
  const float mul0 = m[i + 1] * w0;
  const float sum_lr = m[i] + m[i + 2];
  const float x1 = sum_tb + sum_lr;
  const float mul1 = x1 * w1 + mul0;
  const float sum_t2 = t[i] + t[i + 2];
  const float sum_b2 = b[i] + b[i + 2];
  const float x2 = sum_t2 + sum_b2;
  return x2 * w2 + mul1;
}

// Asynchronous 16-byte global -> shared copies: interior tiles are staged
// without passing through registers, every copy of a tile (all planes) in
// flight at once, and one wait before the CTA's barrier. The hardware
// tracks completion per thread, so the wait is no spin loop.
__device__ __forceinline__ void CpAsync16(void* smem, const void* gmem) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(
                   uint32_t(__cvta_generic_to_shared(smem))),
               "l"(gmem)
               : "memory");
}
__device__ __forceinline__ void CpAsync4(void* smem, const void* gmem) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(
                   uint32_t(__cvta_generic_to_shared(smem))),
               "l"(gmem)
               : "memory");
}
__device__ __forceinline__ void CpAsyncWaitAll() {
  asm volatile("cp.async.commit_group;\n\tcp.async.wait_group 0;" :::
                   "memory");
}

// Stages plane `p` (w x h, row stride w) around (x0, y0) into `t`
// (TH + 2 rows). Interior tiles are copied asynchronously: the caller
// calls CpAsyncWaitAll before its barrier.
template <int TH>
__device__ __forceinline__ void StageTile(const float* p, int w, int h,
                                          int x0, int y0,
                                          float (*t)[kTileSW]) {
  constexpr int kTileSH = TH + 2;
  const bool interior =
      x0 >= 4 && x0 + kTileW + 4 <= w && y0 >= 1 && y0 + TH + 1 <= h;
  if (interior) {
    constexpr int Q = kTileSW / 4;
    for (int i = threadIdx.x; i < kTileSH * Q; i += kTileThreads) {
      const int r = i / Q, q = i % Q;
      CpAsync16(&t[r][4 * q], p + size_t(y0 - 1 + r) * w + x0 - 4 + 4 * q);
    }
  } else {
    for (int i = threadIdx.x; i < kTileSH * kTileSW; i += kTileThreads) {
      const int r = i / kTileSW, col = i % kTileSW;
      t[r][col] = p[size_t(MirrorIdx(y0 - 1 + r, h)) * w +
                    MirrorIdx(x0 - 4 + col, w)];
    }
  }
}

// Staged row r as 6 values: columns 4 lane - 1 .. 4 lane + 4 of the tile.
__device__ __forceinline__ void TileRow6(const float (*t)[kTileSW], int r,
                                         int lane, float v[6]) {
  const float4 q = *reinterpret_cast<const float4*>(&t[r][4 + 4 * lane]);
  float left = __shfl_up_sync(0xFFFFFFFFu, q.w, 1);
  float right = __shfl_down_sync(0xFFFFFFFFu, q.x, 1);
  if (lane == 0) left = t[r][3];
  if (lane == 31) right = t[r][4 + kTileW];
  v[0] = left;
  v[1] = q.x, v[2] = q.y, v[3] = q.z, v[4] = q.w;
  v[5] = right;
}

__global__ void __launch_bounds__(kTileThreads)
    k_gaborish_tile(const float* in, int w, int h, int strength, float* out) {
  constexpr int TH = kGabTileH, R = TH / 8;
  __shared__ __align__(16) float t[TH + 2][kTileSW];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int c = blockIdx.z;
  const size_t plane = size_t(w) * h;
  const int x0 = blockIdx.x * kTileW, y0 = blockIdx.y * TH;
  StageTile<TH>(in + c * plane, w, h, x0, y0, t);
  CpAsyncWaitAll();
  __syncthreads();
  const float* wt = c_t.gaborish[strength];
  const float w0 = wt[0], w1 = wt[1], w2 = wt[2];
  const int x = x0 + 4 * lane;
  float a[6], m[6], b[6];
  TileRow6(t, R * warp, lane, a);
  TileRow6(t, R * warp + 1, lane, m);
#pragma unroll
  for (int j = 0; j < R; ++j) {
    TileRow6(t, R * warp + j + 2, lane, b);
    const int y = y0 + R * warp + j;
    if (x < w && y < h) {
      float r[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) r[i] = Sym3Rows(a, m, b, i, w0, w1, w2);
      *reinterpret_cast<float4*>(out + c * plane + size_t(y) * w + x) =
          make_float4(r[0], r[1], r[2], r[3]);
    }
#pragma unroll
    for (int i = 0; i < 6; ++i) {
      a[i] = m[i];
      m[i] = b[i];
    }
  }
}

// A warp's strip of a plane row for the 3x3 stencils: 30 lanes own 4 columns
// each, and lanes 0 and 31 hold the columns beside the strip, so that every
// lane's left and right neighbours come from the adjacent lanes (with 32
// owning lanes the outer neighbours were loads of single lanes and a select
// per value). Beyond the plane's border the neighbour mirrors to the border
// column itself.
constexpr int kStripW = 120;
struct StripLane {
  int x;     // first column; a halo lane's may lie outside
  int load;  // where its four values are read
  bool edge;  // warp-uniform: some lane lies outside
  __device__ StripLane(int x0, int w) {
    const int lane = threadIdx.x & 31;
    x = x0 - 4 + 4 * lane;
    load = min(max(x, 0), w - 4);
    edge = x0 == 0 || x0 + kStripW >= w;
  }
  // The lane's values of a row, mirrored at the border.
  __device__ float4 Load(const float* row, int w) const {
    float4 q = *reinterpret_cast<const float4*>(row + load);
    if (edge) {
      if (x < 0) q.w = q.x;
      if (x >= w) q.x = q.w;
    }
    return q;
  }
};
// Columns x - 1 .. x + 4 of an owning lane.
__device__ __forceinline__ void StripRow6(const float4& q, float (&v)[6]) {
  v[0] = __shfl_up_sync(0xFFFFFFFFu, q.w, 1);
  v[1] = q.x, v[2] = q.y, v[3] = q.z, v[4] = q.w;
  v[5] = __shfl_down_sync(0xFFFFFFFFu, q.x, 1);
}

// The frame's u8 guide with the 6-pixel mirrored border, 3 x (h + 12) x
// (w + 12), as the EPF takes it from `src` (gab > 0: smoothed by gaborish of
// that strength): the verification export and the adjoint's guide. A word of
// four pixels per thread (w + 12 is a multiple of 4), from the values at the
// mirrored coordinates around it, which is the smoothed value at the mirrored
// position: Sym3Rows adds each pair of neighbours first. At 1024x1024 a pixel
// per thread took 26 us, and with the smoothed plane written and read again
// 37 and a host synchronisation; this takes 14.
__global__ void __launch_bounds__(256)
    k_export_guide(const float* src, int gab, int w, int h, const uint32_t* mm,
                   uint8_t* guide) {
  const int wd = blockIdx.x * blockDim.x + threadIdx.x;
  const int gy = blockIdx.y * blockDim.y + threadIdx.y;
  const int c = blockIdx.z;
  if (4 * wd >= w + 12 || gy >= h + 12) return;
  float amin, mul, stretch;
  GuideParams(mm, &amin, &mul, &stretch);
  const float* p = src + size_t(c) * w * h;
  int x[6];
#pragma unroll
  for (int i = 0; i < 6; ++i) x[i] = MirrorIdx(4 * wd - 7 + i, w);
  float v[3][6];
#pragma unroll
  for (int r = 0; r < 3; ++r) {
    if (!gab && r != 1) continue;
    const float* row = p + size_t(MirrorIdx(gy - 7 + r, h)) * w;
#pragma unroll
    for (int i = 0; i < 6; ++i) v[r][i] = row[x[i]];
  }
  const float* wt = c_t.gaborish[gab];
  uint32_t word = 0;
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const float s = gab ? Sym3Rows(v[0], v[1], v[2], i, wt[0], wt[1], wt[2])
                        : v[1][i + 1];
    word |= uint32_t(uint8_t(uint32_t(__float2int_rz((s - amin) * mul))))
            << (8 * i);
  }
  *reinterpret_cast<uint32_t*>(
      guide + (size_t(c) * (h + 12) + gy) * (w + 12) + 4 * wd) = word;
}

// Minimum and maximum of three values, NaN if any is.
__device__ __forceinline__ float Min3NaN(float a, float b, float c) {
  float d;
  asm("min.NaN.f32 %0, %1, %2, %3;" : "=f"(d) : "f"(a), "f"(b), "f"(c));
  return d;
}
__device__ __forceinline__ float Max3NaN(float a, float b, float c) {
  float d;
  asm("max.NaN.f32 %0, %1, %2, %3;" : "=f"(d) : "f"(a), "f"(b), "f"(c));
  return d;
}

// Ordered min/max of gaborish #1 over n columns from x and rows y0 .. y1 - 1
// of a plane, value by value (the order of NaNs, which min.NaN and max.NaN
// do not keep, is that of their bits).
__device__ __noinline__ void GaborishMinMaxScalar(const float* p, int w, int h,
                                                  int strength, int x, int n,
                                                  int y0, int y1, uint32_t* lo,
                                                  uint32_t* hi) {
  const float* wt = c_t.gaborish[strength];
  for (int y = y0; y < y1; ++y) {
    for (int i = x; i < x + n; ++i) {
      float v[3][6];  // columns i - 1 .. i + 1 of the three rows
      for (int r = 0; r < 3; ++r)
        for (int k = 0; k < 3; ++k)
          v[r][k] = p[size_t(MirrorIdx(y - 1 + r, h)) * w +
                      MirrorIdx(i - 1 + k, w)];
      const uint32_t ob =
          OrderedBits(Sym3Rows(v[0], v[1], v[2], 0, wt[0], wt[1], wt[2]));
      *lo = min(*lo, ob);
      *hi = max(*hi, ob);
    }
  }
}

// Min/max of gaborish #1 without staging or barriers: each warp owns a strip
// of kGmmRows rows and loads its kGmmRows + 2 input rows as independent
// 16-byte loads (all in flight at once). Coordinates mirror at the image
// border and each output follows Sym3's operation order, so the min/max equal
// those of k_gaborish_tile. Grid: (warps of a plane / 8, 3). Issue bound it:
// with an integer min and max of every value's ordered bits, and edge loads
// by single lanes, it took 36 us at 4K and 260 at 8192x8192; now 28 and 191
// (4.2 TB/s).
constexpr int kGmmRows = 8;
__global__ void __launch_bounds__(256, 3)
    k_gaborish_minmax(const float* in, int w, int h, int strength,
                      uint32_t* mm) {
  PdlLaunchDependents();  // the plan may start on free SMs
  constexpr int R = kGmmRows;
  __shared__ uint32_t s_lo[8], s_hi[8];
  const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
  const int c = blockIdx.y;
  const int tiles_x = (w + kStripW - 1) / kStripW;
  const int wg = blockIdx.x * 8 + wib;
  const int x0 = (wg % tiles_x) * kStripW, y0 = (wg / tiles_x) * R;
  uint32_t lo = 0xFFFFFFFFu, hi = 0u;
  if (y0 < h) {  // warp-uniform
    const float* p = in + c * size_t(w) * h;
    const StripLane sl(x0, w);
    float4 q[R + 2];
#pragma unroll
    for (int r = 0; r < R + 2; ++r) {
      q[r] = sl.Load(p + size_t(MirrorIdx(y0 - 1 + r, h)) * w, w);
    }
    const float* wt = c_t.gaborish[strength];
    const float w0 = wt[0], w1 = wt[1], w2 = wt[2];
    const float inf = __int_as_float(0x7F800000);
    float mn = inf, mx = -inf;
    float a[6], m[6], b[6];
    StripRow6(q[0], a);
    StripRow6(q[1], m);
#pragma unroll
    for (int j = 0; j < R; ++j) {
      StripRow6(q[j + 2], b);
#pragma unroll
      for (int i = 0; i < 4; i += 2) {
        const float v0 = Sym3Rows(a, m, b, i, w0, w1, w2);
        const float v1 = Sym3Rows(a, m, b, i + 1, w0, w1, w2);
        mn = Min3NaN(mn, v0, v1);
        mx = Max3NaN(mx, v0, v1);
      }
#pragma unroll
      for (int i = 0; i < 6; ++i) {
        a[i] = m[i];
        m[i] = b[i];
      }
    }
    // Planes are a multiple of 8 rows: all of the strip's exist.
    if (lane >= 1 && lane <= 30 && sl.x < w) {
      lo = OrderedBits(mn);
      hi = OrderedBits(mx);
      if (mn != mn || mx != mx) {
        lo = 0xFFFFFFFFu, hi = 0u;
        GaborishMinMaxScalar(p, w, h, strength, sl.x, 4, y0, y0 + R, &lo, &hi);
      }
    }
  }
  for (int off = 16; off; off >>= 1) {
    lo = min(lo, __shfl_xor_sync(0xFFFFFFFFu, lo, off));
    hi = max(hi, __shfl_xor_sync(0xFFFFFFFFu, hi, off));
  }
  if (lane == 0) {
    s_lo[wib] = lo;
    s_hi[wib] = hi;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int i = 1; i < 8; ++i) {
      lo = min(lo, s_lo[i]);
      hi = max(hi, s_hi[i]);
    }
    if (lo <= hi) {
      atomicMin(&mm[c], lo);
      atomicMax(&mm[3 + c], hi);
    }
  }
}

// Opsin inverse of one pixel (XybToRgb), same operation order as before.
__device__ __forceinline__ void XybToRgb(float x, float y, float b, float* r,
                                         float* g, float* bl) {
  const float* m = c_t.opsin_inv;
  const float gr = 1.0f * (y + x);
  const float gg = 1.0f * (y - x);
  const float gb = b;
  const float mr = gr * gr * gr + c_t.opsin_neg_bias[0];
  const float mg = gg * gg * gg + c_t.opsin_neg_bias[1];
  const float mb = gb * gb * gb + c_t.opsin_neg_bias[2];
  float lr = m[0] * mr, lg = m[3] * mr, lb = m[6] * mr;
  const float tr = m[1] * mg, tg = m[4] * mg, tb = m[7] * mg;
  lr = m[2] * mb + lr;
  lg = m[5] * mb + lg;
  lb = m[8] * mb + lb;
  *r = lr + tr;
  *g = lg + tg;
  *bl = lb + tb;
}

// Completes the EPF's output planes for the stage export: regions that it
// left out get its input. One thread per 4 pixels of a plane.
__global__ void k_fill_regions(const float* in, const uint32_t* region, int w,
                               int h, float* out) {
  const size_t o = 4 * (blockIdx.x * size_t(blockDim.x) + threadIdx.x);
  if (o >= 3 * size_t(w) * h) return;
  const int x = int(o % w), y = int(o / w % h);
  const int rw = (w + kRegionW - 1) / kRegionW;
  if (region[(y / kRegionH) * rw + x / kRegionW]) return;
  *reinterpret_cast<float4*>(out + o) =
      *reinterpret_cast<const float4*>(in + o);
}

// The final pass without staging or barriers: each warp owns a strip of
// kFinRows output rows of the three planes and loads its input rows
// (kFinRows + 2 per plane with gaborish, kFinRows without) as independent
// 16-byte loads; the horizontal neighbours come from the adjacent lanes
// (StripLane). Coordinates mirror at the padded plane's border (pw x ph).
// `region` (NULL: always `in`): the EPF's region flags; where a region's flag
// is 0 its pixels are read from `alt` (the EPF's input). `vec_lin`: the
// linear outputs may be written as float4 (width, stride and base all
// multiples of 4 floats / 16 bytes); `vec_rgb`: the 8-bit rows of 4 pixels as
// three words (stride and base multiples of 4 bytes). Grid: warps / 8.
//
// Issue bound it too: with 128 owned columns per warp, the rows of all planes
// held at once (122 registers) and byte stores it took 55 us at 4K, 416 at
// 8192x8192 and 30 at 1920x1080 with the 8-bit output; now 43, 307 (5.2 TB/s)
// and 24. One row per warp: 48, 354 and 24; four: 44, 310 and 29.
constexpr int kFinRows = 2;
template <bool kGab>
__host__ __device__ constexpr int FinalStripW() {
  return kGab ? kStripW : 128;
}
template <bool kGab>
__global__ void __launch_bounds__(256, 2)
    k_final_direct(const float* in, const float* alt, const uint32_t* region,
                   int pw, int ph, int w, int h, int strength, float* pre,
                   float* lin, size_t lin_stride, int vec_lin, uint8_t* rgb8,
                   size_t rgb8_stride, int vec_rgb) {
  constexpr int R = kFinRows, NR = kGab ? R + 2 : R;
  const int lane = threadIdx.x & 31;
  const int wg = blockIdx.x * 8 + (threadIdx.x >> 5);
  constexpr int kW = FinalStripW<kGab>();
  const int tiles_x = (w + kW - 1) / kW;
  const int x0 = (wg % tiles_x) * kW, y0 = (wg / tiles_x) * R;
  if (y0 >= h) return;  // warp-uniform; no barriers below
  const size_t plane = size_t(pw) * ph;
  StripLane sl(x0, pw);
  if (!kGab) {
    sl.x = x0 + 4 * lane;
    sl.load = min(sl.x, pw - 4);
    sl.edge = false;
  }
  const int x = sl.x;
  const int rw = (pw + kRegionW - 1) / kRegionW;
  const float* row[NR];
#pragma unroll
  for (int r = 0; r < NR; ++r) {
    const int y = MirrorIdx(kGab ? y0 - 1 + r : y0 + r, ph);
    const float* src =
        !region || region[(y / kRegionH) * rw + sl.load / kRegionW] ? in : alt;
    row[r] = src + size_t(y) * pw;
  }
  const float* wt = c_t.gaborish[strength];
  const float w0 = wt[0], w1 = wt[1], w2 = wt[2];
  float v[R][3][4];
#pragma unroll
  for (int c = 0; c < 3; ++c) {
    float4 q[NR];
#pragma unroll
    for (int r = 0; r < NR; ++r) q[r] = sl.Load(row[r] + c * plane, pw);
    if (kGab) {
      float a[6], m[6], b[6];
      StripRow6(q[0], a);
      StripRow6(q[1], m);
#pragma unroll
      for (int j = 0; j < R; ++j) {
        StripRow6(q[j + 2], b);
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          v[j][c][i] = Sym3Rows(a, m, b, i, w0, w1, w2);
        }
#pragma unroll
        for (int i = 0; i < 6; ++i) a[i] = m[i], m[i] = b[i];
      }
    } else {
#pragma unroll
      for (int j = 0; j < R; ++j) {
        v[j][c][0] = q[j].x, v[j][c][1] = q[j].y;
        v[j][c][2] = q[j].z, v[j][c][3] = q[j].w;
      }
    }
  }
  if (x >= w || (kGab && (lane == 0 || lane == 31))) return;
  const int n = min(4, w - x);
#pragma unroll
  for (int j = 0; j < R; ++j) {
    const int y = y0 + j;
    if (y >= h) break;
    if (pre) {
#pragma unroll
      for (int c = 0; c < 3; ++c)
#pragma unroll
        for (int i = 0; i < 4; ++i)
          if (i < n) pre[(size_t(c) * h + y) * w + x + i] = v[j][c][i];
    }
    float r[4], g[4], bl[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      XybToRgb(v[j][0][i], v[j][1][i], v[j][2][i], &r[i], &g[i], &bl[i]);
    }
    if (lin) {
      float* o0 = lin + size_t(y) * lin_stride + x;
      float* o1 = o0 + lin_stride * h;
      float* o2 = o1 + lin_stride * h;
      if (vec_lin) {
        *reinterpret_cast<float4*>(o0) = make_float4(r[0], r[1], r[2], r[3]);
        *reinterpret_cast<float4*>(o1) = make_float4(g[0], g[1], g[2], g[3]);
        *reinterpret_cast<float4*>(o2) =
            make_float4(bl[0], bl[1], bl[2], bl[3]);
      } else {
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          if (i < n) {
            o0[i] = r[i];
            o1[i] = g[i];
            o2[i] = bl[i];
          }
        }
      }
    }
    if (rgb8) {
      uint8_t* o = rgb8 + size_t(y) * rgb8_stride + 3 * size_t(x);
      uint32_t px[12];
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        px[3 * i] = Srgb8(r[i]);
        px[3 * i + 1] = Srgb8(g[i]);
        px[3 * i + 2] = Srgb8(bl[i]);
      }
      if (vec_rgb && n == 4) {
#pragma unroll
        for (int k = 0; k < 3; ++k) {
          reinterpret_cast<uint32_t*>(o)[k] = px[4 * k] | px[4 * k + 1] << 8 |
                                              px[4 * k + 2] << 16 |
                                              px[4 * k + 3] << 24;
        }
      } else {
#pragma unroll
        for (int k = 0; k < 12; ++k) {
          if (k < 3 * n) o[k] = uint8_t(px[k]);
        }
      }
    }
  }
}

}  // namespace pikgpu
