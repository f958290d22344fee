// Edge-preserving filter (AdaptiveFilter + WeightedSum,
// pik/epf_target.cc:526-801, 1113-1278) on packed guide bytes.
//
// A CTA filters a 64 x TH pixel tile, a thread ROWS rows of one column: lane
// l of warp w owns the pixels (x0 + 32 (w mod 2) + l, y0 + ROWS (w / 2) + j),
// j < ROWS (the 32 lanes of a warp read 32 consecutive values of every
// shared-memory row; the rows lie inside one 8x8 block row).
//
// The u8 guide is staged in shared memory as one 32-bit word per byte
// offset: word o of a row holds the guide bytes o .. o + 3. The 4 guide bytes
// of a patch row at any offset are then one 32-bit load (and the 32 lanes'
// loads of 32 consecutive offsets hit 32 consecutive words, free of bank
// conflicts), and the sum of absolute differences against the centre
// pixel's patch row is one __vsadu4. For every displacement (cy, cx) of the
// 7 x 8 neighbourhood and every channel, a lane forms ROWS + 2 patch-row SADs
// of its column and sums them vertically into the 3 x 4 patch SADs of its
// rows; the SAD is the maximum over the channels. The SADs are exact integers; the weights
// (WeightFast's bit construction) and the weighted sums follow the
// reference's neighbour order (cy = -3..3, cx = -3..4) with separately
// rounded products and sums, so the output equals the per-pixel formulation
// bit for bit.
//
// The guide is quantised from the verification override (bytes), or from the
// staged input tile: its values (the sharpened guide, a frame without
// gaborish, the DC image) or -- the common case -- gaborish of them (the
// smoothed plane is then never written to memory; `gab` > 0 selects it and
// its strength). Border tiles hold mirrored values and take the same steps:
// 402 -> 380 us at 3001x2003, 22 -> 14 on the DC image of a 256x256 frame,
// against mirroring every guide byte's coordinates.
// Bound by the issue slots and the shared-memory reads. A thread takes eight
// rows, a whole block row: against four, ten row SADs serve eight patches
// instead of six serving four, and fewer guide rows are read per pixel; the
// packed products and sums (packed_fp32.cuh) take another 4% (FP32) and 5%.
// Together 220 -> 198 us on a 4K frame with a third of the blocks filtered
// (FP32; split-BF16 176 -> 164) and 375 -> 342 at 3001x2003 with all of them.
// Tiles of 32 rows: 8% slower (two CTAs fewer per SM).
// Included by recon_kernels.cu.
#pragma once

namespace pikgpu {

constexpr int kEpfW = 64;               // tile width
constexpr int kEpfH = 16, kEpfRows = 8;  // its rows, and those of a thread
constexpr int kEpfGBytes = 80;          // guide bytes x0 - 8 .. x0 + 71
constexpr int kEpfGRow = kEpfGBytes;    // words per guide row (one per byte)
// Input tile with a 5-pixel halo (enough for gaborish at the guide's
// 4-pixel halo): rows y0 - 5 .. y0 + TH + 4, cols x0 - 12 .. x0 + 75 (the
// column range is widened to 16-byte boundaries for vector loads).
constexpr int kEpfTW = kEpfW + 24;
constexpr int kEpfTS = kEpfTW;               // row stride in floats
constexpr int kEpfTRow0 = 2, kEpfTCol0 = 9;  // tile index of (y0-3, x0-3)
constexpr int kEpfAligned = kEpfGBytes / 4;  // aligned guide words per row
// Shared memory of k_epf_box with a tile of `th` rows: the guide words (one
// per byte offset), the input tile and the aligned guide words.
constexpr size_t EpfSmemBytes(int th) {
  return size_t(3) * (th + 8) * kEpfGRow * 4 +
         size_t(3) * (th + 10) * kEpfTS * 4 +
         size_t(3) * (th + 8) * kEpfAligned * 4 + 16;  // + the TMA mbarrier
}
// Bytes of one tile's TMA copy (three planes of TH + 10 rows of kEpfTW).
__host__ __device__ constexpr uint32_t EpfTileBytes(int th) {
  return uint32_t(3 * (th + 10) * kEpfTW * 4);
}

// WeightFast (pik/epf_target.cc:304-428) as 4 integer operations:
// ((int16(min(sad, 507) << 6) * mul) >> 16 + (127 << 7)) in the high half of
// a float equals ((min(sad, 507) * 64 mul) & 0xFFFF0000) + 0x3F800000 for
// every sad >= 0 and -32768 <= mul < 0 (the product fits in int32).
__device__ __forceinline__ float EpfWeight(int mul64, int sad) {
  const int t = min(sad, 507) * mul64;
  return __uint_as_float((uint32_t(t) & 0xFFFF0000u) + 0x3F800000u);
}

// The weight with the reference's cut-off (weights below 0.05 are 0) in
// four integer operations. EpfWeight falls as the SAD grows (mul < 0), so
// the cut-off is a SAD threshold `thr` per sigma (c_t.epf_thr); above it
// the weight is `cap`: 0, or EpfWeight(507) when even the largest clamped
// SAD keeps its weight (then thr = 507). For sad <= thr <= 507 the product
// has no wrap and the clamp is the identity; larger SADs only select `cap`.
struct EpfCut {
  uint32_t thr;
  float cap;
};
__device__ __forceinline__ EpfCut EpfCutOf(int sigma, int mul64) {
  EpfCut k;
  k.thr = uint32_t(c_t.epf_thr[sigma]);
  k.cap = k.thr == 507u ? EpfWeight(mul64, 507) : 0.0f;
  return k;
}
__device__ __forceinline__ float EpfCutWeight(int mul64, EpfCut k,
                                              uint32_t sad) {
  const uint32_t u = sad * uint32_t(mul64) + 0x3F800000u;
  return sad <= k.thr ? __uint_as_float(u & 0xFFFF0000u) : k.cap;
}

// Sum of the absolute differences of the four bytes of a and b, plus c
// (the accumulating form of __vsadu4).
__device__ __forceinline__ uint32_t Sad4(uint32_t a, uint32_t b, uint32_t c) {
  uint32_t d;
  asm("vabsdiff4.u32.u32.u32.add %0, %1, %2, %3;"
      : "=r"(d)
      : "r"(a), "r"(b), "r"(c));
  return d;
}

// The 3-row patch SADs of R = 8, 4, 2 or 1 pixel rows from R + 2 patch-row
// pairs (centre row r against window row r): for eight rows ten byte-SADs,
// where the sums of two neighbouring rows accumulate one onto the other, and
// eight adds, which need not run on the integer ALU. c0: the first channel
// (no maximum).
template <bool c0, int R>
__device__ __forceinline__ void PatchSads(const uint32_t* rf,
                                          const uint32_t* wd, uint32_t* sad) {
  static_assert(R == 8 || R == 4 || R == 2 || R == 1, "rows per thread");
  uint32_t s[R];
  if constexpr (R == 8) {
    const uint32_t h2 = Sad4(rf[2], wd[2], 0u);
    const uint32_t h3 = Sad4(rf[3], wd[3], 0u);
    const uint32_t h4 = Sad4(rf[4], wd[4], 0u);
    const uint32_t h5 = Sad4(rf[5], wd[5], 0u);
    const uint32_t h7 = Sad4(rf[7], wd[7], 0u);
    const uint32_t p12 = Sad4(rf[1], wd[1], h2);
    const uint32_t p34 = h3 + h4;
    const uint32_t p56 = Sad4(rf[6], wd[6], h5);
    const uint32_t p78 = Sad4(rf[8], wd[8], h7);
    s[0] = Sad4(rf[0], wd[0], p12);
    s[1] = p12 + h3;
    s[2] = p34 + h2;
    s[3] = p34 + h5;
    s[4] = p56 + h4;
    s[5] = p56 + h7;
    s[6] = p78 + (p56 - h5);
    s[7] = Sad4(rf[9], wd[9], p78);
  } else if constexpr (R == 4) {
    const uint32_t h2 = Sad4(rf[2], wd[2], 0u);
    const uint32_t h3 = Sad4(rf[3], wd[3], 0u);
    const uint32_t p12 = Sad4(rf[1], wd[1], h2);
    const uint32_t p34 = Sad4(rf[4], wd[4], h3);
    s[0] = Sad4(rf[0], wd[0], p12);
    s[1] = p12 + h3;
    s[2] = p34 + h2;
    s[3] = Sad4(rf[5], wd[5], p34);
  } else {
    uint32_t p = 0u;  // the rows that all R patches share
#pragma unroll
    for (int i = R - 1; i < 3; ++i) p = Sad4(rf[i], wd[i], p);
    s[0] = p;
    if constexpr (R == 2) {
      s[0] = Sad4(rf[0], wd[0], p);
      s[1] = Sad4(rf[3], wd[3], p);
    }
  }
#pragma unroll
  for (int j = 0; j < R; ++j) sad[j] = c0 ? s[j] : max(sad[j], s[j]);
}

// The frame EPF's work list, made by k_epf_plan: the regions of kEpfW x
// kEpfRegionH pixels that hold a filtered block. The output of the others is
// the input, and is not written: their readers take the input there
// (k_final_direct; the clamp only visits filtered blocks, and no block
// crosses regions). `sigma` is the blocks' sigma. The DC image's tiles are
// all taken; its blocks share one sigma (SigmaFromQuant of the constant
// `dc_qf` with a DCT strategy and LUT 0, AdaptiveDCReconstruction,
// pik/adaptive_reconstruction.cc:300-318).
// `sum_w` (NULL: not written): the plane of the filtered pixels' weight sums,
// for the adjoint.
struct EpfWork {
  const uint32_t* list;
  const int* count;
  const int32_t* sigma;
  int dc_qf;
  float* sum_w;
};
constexpr int kEpfRegionH = kRegionH;  // every tile height divides it
static_assert(kEpfW == kRegionW, "a region is as wide as a tile");

// The DC image's output: instead of storing the filtered value, the clamp
// of AdaptiveDCReconstruction (pik/adaptive_reconstruction.cc:319-331),
// dc = max(dc - hs, min(filtered, dc + hs)), into the w x h planes at `dc`
// (the padding is dropped). dc NULL: the frame EPF, which stores `out`.
struct EpfDc {
  float* dc;
  int w, h;
  float hs0, hs1, hs2;
};

// Stores the value of channel c at pixel (px, y) of the tile's output.
__device__ __forceinline__ void EpfStore(float* out, const EpfDc& dco,
                                         size_t plane, int w, int c, int px,
                                         int y, float v) {
  if (dco.dc) {
    if (px < dco.w && y < dco.h) {
      float& d = dco.dc[(size_t(c) * dco.h + y) * dco.w + px];
      const float hs = c == 0 ? dco.hs0 : c == 1 ? dco.hs1 : dco.hs2;
      const float lo = d - hs, hi = d + hs;
      const float m = v < hi ? v : hi;
      d = lo < m ? m : lo;
    }
  } else {
    out[c * plane + size_t(y) * w + px] = v;
  }
}

// Tiles whose halo lies inside the image take vector copies and no
// mirroring; border tiles mirror every coordinate.
template <int TH>
__device__ __forceinline__ bool EpfInterior(int w, int h, int x0, int y0) {
  return x0 >= 12 && x0 + kEpfW + 12 <= w && y0 >= 5 && y0 + TH + 5 <= h;
}

// Stages input rows y0 - 5 .. y0 + TH + 4, columns x0 - 12 .. x0 + 75 of
// the three planes into `tile` by asynchronous copies: 16 bytes each for
// interior tiles, 4 bytes per mirrored coordinate at the image border. The
// caller commits them and waits.
template <int TH, int NT>
__device__ __forceinline__ void EpfStage(const float* in, int w, int h, int x0,
                                         int y0,
                                         float (*tile)[TH + 10][kEpfTS],
                                         int tid) {
  constexpr int kTH = TH + 10, kThreads = NT;
  const size_t plane = size_t(w) * h;
  if (EpfInterior<TH>(w, h, x0, y0)) {
    constexpr int Q = kEpfTW / 4;
    for (int i = tid; i < 3 * kTH * Q; i += kThreads) {
      const int c = i / (kTH * Q);
      const int r = (i / Q) % kTH, q = i % Q;
      CpAsync16(&tile[c][r][4 * q],
                in + c * plane + size_t(y0 - 5 + r) * w + x0 - 12 + 4 * q);
    }
  } else {
    // A row per warp and turn; a lane's columns mirror once.
    const int lane = tid & 31;
    int gx[3];
#pragma unroll
    for (int i = 0; i < 3; ++i) gx[i] = MirrorIdx(x0 - 12 + lane + 32 * i, w);
    for (int cr = tid >> 5; cr < 3 * kTH; cr += kThreads / 32) {
      const int c = cr / kTH, r = cr - c * kTH;
      const float* row = in + c * plane + size_t(MirrorIdx(y0 - 5 + r, h)) * w;
#pragma unroll
      for (int i = 0; i < 3; ++i) {
        const int col = lane + 32 * i;
        if (col < kEpfTW) CpAsync4(&tile[c][r][col], row + gx[i]);
      }
    }
  }
}

// Builds the tile's u8 guide (MakeGuide, pik/epf_target.cc:1009-1070) in
// shared memory: the aligned words (bytes 4 wd .. 4 wd + 3 of a row) into
// `sa` (row-major, kEpfAligned words per channel and guide row), then one
// word per byte offset into `sg`. NT threads take part (this thread is `tid`
// of them), and `sync` is their barrier; the tile's copies are complete and
// published. Returns after the last barrier.
//
// The guide's position (gy, gx) is the tile's (gy - (y0 - 5), gx - (x0 - 12)),
// beyond the image's border too, where the tile holds the mirrored values:
// the smoothed value at a mirrored position has the same pairs of neighbours,
// and Sym3 adds each pair first.
template <int TH, int NT, typename Sync>
__device__ __forceinline__ void EpfBuildGuide(
    int tid, Sync sync, const uint8_t* guide_ovr, int gab, int w, int h,
    float amin, float mul, uint32_t* sg, uint32_t* sa,
    float (*tile)[TH + 10][kEpfTS], int x0, int y0) {
  constexpr int kGH = TH + 8;
  constexpr int kAligned = kEpfAligned;
  const float* gw = c_t.gaborish[gab];
  auto quant = [&](float v) {
    return uint32_t(uint8_t(uint32_t(__float2int_rz((v - amin) * mul))));
  };
  // The smoothed guide: each thread takes a vertical strip of kStrip words of
  // one channel and column, with its three input rows rolling down the strip,
  // so that each input row is loaded once and its pair sums v[i] + v[i + 2]
  // (Sym3's left/right and corner sums) are formed once for the three output
  // rows that use them. The arithmetic of each value is Sym3Rows', in its
  // order.
  constexpr int kStrip = (3 * kGH * kAligned + NT - 1) / NT;
  static_assert(kGH % kStrip == 0, "whole strips");
  constexpr int kStrips = kGH / kStrip;
  const bool strips = !guide_ovr && gab;
  if (strips && tid < 3 * kAligned * kStrips) {
    const int wd = tid % kAligned, c = (tid / kAligned) % 3;
    const int r0 = (tid / (3 * kAligned)) * kStrip;
    const int lx = 4 * wd + 4;
    float t[6], m[6], b[6], ht[4], hm[4], hb[4];
    auto load = [&](int r, float* v, float* hv) {
      const float* row = &tile[c][r][lx];
      const float4 q = *reinterpret_cast<const float4*>(row);
      v[0] = row[-1];
      v[1] = q.x, v[2] = q.y, v[3] = q.z, v[4] = q.w;
      v[5] = row[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) hv[i] = v[i] + v[i + 2];
    };
    load(r0, t, ht);
    load(r0 + 1, m, hm);
#pragma unroll
    for (int j = 0; j < kStrip; ++j) {
      load(r0 + j + 2, b, hb);
      uint32_t word = 0;
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const float sum_tb = t[i + 1] + b[i + 1];
        const float mul0 = m[i + 1] * gw[0];
        const float x1 = sum_tb + hm[i];
        const float mul1 = x1 * gw[1] + mul0;
        const float x2 = ht[i] + hb[i];
        word |= quant(x2 * gw[2] + mul1) << (8 * i);
      }
      sa[(c * kGH + r0 + j) * kAligned + wd] = word;
#pragma unroll
      for (int i = 0; i < 6; ++i) t[i] = m[i], m[i] = b[i];
#pragma unroll
      for (int i = 0; i < 4; ++i) ht[i] = hm[i], hm[i] = hb[i];
    }
  }
  for (int i = tid; i < 3 * kGH * kAligned && !strips; i += NT) {
    const int cr = i / kAligned, wd = i - cr * kAligned;
    const int c = cr / kGH, r = cr - c * kGH;
    uint32_t word = 0;
    if (guide_ovr) {
      const int gy = y0 - 4 + r;
      for (int b = 0; b < 4; ++b) {
        const int gx = x0 - 8 + 4 * wd + b;
        const bool ok = gx >= -6 && gx < w + 6 && gy >= -6 && gy < h + 6;
        const uint32_t v =
            ok ? guide_ovr[(size_t(c) * (h + 12) + gy + 6) * (w + 12) + gx + 6]
               : 0u;
        word |= v << (8 * b);
      }
    } else {
      const float4 q =
          *reinterpret_cast<const float4*>(&tile[c][r + 1][4 * wd + 4]);
      word = quant(q.x) | quant(q.y) << 8 | quant(q.z) << 16 |
             quant(q.w) << 24;
    }
    sa[i] = word;
  }
  sync();
  // The words of offsets 4 wd .. 4 wd + 3 from the two aligned neighbours
  // (bytes past the row end read as 0), one 16-byte store each.
  for (int i = tid; i < 3 * kGH * kAligned; i += NT) {
    const int cr = i / kAligned, wd = i - cr * kAligned;
    const uint32_t lo = sa[i];
    const uint32_t hi = wd + 1 < kAligned ? sa[i + 1] : 0u;
    *reinterpret_cast<uint4*>(sg + cr * kEpfGRow + 4 * wd) =
        make_uint4(lo, __funnelshift_r(lo, hi, 8), __funnelshift_r(lo, hi, 16),
                   __funnelshift_r(lo, hi, 24));
  }
  sync();
}

// Threads of a 64 x TH tile whose threads own R rows of a column each.
template <int TH, int R>
__host__ __device__ constexpr int EpfThreads() {
  return kEpfW * TH / R;
}

// Filters the tile from its staged input and guide, with `sig` the sigma of
// this thread's block, and stores the result. No CTA barrier.
template <bool kFma, int TH, int ROWS>
__device__ __forceinline__ void EpfFilterCore(
    int tid, int sig, float* out, float* sum_w, const EpfDc& dco, int w, int h,
    const uint32_t* sg, float (*tile)[TH + 10][kEpfTS], int x0, int y0) {
  constexpr int kGH = TH + 8;
  constexpr int kGPlane = kGH * kEpfGRow;
  const int lane = tid & 31, wp = tid >> 5;
  // The warp's rows and its first column (tile-local).
  const int row0 = ROWS * (wp >> 1), col0 = 32 * (wp & 1);
  const size_t plane = size_t(w) * h;
  const int px = x0 + lane + col0, py0 = y0 + row0;
  const bool inside = px < w && py0 < h;  // w and h are multiples of 8
  const bool filtered = sig >= kMinSigma;
  // Tile position of the pixel (px, py0).
  const int tr0 = row0 + 3 + kEpfTRow0, tc0 = lane + col0 + 3 + kEpfTCol0;

  // Warps (half a block row of 8 blocks) without filtered blocks copy.
  if (!__any_sync(0xFFFFFFFFu, filtered)) {
    if (inside) {
#pragma unroll
      for (int c = 0; c < 3; ++c)
#pragma unroll
        for (int j = 0; j < ROWS; ++j)
          EpfStore(out, dco, plane, w, c, px, py0 + j, tile[c][tr0 + j][tc0]);
    }
    return;
  }
  const int m64 = c_t.mul_table[filtered ? sig : kMinSigma] * 64;
  const EpfCut cut = EpfCutOf(filtered ? sig : kMinSigma, m64);

  // Centre patch rows: guide rows py0 - 1 .. py0 + ROWS, bytes px - 1 .. px + 2
  // (byte offset of px - 1 from x0 - 8).
  const int gr0 = row0 + 3;  // guide smem row of py0 - 1
  const int gc0 = lane + col0 + 7;
  float ws[3][ROWS], sw[ROWS];
#pragma unroll
  for (int j = 0; j < ROWS; ++j) {
    ws[0][j] = ws[1][j] = ws[2][j] = 0.f;
    sw[j] = 0.f;
  }
  if constexpr (kFma) {
    // Tensor-core forms: cx outermost. For one cx the 7 vertical offsets
    // read ROWS + 8 distinct guide rows per channel (one load each), and
    // each staged input row serves every pixel of the lane it reaches: for
    // eight rows about 120 shared-memory loads per cx and lane instead of
    // 378. Each pixel's sums run cx-major, not in the reference's cy-major
    // order (these forms are not bound to its rounding), two neighbouring
    // rows' at a time.
#pragma unroll 1
    for (int cx = -3; cx <= 4; ++cx) {
      const uint32_t* g = sg + (gr0 - 3) * kEpfGRow + gc0 + cx;
      uint32_t sad[7][ROWS];
#pragma unroll
      for (int c = 0; c < 3; ++c) {
        uint32_t wd[ROWS + 8];  // guide rows gr0 - 3 .. at this cx
#pragma unroll
        for (int t = 0; t < ROWS + 8; ++t) wd[t] = g[c * kGPlane + t * kEpfGRow];
        // The centre patch words again from shared memory (registers are
        // the limit).
        uint32_t rf[ROWS + 2];
#pragma unroll
        for (int r = 0; r < ROWS + 2; ++r) {
          rf[r] = sg[c * kGPlane + (gr0 + r) * kEpfGRow + gc0];
        }
#pragma unroll
        for (int k = 0; k < 7; ++k) {  // cy = k - 3: rows k ..
          if (c == 0) {
            PatchSads<true, ROWS>(rf, wd + k, sad[k]);
          } else {
            PatchSads<false, ROWS>(rf, wd + k, sad[k]);
          }
        }
      }
      float wt[ROWS][7];
#pragma unroll
      for (int j = 0; j < ROWS; ++j)
#pragma unroll
        for (int k = 0; k < 7; ++k) {
          const float wgt = EpfCutWeight(m64, cut, sad[k][j]);
          wt[j][k] = wgt;
          sw[j] += wgt;
        }
      // Input rows R - 3 (R = j + cy + 3) at column px + cx.
      const int col = tc0 + cx;
#pragma unroll
      for (int R = 0; R < ROWS + 6; ++R) {
        const int ir = tr0 - 3 + R;
        const float v0 = tile[0][ir][col], v1 = tile[1][ir][col],
                    v2 = tile[2][ir][col];
#pragma unroll
        for (int j = 0; j < ROWS; ++j) {
          const int k = R - j;  // cy + 3
          if (k < 0 || k > 6) continue;
          if (j % 2 == 0 && j + 1 < ROWS && k > 0) {
            Fma2(ws[0][j], ws[0][j + 1], v0, wt[j][k], wt[j + 1][k - 1]);
            Fma2(ws[1][j], ws[1][j + 1], v1, wt[j][k], wt[j + 1][k - 1]);
            Fma2(ws[2][j], ws[2][j + 1], v2, wt[j][k], wt[j + 1][k - 1]);
          } else if (j % 2 == 0 || k == 6) {  // no such pair
            ws[0][j] = fmaf(v0, wt[j][k], ws[0][j]);
            ws[1][j] = fmaf(v1, wt[j][k], ws[1][j]);
            ws[2][j] = fmaf(v2, wt[j][k], ws[2][j]);
          }
        }
      }
    }
  } else {
    // The reference's order: cy-major, products and sums rounded separately
    // (two rows' products in one instruction).
    uint32_t ref[3][ROWS + 2];
#pragma unroll
    for (int c = 0; c < 3; ++c)
#pragma unroll
      for (int r = 0; r < ROWS + 2; ++r)
        ref[c][r] = sg[c * kGPlane + (gr0 + r) * kEpfGRow + gc0];
#pragma unroll 1
    for (int cy = -3; cy <= 3; ++cy) {
#pragma unroll(ROWS > 2 ? 1 : 4)
      for (int cx = -3; cx <= 4; ++cx) {
        // Window byte offset: the patch start moved by cx.
        const uint32_t* g = sg + (gr0 + cy) * kEpfGRow + gc0 + cx;
        uint32_t sad[ROWS];
#pragma unroll
        for (int c = 0; c < 3; ++c) {
          uint32_t wd[ROWS + 2];
#pragma unroll
          for (int r = 0; r < ROWS + 2; ++r) wd[r] = g[c * kGPlane + r * kEpfGRow];
          if (c == 0) {
            PatchSads<true, ROWS>(ref[c], wd, sad);
          } else {
            PatchSads<false, ROWS>(ref[c], wd, sad);
          }
        }
        const int col = tc0 + cx;
        float wt[ROWS];
#pragma unroll
        for (int j = 0; j < ROWS; ++j) wt[j] = EpfCutWeight(m64, cut, sad[j]);
#pragma unroll
        for (int j = 0; j < ROWS; j += 2) {
          const int ir = tr0 + j + cy;
          if constexpr (ROWS == 1) {
#pragma unroll
            for (int c = 0; c < 3; ++c) ws[c][j] += tile[c][ir][col] * wt[j];
            sw[j] += wt[j];
          } else {
#pragma unroll
            for (int c = 0; c < 3; ++c) {
              float p0, p1;
              Mul2(p0, p1, tile[c][ir][col], tile[c][ir + 1][col], wt[j],
                   wt[j + 1]);
              ws[c][j] += p0;
              ws[c][j + 1] += p1;
            }
            Add2(sw[j], sw[j + 1], wt[j], wt[j + 1]);
          }
        }
      }
    }
  }
  if (!inside) return;
  if (sum_w) {
#pragma unroll
    for (int j = 0; j < ROWS; ++j) sum_w[size_t(py0 + j) * w + px] = sw[j];
  }
  // The normalisation: an IEEE division in the FP32 form (the reference's
  // rounding); in the tensor-core forms one reciprocal per row (the weight
  // sum is in [1, 56]) and a multiply per channel, within 2 ulp.
  float inv[ROWS];
#pragma unroll
  for (int j = 0; j < ROWS; ++j) inv[j] = kFma ? __frcp_rn(sw[j]) : 0.f;
#pragma unroll
  for (int c = 0; c < 3; ++c)
#pragma unroll
    for (int j = 0; j < ROWS; ++j) {
      const float v = kFma ? ws[c][j] * inv[j] : ws[c][j] / sw[j];
      EpfStore(out, dco, plane, w, c, px, py0 + j,
               filtered ? v : tile[c][tr0 + j][tc0]);
    }
}

// Filters the staged tile at (x0, y0) into `out` (or, for the DC image,
// into dco's clamp), with every thread of the CTA: the guide, then the
// filter. The tile's copies are complete in every thread (the first
// barrier below publishes them); `sig` is the sigma of this thread's block;
// (amin, mul) quantise the guide (GuideParams). `sa` holds the aligned
// guide words while the guide is built.
//
// kFma: the weighted sums with fused multiply-adds (the tensor-core forms,
// which are not bound to the reference's rounding); otherwise every product
// and sum is rounded separately, as the reference does.
template <bool kFma, int TH, int ROWS>
__device__ __forceinline__ void EpfFilterTile(
    const uint8_t* guide_ovr, int gab, int w, int h, float amin, float mul,
    int sig, float* out, float* sum_w, const EpfDc& dco, uint32_t* sg,
    uint32_t* sa, float (*tile)[TH + 10][kEpfTS], int x0, int y0) {
  const int tid = threadIdx.x;
  // Tiles without filtered blocks are copies (CopyOriginalBlock): every warp
  // copies, and no guide is needed.
  if (__syncthreads_or(sig >= kMinSigma)) {
    EpfBuildGuide<TH, EpfThreads<TH, ROWS>()>(tid, [] { __syncthreads(); },
                                              guide_ovr, gab, w, h, amin, mul,
                                              sg, sa, tile, x0, y0);
  }
  EpfFilterCore<kFma, TH, ROWS>(tid, sig, out, sum_w, dco, w, h, sg, tile, x0,
                                y0);
}

// One CTA per 64 x TH tile (1-D grid). More CTAs than resident slots balance
// the uneven tiles (copies, border tiles) better than CTAs that loop over
// tiles. kList: the tiles of the regions in the work list; the grid has a CTA
// for every tile that the list may hold, and those past its end leave at
// once. Against a CTA per tile that reads, and where nothing is filtered
// copies, every tile: 426 -> 76 us at 8192x8192 with 4% of the blocks
// filtered, 218 -> 188 at 4K with a third, and 402 -> 404 at 3001x2003 with
// all of them. CTAs that loop over the list's tiles took 105, 211 and 439: a
// new CTA's list entry and copy overlap the filtering of its neighbours.
//
// Interior tiles are staged by the Tensor Memory Accelerator when `tmap`
// is valid (use_tma): one thread issues a 3-D tiled bulk copy
// (cp.async.bulk.tensor, a tensor map over this GPU's input planes, no
// multicast) of the tile's rows y0 - 5 .. y0 + TH + 4, columns
// x0 - 12 .. x0 + 75 of the three planes, straight into `tile` (whose
// layout is the copy's box), completing on an mbarrier with the byte count.
// The innermost coordinate x0 - 12 is a multiple of 4 floats (x0 is a
// multiple of 64), as the copy requires. The wait is bounded (`polls`, the
// context's PIKGPU_OPT_TC_WAIT_POLLS): if it runs out, the kernel sets
// *err = 2 (the host reports the frame as failed) and waits once more,
// bounded, so that no copy is in flight when the CTA exits. Border tiles,
// and all tiles without a tensor map, are staged with cp.async (EpfStage).
template <bool kFma, int TH, int ROWS, bool kList>
__global__ void __launch_bounds__(EpfThreads<TH, ROWS>(),
                                  ROWS < 8 ? 2 : kFma ? 3 : 4)
    k_epf_box(const float* in, const uint8_t* guide_ovr, int gab, int w, int h,
              const uint32_t* mm, EpfWork work, float* out, EpfDc dco,
              const __grid_constant__ CUtensorMap tmap, int use_tma,
              int* err, uint32_t polls) {
  extern __shared__ __align__(128) uint32_t epf_smem[];
  uint32_t* sg = epf_smem;  // [3][TH + 8][kEpfGRow]
  auto* tile = reinterpret_cast<float(*)[TH + 10][kEpfTS]>(
      epf_smem + 3 * (TH + 8) * kEpfGRow);
  uint32_t* sa = epf_smem + 3 * (TH + 8) * kEpfGRow + 3 * (TH + 10) * kEpfTS;
  uint64_t* mbar = reinterpret_cast<uint64_t*>(sa + 3 * (TH + 8) * kEpfAligned);
  PdlLaunchDependents();
  const int tiles_x = (w + kEpfW - 1) / kEpfW;
  const uint32_t tile_s = tc::SmemU32(tile), mbar_s = tc::SmemU32(mbar);
  const int tid = threadIdx.x, lane = tid & 31;
  int x0, y0;
  if (kList) {
    constexpr int kSub = kEpfRegionH / TH;  // tiles per region
    PdlWait();  // the list is the output of the kernel before this one
    const int region = int(work.list[blockIdx.x / kSub]);
    if (int(blockIdx.x) >= *work.count * kSub) return;
    x0 = (region % tiles_x) * kEpfW;
    y0 = (region / tiles_x) * kEpfRegionH + (blockIdx.x % kSub) * TH;
    if (y0 >= h) return;
  } else {
    x0 = (blockIdx.x % tiles_x) * kEpfW;
    y0 = (blockIdx.x / tiles_x) * TH;
  }
  const bool tma = use_tma && EpfInterior<TH>(w, h, x0, y0) &&
                   (tile_s & 127u) == 0;
  if (tma) {
    if (tid == 0) {
      asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(mbar_s)
                   : "memory");
      asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
      asm volatile(
          "mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(
              mbar_s),
          "r"(EpfTileBytes(TH))
          : "memory");
      asm volatile(
          "cp.async.bulk.tensor.3d.shared::cluster.global.tile.mbarrier::"
          "complete_tx::bytes [%0], [%1, {%2, %3, %4}], [%5];" ::"r"(tile_s),
          "l"(reinterpret_cast<uint64_t>(&tmap)), "r"(x0 - 12), "r"(y0 - 5),
          "r"(0), "r"(mbar_s)
          : "memory");
    }
  } else {
    EpfStage<TH, EpfThreads<TH, ROWS>()>(in, w, h, x0, y0, tile, tid);
  }
  float amin, mul, stretch;
  GuideParams(mm, &amin, &mul, &stretch);
  int sig = 0;
  const int px = x0 + lane + 32 * ((tid >> 5) & 1);
  const int py = y0 + ROWS * (tid >> 6);
  if (px < w && py < h) {
    sig = kList ? work.sigma[(py >> 3) * (w / 8) + (px >> 3)]
                : ScaledSigma(UnscaledSigma(float(work.dc_qf), 1.0f, 0),
                              stretch);
  }
  if (tma) {
    __syncthreads();  // the mbarrier is initialised before anyone waits
    // (tc::WaitMma is the bounded mbarrier wait of the tensor-core kernels)
    if (!tc::WaitMma(mbar_s, 0, polls) && tid == 0) {
      tc::ReportTimeout(err, 2);
    }
  } else {
    CpAsyncWaitAll();
  }
  EpfFilterTile<kFma, TH, ROWS>(guide_ovr, gab, w, h, amin, mul, sig, out,
                                kList ? work.sum_w : nullptr, dco, sg, sa,
                                tile, x0, y0);
}

}  // namespace pikgpu
