// Adjoint of the reconstruction (pikgpu_adjoint): the gradient of
//   L = sum over the xsize x ysize pixels and X, Y, B of
//       (pre_opsin - target)^2
// with respect to the dequantised AC coefficients (the output of
// Dequant::DoAC, pik/compressed_image.cc:586-707, frame layout) and the
// per-cell quant field taken as a real number. pre_opsin is the frame after
// gaborish #2, before OpsinToLinear (pik/compressed_image.cc:1144-1181).
//
// The EPF's discrete decisions -- the u8 guide and the per-block sigma of
// MakeGuide / SigmaFromQuant (pik/epf_target.cc:1009-1111) -- are piecewise
// constant in every input, so they are held at their forward values (their
// derivative is zero almost everywhere). With them fixed the reconstruction
// is linear in the coefficients except for AdaptiveReconstruction's clamp
// (pik/adaptive_reconstruction.cc:72-244), whose ratio
// (interval / 2) / |correction| is differentiated where it is active. The
// quant field enters through the dequantisation (a cell's coefficients
// scale with 1 / qf) and the clamp intervals (half a step, also 1 / qf).
//
// The forward pass runs first (LaunchAll, keeping the dequantised AC, the
// EPF output and pre_opsin); the backward pass then transposes each stage:
//   k_adj_loss      2 (pre - target) on the padded frame, loss partials
//   k_adj_gab       gaborish #2 transposed (mirrored stencil, gathered)
//   k_adj_ar*       the clamp, per first block: DCT of (EPF - IDCT) again,
//                   the branch of every coefficient from the clamp tape the
//                   forward's clamp kernels wrote (which channel set the
//                   minimum ratio, or none, or a +0.0 correction), the
//                   gradients of the correction and of the quant field
//   k_adj_epf*      the EPF with frozen weights: every pixel gathers the
//                   normalised weights of its filtered neighbours, and the
//                   border pixels' mirrored terms are scattered
//   k_adj_topix*    TransformToPixels transposed per first block, and for HF
//                   prediction TransformFromPixels transposed of the masked
//                   coefficient gradient (the upsampled prediction's
//                   gradient)
//   k_adj_upsample  UpSample4x4BlurDCT transposed into the group's pred2x2
//   k_adj_lf        DC2x2FromLowFrequencies transposed into each block's LF
//                   corner (pik/ac_predictions.cc:560-635); LLF gets zero
//                   (it is overwritten from DC)
//   k_adj_qf        the quant field: -sum(g * ac) / qf per cell
// Square DCT blocks use the separable transforms with transposed matrices;
// the other 8x8 types use dense 64 x 64 Jacobians built on the device from
// the forward transforms applied to unit vectors (k_adj_build_jac). The
// backward arithmetic is FP32 (sums of the quant
// field gradient and the loss in FP64).
//
// Included by pikgpu.cu (single translation unit).

namespace pikgpu {
namespace {

constexpr int kJTypes = 4;  // IDENTITY, DCT2X2, DCT4X4, LINES

__host__ __device__ inline int JIndex(int type) {
  switch (type) {
    case kDCT2X2:
      return 1;
    case kDCT4X4:
    case kDCT4X4_NOHF:
      return 2;
    case kLINES:
      return 3;
  }
  return 0;  // kIDENTITY
}

struct AdjJac {
  float j0[kJTypes][64][64];   // TransformToPixels, [pixel][coefficient]
  float j1[kJTypes][64][64];   // TransformFromPixels, [coefficient][pixel]
  float j1t[kJTypes][64][64];  // j1 transposed, [pixel][coefficient]
  float j2[9][64][64];         // DC2x2 of the LF corner, [cell][LF input]
};

// TransformToPixels of one of the kJTypes (AcStrategy::TransformToPixels,
// pik/ac_strategy.cc:741-849): coefficients and pixels 8x8 row-major.
__device__ void ToPixels8(int type, const float* co, float* px) {
  if (type == kDCT4X4 || type == kDCT4X4_NOHF) {
    const float b00 = co[0], b01 = co[1], b10 = co[8], b11 = co[9];
    const float d[4] = {b00 + b01 + b10 + b11, b00 + b01 - b10 - b11,
                        b00 - b01 + b10 - b11, b00 - b01 - b10 + b11};
    for (int sy = 0; sy < 2; ++sy) {
      for (int sx = 0; sx < 2; ++sx) {
        float in4[16], out4[16];
        for (int iy = 0; iy < 4; ++iy)
          for (int ix = 0; ix < 4; ++ix)
            in4[iy * 4 + ix] = (iy == 0 && ix == 0)
                                   ? d[sy * 2 + sx]
                                   : co[(sy + iy * 2) * 8 + sx + ix * 2];
        TsIdct1(4, in4, 4, out4, 4);
        for (int py = 0; py < 4; ++py)
          for (int q = 0; q < 4; ++q)
            px[(sy * 4 + py) * 8 + sx * 4 + q] = out4[py * 4 + q];
      }
    }
  } else {
    SmallInverse(type, co, px, 8);
  }
}

// TransformFromPixels of one of the kJTypes (pik/ac_strategy.cc:531-663).
__device__ void FromPixels8(int type, const float* px, float* co) {
  if (type == kDCT4X4 || type == kDCT4X4_NOHF) {
    for (int sy = 0; sy < 2; ++sy) {
      for (int sx = 0; sx < 2; ++sx) {
        float in4[16], r4[16];
        for (int py = 0; py < 4; ++py)
          for (int q = 0; q < 4; ++q)
            in4[py * 4 + q] = px[(sy * 4 + py) * 8 + sx * 4 + q];
        TsDct1(4, in4, 4, r4, 4);
        for (int iy = 0; iy < 4; ++iy)
          for (int ix = 0; ix < 4; ++ix)
            co[(sy + iy * 2) * 8 + sx + ix * 2] = r4[iy * 4 + ix];
      }
    }
    const float b00 = co[0], b01 = co[1], b10 = co[8], b11 = co[9];
    co[0] = (b00 + b01 + b10 + b11) * 0.25f;
    co[1] = (b00 + b01 - b10 - b11) * 0.25f;
    co[8] = (b00 - b01 + b10 - b11) * 0.25f;
    co[9] = (b00 - b01 - b10 + b11) * 0.25f;
  } else {
    SmallForward(type, px, 8, co);
  }
}

// Block 2 kJTypes + 9 CTAs of 64 threads; thread j builds column j.
__global__ void k_adj_build_jac(AdjJac* J) {
  const int which = blockIdx.x, j = threadIdx.x;
  const int kTypes[kJTypes] = {kIDENTITY, kDCT2X2, kDCT4X4, kLINES};
  float in[64], out[64];
  for (int i = 0; i < 64; ++i) {
    in[i] = i == j ? 1.0f : 0.0f;
    out[i] = 0.0f;
  }
  if (which < kJTypes) {
    ToPixels8(kTypes[which], in, out);
    for (int r = 0; r < 64; ++r) J->j0[which][r][j] = out[r];
  } else if (which < 2 * kJTypes) {
    const int t = which - kJTypes;
    FromPixels8(kTypes[t], in, out);
    for (int r = 0; r < 64; ++r) {
      J->j1[t][r][j] = out[r];
      J->j1t[t][j][r] = out[r];
    }
  } else {
    const int type = which - 2 * kJTypes;
    const int cov = Covered(type), n = 8 * cov, m = 2 * cov;
    if (j < m * m) {
      const int idx = (j / m) * n + j % m;
      DC2x2FromLowFreq(type, [&](int i) { return i == idx ? 1.0f : 0.0f; },
                       out, m);
    }
    for (int r = 0; r < 64; ++r) {
      J->j2[type][r][j] = (j < m * m && r < m * m) ? out[r] : 0.0f;
    }
  }
}

constexpr int kAdjLossBlocks = 592, kAdjThreads = 256;

// g_pre = 2 (pre - target) inside xsize x ysize, 0 in the padding; the loss
// partial sums of each CTA in FP64. A warp per 256 columns of a row and turn,
// eight loads of each plane in flight per lane (a flat index divided into
// plane, row and column, with one, took 22 us at 1024x1024, this 8).
constexpr int kAdjLossCols = 256;
__global__ void __launch_bounds__(kAdjThreads)
    k_adj_loss(const float* pre, const float* target, int w, int h, int pw,
               int ph, float* g_pre, double* partial) {
  __shared__ double s_sum[kAdjThreads / 32];
  const int lane = threadIdx.x & 31;
  const int warps = gridDim.x * (kAdjThreads / 32);
  double acc = 0.0;
  const int segs = (pw + kAdjLossCols - 1) / kAdjLossCols;
  for (int i = blockIdx.x * (kAdjThreads / 32) + (threadIdx.x >> 5);
       i < 3 * ph * segs; i += warps) {
    const int cy = i / segs, x0 = (i - cy * segs) * kAdjLossCols + lane;
    const int c = cy / ph, y = cy - c * ph;
    const size_t in = (size_t(c) * h + y) * w;
    const int n = y < h ? w : 0;
    float a[kAdjLossCols / 32], b[kAdjLossCols / 32];
#pragma unroll
    for (int k = 0; k < kAdjLossCols / 32; ++k) {
      const int x = x0 + 32 * k;
      a[k] = x < n ? pre[in + x] : 0.0f;
      b[k] = x < n ? target[in + x] : 0.0f;
    }
#pragma unroll
    for (int k = 0; k < kAdjLossCols / 32; ++k) {
      const int x = x0 + 32 * k;
      const double d = double(a[k]) - double(b[k]);
      acc += d * d;
      if (x < pw) g_pre[size_t(cy) * pw + x] = 2.0f * (a[k] - b[k]);
    }
  }
  for (int off = 16; off; off >>= 1) acc += __shfl_xor_sync(~0u, acc, off);
  if (lane == 0) s_sum[threadIdx.x >> 5] = acc;
  __syncthreads();
  if (threadIdx.x == 0) {
    double t = 0.0;
    for (int i = 0; i < kAdjThreads / 32; ++i) t += s_sum[i];
    partial[blockIdx.x] = t;
  }
}

// One warp (a single thread's chain of dependent adds took 17 us).
__global__ void k_adj_sum(const double* partial, int n, double* out) {
  double t = 0.0;
  for (int i = threadIdx.x; i < n; i += 32) t += partial[i];
  for (int off = 16; off; off >>= 1) t += __shfl_xor_sync(~0u, t, off);
  if (threadIdx.x == 0) *out = t;
}

// Transpose of Symmetric3 with mirrored borders: the stencil again, since
// it is symmetric with its mirrored taps too (a border pixel's tap beyond the
// frame reads that pixel's own row or column, -1 -> 0, at the same distance
// as the tap that reads it). Four columns of a row per thread (pw is a
// multiple of 8): 18 us at 1024x1024 with a pixel per thread, now 6.5.
__global__ void __launch_bounds__(kAdjThreads)
    k_adj_gab(const float* gin, int pw, int ph, int strength, float* gout) {
  const int x0 = 4 * (blockIdx.x * blockDim.x + threadIdx.x);
  const int y = blockIdx.y * blockDim.y + threadIdx.y;
  const int c = blockIdx.z;
  if (x0 >= pw || y >= ph) return;
  const float* wt = c_t.gaborish[strength];
  const float* p = gin + size_t(c) * pw * ph;
  float v[3][6], s[4];
#pragma unroll
  for (int r = 0; r < 3; ++r) {
    const float* row = p + size_t(MirrorIdx(y - 1 + r, ph)) * pw;
    const float4 q = *reinterpret_cast<const float4*>(row + x0);
    v[r][0] = row[max(x0 - 1, 0)];
    v[r][1] = q.x, v[r][2] = q.y, v[r][3] = q.z, v[r][4] = q.w;
    v[r][5] = row[min(x0 + 4, pw - 1)];
  }
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    s[i] = v[1][i + 1] * wt[0] +
           (v[0][i + 1] + v[2][i + 1] + v[1][i] + v[1][i + 2]) * wt[1] +
           (v[0][i] + v[0][i + 2] + v[2][i] + v[2][i + 2]) * wt[2];
  }
  *reinterpret_cast<float4*>(gout + size_t(c) * pw * ph + size_t(y) * pw +
                             x0) = make_float4(s[0], s[1], s[2], s[3]);
}

// Clamp backward of one coefficient, on the branch the forward took (its
// clamp tape code, ClampTapeCode). co: the correction per channel, iv: the
// interval, gs: the gradient of the scaled correction. Writes the
// correction gradient; for a clamped non-LLF coefficient adds the quant
// field's share to *gq: the ratio is (interval / 2) / |co| and
// d interval / d qf = -interval / qf.
__device__ __forceinline__ void ClampBackward(int code, const float co[3],
                                              const float iv[3],
                                              const float gs[3], bool llf,
                                              float qf_eff, float gc[3],
                                              float* gq) {
  const int arg = code >= 1 && code <= 3 ? code - 1 : -1;
  const float mr =
      arg >= 0 ? ClampRatio(co[arg], iv[arg]) : code == 0 ? 1.0f : 0.0f;
  float gmr = 0.0f;
#pragma unroll
  for (int c = 0; c < 3; ++c) {
    gmr += gs[c] * co[c];
    gc[c] = gs[c] * mr;
  }
  if (arg >= 0 && co[arg] != 0.0f) {
    gc[arg] += gmr * (-mr / co[arg]);
    if (!llf) *gq += -gmr * mr / qf_eff;
  }
}

__device__ __forceinline__ float QfEff(const Geo& g, const DevFrame& f,
                                       int bx, int by) {
  const int cell = by * g.Bx + bx;
  const float q = float(f.qf[cell]);
  return f.clamp_scale ? q / f.clamp_scale[cell] : q;
}

// Column e of a 64 x 64 matrix times the three channels' vectors in shared
// memory: one matrix value serves the channels, 16-byte reads four of them.
// 32 matrix values are in flight at a time (few frames have enough of these
// blocks to fill the chip: what they cost is the loads' latency).
__device__ __forceinline__ void DenseCols(const float (*m)[64], int e,
                                          const float (*v)[64], float o[3]) {
  o[0] = o[1] = o[2] = 0.0f;
#pragma unroll 8
  for (int p = 0; p < 64; p += 4) {
    const float m0 = m[p][e], m1 = m[p + 1][e], m2 = m[p + 2][e],
                m3 = m[p + 3][e];
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      const float4 q = *reinterpret_cast<const float4*>(&v[c][p]);
      o[c] = fmaf(m0, q.x, o[c]);
      o[c] = fmaf(m1, q.y, o[c]);
      o[c] = fmaf(m2, q.z, o[c]);
      o[c] = fmaf(m3, q.w, o[c]);
    }
  }
}

// The 8x8 types without a separable transform (DCT4X4 and the small ones):
// two launches of 23 and 23 us at 1024x1024, one per class and with a channel
// after the other, now 19.
constexpr int kAdj8Blocks = 4;  // 8x8 blocks per CTA, 64 threads each
struct Adj8Lists {
  const uint32_t* list[2];
  int count[2];
  __device__ uint32_t At(int i) const {
    return i < count[0] ? list[0][i] : list[1][i - count[0]];
  }
};

// Clamp backward of 8x8 blocks of the types in Adj8Lists from the dense
// Jacobians. Blocks the EPF left unfiltered have EPF output == IDCT output,
// a zero correction and ratio 0: the gradient passes to the IDCT output.
__global__ void __launch_bounds__(kAdjThreads)
    k_adj_ar8(Geo g, DevFrame f, FrameScalars s, const AdjJac* J,
              Adj8Lists lists, const int32_t* sigma, const uint8_t* tape,
              const float* epf, const float* sum_w, const float* g_cur,
              float* g_filt, float* g_idct, float* g_qf) {
  // The difference, then g_corr; the gradient of the output.
  __shared__ __align__(16) float s_a[kAdj8Blocks][3][64];
  __shared__ __align__(16) float s_o[kAdj8Blocks][3][64];
  __shared__ float s_q[kAdj8Blocks][2];
  const int lb = threadIdx.x >> 6, e = threadIdx.x & 63;
  const int item = blockIdx.x * kAdj8Blocks + lb;
  const bool valid = item < lists.count[0] + lists.count[1];
  int bx = 0, by = 0, type = 0;
  bool active = false;
  if (valid) {
    const uint32_t pk = lists.At(item);
    bx = pk & 0xFFFF;
    by = pk >> 16;
    type = f.acs[by * g.Bx + bx] >> 4;
    active = sigma[by * g.Bx + bx] >= kMinSigma;
  }
  const size_t plane = size_t(g.PW) * g.PH;
  const size_t o = size_t(by * 8 + e / 8) * g.PW + bx * 8 + e % 8;
  if (valid) {
    for (int c = 0; c < 3; ++c) {
      s_o[lb][c][e] = g_cur[c * plane + o];
      s_a[lb][c][e] =
          active ? epf[c * plane + o] - f.idct[c * plane + o] : 0.0f;
    }
  }
  __syncthreads();
  const int t = JIndex(type);
  float gq = 0.0f, gc[3] = {0.0f, 0.0f, 0.0f};
  if (valid && active) {
    float co[3], gs[3], iv[3];
    DenseCols(J->j1t[t], e, s_a[lb], co);
    DenseCols(J->j0[t], e, s_o[lb], gs);
    const ArBlockInfo info = ArInfo(g, f, s, bx, by, type);
    for (int c = 0; c < 3; ++c) {
      iv[c] = e == 0 ? 1.0f * s.mul_dc[c] : info.dm[c][e] * info.inv_quant_ac;
    }
    ClampBackward(tape[CoefOffset(g, bx, by, 1, e)], co, iv, gs, e == 0,
                  QfEff(g, f, bx, by), gc, &gq);
  }
  __syncthreads();
  if (valid && active) {
    for (int c = 0; c < 3; ++c) s_a[lb][c][e] = gc[c];
  }
  for (int off = 16; off; off >>= 1) gq += __shfl_xor_sync(~0u, gq, off);
  if ((threadIdx.x & 31) == 0) s_q[lb][(threadIdx.x >> 5) & 1] = gq;
  __syncthreads();
  if (!valid) return;
  if (e == 0 && active) g_qf[by * g.Bx + bx] = s_q[lb][0] + s_q[lb][1];
  float gd[3] = {0.0f, 0.0f, 0.0f};
  if (active) DenseCols(J->j1[t], e, s_a[lb], gd);
  const float sw = active ? sum_w[o] : 1.0f;
  for (int c = 0; c < 3; ++c) {
    g_filt[c * plane + o] = gd[c] / sw;
    g_idct[c * plane + o] = s_o[lb][c][e] - gd[c];
  }
}

// Square-DCT matrices staged in shared memory for the transposed-matrix
// transforms (CoopTsIdctT / CoopTsDctT, which take M^T to apply M): `a` =
// A (applies A^T, the transpose of the IDCT), `b` = B (applies B^T, the
// transpose of the scaled DCT), `bt` = B^T (applies B, the DCT).
template <int N>
__device__ __forceinline__ void StageMatrices(float* a, float* b, float* bt) {
  for (int i = threadIdx.x; i < N * N; i += blockDim.x) {
    const int r = i / N, c = i % N;
    a[i] = IdctMat(N)[i];
    b[i] = DctMat(N)[i];
    if (bt) bt[i] = DctMat(N)[c * N + r];
  }
}

// Clamp backward of one DCT16 / DCT32 block per CTA (separable transforms:
// the transpose of the IDCT is the IDCT routine with A^T, that of the
// scaled DCT the DCT routine with B^T).
template <int N>
__global__ void __launch_bounds__(kAdjThreads)
    k_adj_ar_sq(Geo g, DevFrame f, FrameScalars s, const uint32_t* list,
                int count, const int32_t* sigma, const uint8_t* tape,
                const float* epf, const float* sum_w, const float* g_cur,
                float* g_filt, float* g_idct, float* g_qf) {
  constexpr int NN = N * N, cov = N / 8;
  __shared__ float s_b[NN], s_a[NN], s_bt[NN];
  __shared__ float s_co[3][NN], s_g[3][NN], s_t[NN];
  __shared__ float s_q[kAdjThreads / 32];
  const int item = blockIdx.x;
  if (item >= count) return;
  const uint32_t pk = list[item];
  const int bx = pk & 0xFFFF, by = pk >> 16;
  const int type = f.acs[by * g.Bx + bx] >> 4;
  bool active = false;
  for (int y = 0; y < cov; ++y)
    for (int x = 0; x < cov; ++x)
      active |= sigma[(by + y) * g.Bx + bx + x] >= kMinSigma;
  const size_t plane = size_t(g.PW) * g.PH;
  auto pix = [&](int c, int e) {
    return c * plane + size_t(by * 8 + e / N) * g.PW + bx * 8 + e % N;
  };
  if (!active) {  // CTA-uniform
    for (int i = threadIdx.x; i < 3 * NN; i += blockDim.x) {
      const size_t o = pix(i / NN, i % NN);
      g_idct[o] = g_cur[o];
      g_filt[o] = 0.0f;
    }
    return;
  }
  StageMatrices<N>(s_a, s_b, s_bt);
  for (int i = threadIdx.x; i < 3 * NN; i += blockDim.x) {
    const int c = i / NN, e = i % NN;
    const size_t o = pix(c, e);
    s_co[c][e] = epf[o] - f.idct[o];
    s_g[c][e] = g_cur[o];
  }
  __syncthreads();
  for (int c = 0; c < 3; ++c) {
    CoopTsDctT(N, 1, s_bt, s_co[c], s_t, s_co[c]);   // B
    CoopTsIdctT(N, 1, s_a, s_g[c], s_t, s_g[c]);    // A^T
  }
  const ArBlockInfo info = ArInfo(g, f, s, bx, by, type);
  const float qf_eff = QfEff(g, f, bx, by);
  float gq = 0.0f;
  for (int e = threadIdx.x; e < NN; e += blockDim.x) {
    const int y = e / N, x = e % N;
    const bool llf = y < cov && x < cov;
    float co[3], gs[3], iv[3], gc[3];
    for (int c = 0; c < 3; ++c) {
      co[c] = s_co[c][e];
      gs[c] = s_g[c][e];
      iv[c] = llf ? LlfScale(type, x, y) * s.mul_dc[c]
                  : info.dm[c][e] * info.inv_quant_ac;
    }
    ClampBackward(tape[CoefOffset(g, bx, by, cov, e)], co, iv, gs, llf,
                  qf_eff, gc, &gq);
    for (int c = 0; c < 3; ++c) s_g[c][e] = gc[c];
  }
  __syncthreads();
  for (int c = 0; c < 3; ++c) {
    CoopTsDctT(N, 1, s_b, s_g[c], s_t, s_g[c]);  // B^T
  }
  for (int i = threadIdx.x; i < 3 * NN; i += blockDim.x) {
    const int c = i / NN, e = i % NN;
    const size_t o = pix(c, e);
    const float gd = s_g[c][e];
    const int x = bx * 8 + e % N, y = by * 8 + e / N;
    const bool filtered = sigma[(y >> 3) * g.Bx + (x >> 3)] >= kMinSigma;
    g_filt[o] = filtered ? gd / sum_w[size_t(y) * g.PW + x] : gd;
    g_idct[o] = g_cur[o] - gd;
  }
  for (int off = 16; off; off >>= 1) gq += __shfl_xor_sync(~0u, gq, off);
  if ((threadIdx.x & 31) == 0) s_q[threadIdx.x >> 5] = gq;
  __syncthreads();
  if (threadIdx.x == 0) {
    float t = 0.0f;
    for (int i = 0; i < kAdjThreads / 32; ++i) t += s_q[i];
    g_qf[by * g.Bx + bx] = t;
  }
}

// A row times one of the transform matrices M (the inverse's A, or the
// forward's B): o[k] = sum_i M[k][i] v[i], or with kT sum_i M[i][k] v[i].
template <int N, bool kInverse, bool kT>
__device__ __forceinline__ void MatRow(const float (&v)[N], float (&o)[N]) {
#pragma unroll
  for (int k = 0; k < N; ++k) {
    float a = 0.0f;
#pragma unroll
    for (int i = 0; i < N; ++i) {
      const int at = MatOffset(N) + (kT ? i * N + k : k * N + i);
      a = fmaf(v[i], kInverse ? c_t.idct[at] : c_t.dct[at], a);
    }
    o[k] = a;
  }
}

// The same for 8x8 DCT blocks, by rows in registers: a warp per channel of
// four blocks, the element-wise step on the three channels' coefficients in
// shared memory. With the dense Jacobians of k_adj_ar8 the 8x8 DCT blocks of
// a 1024x1024 frame took 17 us, now 9. (16x16 blocks by the same split, at that size:
// 44 us against 41 for k_adj_ar_sq, which has more warps per block.)
__global__ void __launch_bounds__(kSquareArThreads)
    k_adj_ar_dct8(Geo g, DevFrame f, FrameScalars s, const uint32_t* list,
               int count, const int32_t* sigma, const uint8_t* tape,
               const float* epf, const float* sum_w, const float* g_cur,
               float* g_filt, float* g_idct, float* g_qf) {
  using namespace square;
  constexpr int N = 8, cov = 1, UPW = 32 / N, tile_size = N * (N + 1);
  __shared__ float s_co[kSquareArGroups][UPW][3][tile_size];
  __shared__ float s_g[kSquareArGroups][UPW][3][tile_size];
  __shared__ float s_q[kSquareArGroups][UPW][3];
  constexpr float scale = 1.0f / float(N * N);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int c = warp % 3, grp = warp / 3;
  const int unit = lane / N, r = lane % N;
  const int item = (blockIdx.x * kSquareArGroups + grp) * UPW + unit;
  const bool valid = item < count;
  const uint32_t pk = list[valid ? item : 0];
  const int bx = pk & 0xFFFF, by = pk >> 16;
  const int type = f.acs[by * g.Bx + bx] >> 4;
  const bool active = sigma[by * g.Bx + bx] >= kMinSigma;
  const size_t row = c * size_t(g.PW) * g.PH + size_t(by * 8 + r) * g.PW +
                     bx * 8;
  float G[N], D[N], T[N];
#pragma unroll
  for (int x = 0; x < N; x += 4) {
    const float4 a = *reinterpret_cast<const float4*>(epf + row + x);
    const float4 o = *reinterpret_cast<const float4*>(f.idct + row + x);
    const float4 q = *reinterpret_cast<const float4*>(g_cur + row + x);
    D[x] = a.x - o.x, D[x + 1] = a.y - o.y;
    D[x + 2] = a.z - o.z, D[x + 3] = a.w - o.w;
    G[x] = q.x, G[x + 1] = q.y, G[x + 2] = q.z, G[x + 3] = q.w;
  }
  float* tco = s_co[grp][unit][c];
  float* tg = s_g[grp][unit][c];
  MatRow<N, false, false>(D, T);  // the correction's coefficients
  PutCol<N>(tco, r, T);
  MatRow<N, true, true>(G, T);  // the gradient of the scaled correction
  PutRow<N>(tg, r, T);
  __syncwarp();
  GetRow<N>(tco, r, D);
  MatRow<N, false, false>(D, T);
#pragma unroll
  for (int x = 0; x < N; ++x) T[x] *= scale;
  __syncwarp();
  PutRow<N>(tco, r, T);
  GetCol<N>(tg, r, D);
  MatRow<N, true, true>(D, T);
  __syncwarp();
  PutRow<N>(tg, r, T);
  __syncthreads();
  // A block's 24 lanes share its 64 coefficients.
  const ArBlockInfo info = ArInfo(g, f, s, bx, by, type);
  const float qf_eff = QfEff(g, f, bx, by);
  float gq = 0.0f;
  for (int e = c * N + r; e < N * N && valid && active; e += 3 * N) {
    const int y = e / N, x = e % N, at = y * (N + 1) + x;
    const bool llf = e == 0;
    float co[3], gs[3], iv[3], gc[3];
#pragma unroll
    for (int k = 0; k < 3; ++k) {
      co[k] = s_co[grp][unit][k][at];
      gs[k] = s_g[grp][unit][k][at];
      iv[k] = llf ? s.mul_dc[k]
                  : info.dm[k][e] * info.inv_quant_ac;
    }
    ClampBackward(tape[CoefOffset(g, bx, by, cov, e)], co, iv, gs, llf,
                  qf_eff, gc, &gq);
#pragma unroll
    for (int k = 0; k < 3; ++k) s_g[grp][unit][k][at] = gc[k];
  }
  for (int off = N / 2; off; off >>= 1) {
    gq += __shfl_xor_sync(~0u, gq, off);
  }
  if (r == 0) s_q[grp][unit][c] = gq;
  __syncthreads();
  GetRow<N>(tg, r, D);
  MatRow<N, false, true>(D, T);
  __syncwarp();
  PutCol<N>(tg, r, T);
  __syncwarp();
  GetRow<N>(tg, r, D);
  MatRow<N, false, true>(D, T);
  if (!valid) return;
#pragma unroll
  for (int x = 0; x < N; ++x) T[x] = active ? T[x] * scale : 0.0f;
#pragma unroll
  for (int x = 0; x < N; x += 4) {
    const float4 q = *reinterpret_cast<const float4*>(g_cur + row + x);
    float4 sw = make_float4(1.0f, 1.0f, 1.0f, 1.0f);
    if (active) {
      sw = *reinterpret_cast<const float4*>(
          sum_w + size_t(by * 8 + r) * g.PW + bx * 8 + x);
    }
    *reinterpret_cast<float4*>(g_filt + row + x) = make_float4(
        T[x] / sw.x, T[x + 1] / sw.y, T[x + 2] / sw.z, T[x + 3] / sw.w);
    *reinterpret_cast<float4*>(g_idct + row + x) =
        make_float4(q.x - T[x], q.y - T[x + 1], q.z - T[x + 2],
                    q.w - T[x + 3]);
  }
  if (active && c == 0 && r == 0) {
    const float* q = s_q[grp][unit];
    g_qf[by * g.Bx + bx] = q[0] + q[1] + q[2];
  }
}

// EPF with frozen weights, transposed. The forward pass computes, for a
// filtered pixel p, out(p) = sum_d w(p, d) in(p + d) / sum_d w(p, d) over
// the 7 x 8 window d = (cx, cy), cx in [-3, 4], cy in [-3, 3], where
// w(p, d) = W(mul(p), SAD(p, p + d)) and in() is mirrored at the frame
// border. Its transpose sends gv(p) w(p, d), gv(p) = g(p) / sum_w(p), to
// p + d; the sums are the forward pass's. g_filt holds gv for filtered pixels
// (the clamp's backward kernels divide) and g(p) itself for copied ones. The
// patch SAD is symmetric, SAD(p, p + d) = SAD(q, q - d) for q = p + d, so the
// transpose is a gather at q over the mirrored window e = -d (cx in [-4, 3])
// with the weight of the sending pixel p = q + e:
//   k_adj_epf         g_idct(q) += sum_e gv(q + e) W(mul(q + e),
//                     SAD(q, q + e)) (+ g(q) itself where q was copied), for
//                     q + e inside the frame;
//   k_adj_epf_border  the terms whose target p + d lies outside the frame (p
//                     within 4 pixels of the border), scattered to the
//                     mirrored position.
// k_adj_epf follows the forward kernel's tensor-core form (k_epf_box): 64 x
// 16 tiles, one column of four rows per lane, the u8 guide staged as one
// 32-bit word per byte offset, cx outermost so that the seven vertical
// offsets share their guide rows and staged values, and the weight's cut-off
// as a SAD threshold, here of the sender's block: a lane's senders at one cx
// lie in two block rows. The sums and their normaliser recomputed from the
// guide in a pass of their own, and the offsets one by one, took 53 + 101 us
// at 1024x1024; this takes 53. Eight rows per lane, as the forward has, halve
// the warps of an SM and put a lane's senders in three block rows: 60 us there,
// 23 instead of 20 at 512x512, 139 instead of 115 at 1536x1536, 240 instead of
// 195 at 2048x2048.
constexpr int kAdjEpfH = 16, kAdjEpfThreads = 16 * kAdjEpfH;
constexpr int kAdjEpfGH = kAdjEpfH + 8;   // guide rows y0 - 4 .. y0 + 19
constexpr int kAdjEpfGPlane = kAdjEpfGH * kEpfGRow;
constexpr int kAdjEpfTH = kAdjEpfH + 6;   // gather tile rows y0 - 3 .. y0 + 18
constexpr int kAdjEpfTW = kEpfW + 8;      // gather tile cols x0 - 4 .. x0 + 67
constexpr size_t kAdjEpfSmemBytes = size_t(3) * kAdjEpfGPlane * 4 +
                                    size_t(3) * kAdjEpfTH * kAdjEpfTW * 4;

// CpAsync16, or 16 zero bytes.
__device__ __forceinline__ void CpAsync16OrZero(void* smem, const void* gmem,
                                                bool copy) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(
                   uint32_t(__cvta_generic_to_shared(smem))),
               "l"(gmem), "r"(copy ? 16 : 0)
               : "memory");
}

__global__ void __launch_bounds__(kAdjEpfThreads, 3)
    k_adj_epf(int w, int h, const uint8_t* guide, const int32_t* sigma,
              const float* g_filt, float* out) {
  extern __shared__ __align__(16) uint32_t adj_epf_smem[];
  uint32_t* sg = adj_epf_smem;  // [3][kAdjEpfGH][kEpfGRow]
  float(*tile)[kAdjEpfTH][kAdjEpfTW] =
      reinterpret_cast<float(*)[kAdjEpfTH][kAdjEpfTW]>(adj_epf_smem +
                                                       3 * kAdjEpfGPlane);
  // Blocks y0 / 8 - 1 .., x0 / 8 - 1 ..: mul * 64, the SAD threshold (-1:
  // no weight) and the weight's bits beyond it.
  __shared__ int4 s_cut[4][10];
  const int x0 = blockIdx.x * kEpfW, y0 = blockIdx.y * kAdjEpfH;
  const int tid = threadIdx.x, lane = tid & 31, wp = tid >> 5;
  const int band = wp >> 1, col0 = 32 * (wp & 1);
  const size_t plane = size_t(w) * h;
  const int bw = w / 8, bh = h / 8;
  const int px = x0 + lane + col0, py0 = y0 + 4 * band;
  const bool inside = px < w && py0 < h;
  bool sends = false;
  if (tid < 40) {
    const int by = y0 / 8 - 1 + tid / 10, bx = x0 / 8 - 1 + tid % 10;
    int4 cut = make_int4(0, -1, 0, 0);
    if (by >= 0 && by < bh && bx >= 0 && bx < bw) {
      const int sg_ = sigma[by * bw + bx];
      if (sg_ >= kMinSigma) {
        const int m64 = c_t.mul_table[sg_] * 64;
        const EpfCut k = EpfCutOf(sg_, m64);
        cut = make_int4(m64, int(k.thr), __float_as_int(k.cap), 0);
        sends = true;
      }
    }
    s_cut[tid / 10][tid % 10] = cut;
  }
  if (!__syncthreads_or(sends)) {  // nothing around the tile was filtered
    if (!inside) return;
    for (int c = 0; c < 3; ++c)
      for (int j = 0; j < 4; ++j) {
        const size_t o = c * plane + size_t(py0 + j) * w + px;
        out[o] += g_filt[o];
      }
    return;
  }
  // gv of the filtered pixels around the tile, 0 for the others and outside
  // the frame (those terms are the border kernel's); four pixels of one block
  // per copy.
  constexpr int kQ = kAdjEpfTW / 4;
  for (int i = tid; i < 3 * kAdjEpfTH * kQ; i += kAdjEpfThreads) {
    const int c = i / (kAdjEpfTH * kQ);
    const int r = (i / kQ) % kAdjEpfTH, q = i % kQ;
    const int gx = x0 - 4 + 4 * q, gy = y0 - 3 + r;
    const bool ok = gx >= 0 && gx < w && gy >= 0 && gy < h &&
                    s_cut[(gy >> 3) - y0 / 8 + 1][(gx >> 3) - x0 / 8 + 1].x;
    CpAsync16OrZero(&tile[c][r][4 * q],
                    g_filt + (ok ? c * plane + size_t(gy) * w + gx : 0), ok);
  }
  // The u8 guide (6-pixel mirrored border) as words: bytes x0 - 8 ..
  // x0 + 71 of rows y0 - 4 .. y0 + 19 from the aligned words of its rows
  // (w + 12 is a multiple of 4); what lies outside the buffer reads 0.
  const int gwid = w + 12, ght = h + 12;
  constexpr int kAligned = kEpfGBytes / 4, kWords = 3 * kAdjEpfGH * kAligned;
  constexpr int kTurns = (kWords + kAdjEpfThreads - 1) / kAdjEpfThreads;
  uint32_t lo[kTurns], hi[kTurns];  // all of a thread's loads in flight
#pragma unroll
  for (int t = 0; t < kTurns; ++t) {
    const int i = tid + t * kAdjEpfThreads;
    const int c = i / (kAdjEpfGH * kAligned);
    const int r = (i / kAligned) % kAdjEpfGH, wd = i % kAligned;
    const int gy = y0 - 4 + r + 6, gx = x0 - 8 + 4 * wd + 6 - 2;
    const uint8_t* row = guide + (size_t(c) * ght + gy) * gwid;
    const bool in_row = i < kWords && gy >= 0 && gy < ght;
    lo[t] = in_row && gx >= 0 && gx < gwid
                ? *reinterpret_cast<const uint32_t*>(row + gx)
                : 0u;
    hi[t] = in_row && gx + 4 >= 0 && gx + 4 < gwid
                ? *reinterpret_cast<const uint32_t*>(row + gx + 4)
                : 0u;
  }
#pragma unroll
  for (int t = 0; t < kTurns; ++t) {
    const int i = tid + t * kAdjEpfThreads;
    if (i < kWords) sg[4 * i] = __funnelshift_r(lo[t], hi[t], 16);
  }
  CpAsyncWaitAll();
  __syncthreads();
  // The words of the offsets between (bytes past the row end read as 0).
  for (int i = tid; i < kWords; i += kAdjEpfThreads) {
    const int wd = i % kAligned;
    const uint32_t a = sg[4 * i];
    const uint32_t b = wd + 1 < kAligned ? sg[4 * i + 4] : 0u;
    sg[4 * i + 1] = __funnelshift_r(a, b, 8);
    sg[4 * i + 2] = __funnelshift_r(a, b, 16);
    sg[4 * i + 3] = __funnelshift_r(a, b, 24);
  }
  __syncthreads();
  if (!inside) return;  // no barrier follows
  const int gr0 = 4 * band + 3;  // guide smem row of py0 - 1
  const int gc0 = lane + col0 + 7;
  float acc[3][4];
#pragma unroll
  for (int j = 0; j < 4; ++j) acc[0][j] = acc[1][j] = acc[2][j] = 0.f;
  // Sender rows py0 - 3 + R, R = 0..9, lie in block rows first (R < 3, or
  // R < 7 if py0 is in a block's lower half) and first + 1.
  const bool low = (py0 & 4) != 0;
  const int first = (py0 >> 3) - y0 / 8 + (low ? 1 : 0);
#pragma unroll 1
  for (int cx = -4; cx <= 3; ++cx) {
    const uint32_t* g = sg + (gr0 - 3) * kEpfGRow + gc0 + cx;
    uint32_t sad[7][4];
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      uint32_t wd[12];
#pragma unroll
      for (int t = 0; t < 12; ++t) wd[t] = g[c * kAdjEpfGPlane + t * kEpfGRow];
      uint32_t rf[6];
#pragma unroll
      for (int r = 0; r < 6; ++r) {
        rf[r] = sg[c * kAdjEpfGPlane + (gr0 + r) * kEpfGRow + gc0];
      }
#pragma unroll
      for (int k = 0; k < 7; ++k) {
        if (c == 0) {
          PatchSads<true, 4>(rf, wd + k, sad[k]);
        } else {
          PatchSads<false, 4>(rf, wd + k, sad[k]);
        }
      }
    }
    const int bxi = ((px + cx) >> 3) - x0 / 8 + 1;
    const int4 up = s_cut[first][bxi], dn = s_cut[first + 1][bxi];
    const int4 mid = low ? up : dn;
    const int col = lane + col0 + 4 + cx;
#pragma unroll
    for (int R = 0; R < 10; ++R) {
      const int4 cut = R < 3 ? up : R >= 7 ? dn : mid;
      const int tr = 4 * band + R;
      const float v0 = tile[0][tr][col], v1 = tile[1][tr][col],
                  v2 = tile[2][tr][col];
      auto weight = [&](int k, int j) {
        const uint32_t u = sad[k][j] * uint32_t(cut.x) + 0x3F800000u;
        return int(sad[k][j]) <= cut.y ? __uint_as_float(u & 0xFFFF0000u)
                                       : __int_as_float(cut.z);
      };
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const int k = R - j;  // cy + 3
        if (k < 0 || k > 6) continue;
        if (j % 2 == 0 && k > 0) {  // with row j + 1, whose offset is k - 1
          const float w0 = weight(k, j), w1 = weight(k - 1, j + 1);
          Fma2(acc[0][j], acc[0][j + 1], v0, w0, w1);
          Fma2(acc[1][j], acc[1][j + 1], v1, w0, w1);
          Fma2(acc[2][j], acc[2][j + 1], v2, w0, w1);
        } else if (j % 2 == 0 || k == 6) {
          const float w0 = weight(k, j);
          acc[0][j] = fmaf(v0, w0, acc[0][j]);
          acc[1][j] = fmaf(v1, w0, acc[1][j]);
          acc[2][j] = fmaf(v2, w0, acc[2][j]);
        }
      }
    }
  }
  const bool filtered = sigma[(py0 >> 3) * bw + (px >> 3)] >= kMinSigma;
#pragma unroll
  for (int c = 0; c < 3; ++c)
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const size_t o = c * plane + size_t(py0 + j) * w + px;
      out[o] += acc[c][j] + (filtered ? 0.0f : g_filt[o]);
    }
}

// Pass 3: the EPF terms that the forward mirrored back into the frame
// (p + d outside it), scattered from the border band: the rows y < 3 and
// y >= h - 3, and the columns x < 3 and x >= w - 4 of the others. One thread
// per pixel of the band and offset d (a pixel per thread, its 56 offsets in
// turn: 79 us at 1024x1024, now 9).
constexpr int kAdjBand = 4;  // pixels per CTA
__host__ __device__ inline size_t AdjBandPixels(int w, int h) {
  // (an 8-row frame has two rows between its bands, an 8-column one a column)
  return size_t(6) * w + size_t(7) * (h - 6);
}
__global__ void __launch_bounds__(64 * kAdjBand, 4)
    k_adj_epf_border(int w, int h, const uint8_t* guide, const int32_t* sigma,
                     const float* gv, float* g_idct) {
  const size_t i =
      blockIdx.x * size_t(kAdjBand) + (threadIdx.x >> 6);
  const int d = threadIdx.x & 63;
  if (i >= AdjBandPixels(w, h) || d >= 56) return;
  int x, y;
  if (i < size_t(6) * w) {
    x = int(i % w);
    y = int(i / w);
    if (y >= 3) y = h - 6 + y;
  } else {
    const size_t j = i - size_t(6) * w;
    x = int(j % 7);
    y = 3 + int(j / 7);
    if (x >= 3) x = w - 7 + x;
  }
  const int sg = sigma[(y >> 3) * (w / 8) + (x >> 3)];
  if (sg < kMinSigma) return;
  const int cy = d / 8 - 3, cx = d % 8 - 3;
  const int tx = x + cx, ty = y + cy;
  if (tx >= 0 && tx < w && ty >= 0 && ty < h) return;  // gathered
  const size_t plane = size_t(w) * h;
  const int gwid = w + 12, ght = h + 12;
  // The guide's four bytes x .. x + 3 of a row from the two aligned words
  // around them (gwid is a multiple of 4; the rows read lie at least two
  // above the buffer's end, so the second word is always inside it).
  auto gw = [&](int c, int yy, int xx) {
    const size_t o = (size_t(c) * ght + yy + 6) * gwid + xx + 6;
    const uint32_t* p =
        reinterpret_cast<const uint32_t*>(guide + (o & ~size_t(3)));
    return __funnelshift_r(p[0], p[1], 8 * uint32_t(o & 3));
  };
  uint32_t sad_max = 0;
#pragma unroll
  for (int c = 0; c < 3; ++c) {
    uint32_t sad = 0;
#pragma unroll
    for (int py = -1; py <= 1; ++py) {
      sad = Sad4(gw(c, y + py, x - 1), gw(c, ty + py, tx - 1), sad);
    }
    sad_max = max(sad_max, sad);
  }
  const float wgt = EpfWeight(c_t.mul_table[sg] * 64, int(sad_max));
  if (!(wgt >= 0.05f)) return;
  const size_t o = size_t(MirrorIdx(ty, h)) * w + MirrorIdx(tx, w);
  for (int c = 0; c < 3; ++c) {
    atomicAdd(&g_idct[c * plane + o],
              gv[c * plane + size_t(y) * w + x] * wgt);
  }
}

// TransformToPixels transposed for the same blocks; for HF-predicting types
// the masked coefficient gradient (all but 0, 1, 8, 9) through
// TransformFromPixels transposed into the upsampled-prediction gradient.
__global__ void __launch_bounds__(kAdjThreads)
    k_adj_topix8(Geo g, DevFrame f, const AdjJac* J, Adj8Lists lists,
                 int predict_hf, const float* g_idct,
                 float* g_coef, float* g_up) {
  __shared__ __align__(16) float s_p[kAdj8Blocks][3][64];
  __shared__ __align__(16) float s_m[kAdj8Blocks][3][64];
  const int lb = threadIdx.x >> 6, e = threadIdx.x & 63;
  const int item = blockIdx.x * kAdj8Blocks + lb;
  const bool valid = item < lists.count[0] + lists.count[1];
  int bx = 0, by = 0, type = 0;
  if (valid) {
    const uint32_t pk = lists.At(item);
    bx = pk & 0xFFFF;
    by = pk >> 16;
    type = f.acs[by * g.Bx + bx] >> 4;
  }
  const size_t plane = size_t(g.PW) * g.PH;
  const size_t plane_ac = size_t(g.ac_stride) * g.By;
  const size_t o = size_t(by * 8 + e / 8) * g.PW + bx * 8 + e % 8;
  if (valid) {
    for (int c = 0; c < 3; ++c) s_p[lb][c][e] = g_idct[c * plane + o];
  }
  __syncthreads();
  const int t = JIndex(type);
  const bool masked = e == 0 || e == 1 || e == 8 || e == 9;
  if (valid) {
    float gc[3];
    DenseCols(J->j0[t], e, s_p[lb], gc);
    for (int c = 0; c < 3; ++c) {
      g_coef[c * plane_ac + size_t(by) * g.ac_stride + bx * 64 + e] = gc[c];
      s_m[lb][c][e] = masked ? 0.0f : gc[c];
    }
  }
  __syncthreads();
  if (!valid || !predict_hf || !PredictHFOf(type)) return;
  float gp[3];
  DenseCols(J->j1[t], e, s_m[lb], gp);
  for (int c = 0; c < 3; ++c) g_up[c * plane + o] = gp[c];
}

// The same for 8x8 and 16x16 DCT blocks, by rows in registers (a unit of N
// lanes per block and channel, as k_square_idct_rows). At 1024x1024 the 16x16
// blocks took 55 us with a CTA per block and the cooperative transforms, now
// 25; the 8x8 ones 9 us with the dense Jacobians, now 3.5.
template <int N>
__global__ void __launch_bounds__(kSquareThreads)
    k_adj_topix_rows(Geo g, DevFrame f, const uint32_t* list, int count,
                  int predict_hf, const float* g_idct, float* g_coef,
                  float* g_up) {
  using namespace square;
  constexpr int cov = N / 8;
  __shared__ float s_tile[kSquareThreads / N][N * (N + 1)];
  const int unit = threadIdx.x / N, r = threadIdx.x % N;
  const int item = blockIdx.x * (kSquareThreads / N) + unit;
  const bool active = item < 3 * count;
  float* tile = s_tile[unit];
  const int c = active ? item % 3 : 0;
  const uint32_t pk = list[active ? item / 3 : 0];
  const int bx = pk & 0xFFFF, by = pk >> 16;
  const size_t px =
      c * size_t(g.PW) * g.PH + size_t(by * 8 + r) * g.PW + bx * 8;
  float X[N], T[N];
#pragma unroll
  for (int i = 0; i < N; i += 4) {
    const float4 v = *reinterpret_cast<const float4*>(g_idct + px + i);
    X[i] = v.x, X[i + 1] = v.y, X[i + 2] = v.z, X[i + 3] = v.w;
  }
  MatRow<N, true, true>(X, T);
  PutRow<N>(tile, r, T);
  __syncwarp();
  GetCol<N>(tile, r, X);
  MatRow<N, true, true>(X, T);  // row r of the coefficient gradient
  __syncwarp();
  if (active) {
    float* out = g_coef + c * size_t(g.ac_stride) * g.By +
                 CoefRowOffset(g, bx, by, N, r);
#pragma unroll
    for (int i = 0; i < N; i += 4) {
      *reinterpret_cast<float4*>(out + i) =
          make_float4(T[i], T[i + 1], T[i + 2], T[i + 3]);
    }
  }
  if (!predict_hf) return;
  // DCT_NOHF shares the 8x8 class; its gradient is formed but not stored.
  const bool hf = active && PredictHFOf(f.acs[by * g.Bx + bx] >> 4);
  if (r < 2 * cov) {
#pragma unroll
    for (int i = 0; i < 2 * cov; ++i) T[i] = 0.0f;
  }
  MatRow<N, false, true>(T, X);
  PutCol<N>(tile, r, X);
  __syncwarp();
  GetRow<N>(tile, r, X);
  MatRow<N, false, true>(X, T);
  if (hf) {
    constexpr float scale = 1.0f / float(N * N);
#pragma unroll
    for (int i = 0; i < N; i += 4) {
      *reinterpret_cast<float4*>(g_up + px + i) =
          make_float4(T[i] * scale, T[i + 1] * scale, T[i + 2] * scale,
                      T[i + 3] * scale);
    }
  }
}

template <int N>
__global__ void __launch_bounds__(kAdjThreads)
    k_adj_topix_sq(Geo g, DevFrame f, const uint32_t* list, int count,
                   int predict_hf, const float* g_idct, float* g_coef,
                   float* g_up) {
  constexpr int NN = N * N, cov = N / 8, chunk = 64 * cov;
  __shared__ float s_a[NN], s_b[NN], s_x[NN], s_t[NN];
  const int item = blockIdx.x;
  if (item >= count) return;
  const uint32_t pk = list[item];
  const int bx = pk & 0xFFFF, by = pk >> 16;
  const size_t plane = size_t(g.PW) * g.PH;
  const size_t plane_ac = size_t(g.ac_stride) * g.By;
  StageMatrices<N>(s_a, s_b, nullptr);
  for (int c = 0; c < 3; ++c) {
    for (int e = threadIdx.x; e < NN; e += blockDim.x) {
      s_x[e] = g_idct[c * plane + size_t(by * 8 + e / N) * g.PW + bx * 8 +
                      e % N];
    }
    __syncthreads();
    CoopTsIdctT(N, 1, s_a, s_x, s_t, s_x);  // A^T
    float* base = g_coef + c * plane_ac + size_t(by) * g.ac_stride +
                  size_t(bx) * 64;
    for (int e = threadIdx.x; e < NN; e += blockDim.x) {
      base[(e / chunk) * size_t(g.ac_stride) + e % chunk] = s_x[e];
      if (e / N < 2 * cov && e % N < 2 * cov) s_x[e] = 0.0f;
    }
    __syncthreads();
    if (!predict_hf) continue;  // CTA-uniform
    CoopTsDctT(N, 1, s_b, s_x, s_t, s_x);  // B^T
    for (int e = threadIdx.x; e < NN; e += blockDim.x) {
      g_up[c * plane + size_t(by * 8 + e / N) * g.PW + bx * 8 + e % N] =
          s_x[e];
    }
    __syncthreads();
  }
}

// UpSample4x4BlurDCT (pik/ac_predictions.cc:263-374) transposed: the
// gradient of each block-interior pred2x2 cell of a group gathered from the
// 12 x 12 upsampled pixels that read it.
__global__ void k_adj_upsample(Geo g, const float* g_up, float* g_pred) {
  const int gi = blockIdx.z / 3, c = blockIdx.z % 3;
  int x0, y0, gxs, gys;
  GroupDims(g, gi, &x0, &y0, &gxs, &gys);
  const int Q = 2 + blockIdx.x * blockDim.x + threadIdx.x;
  const int R = 2 + blockIdx.y * blockDim.y + threadIdx.y;
  if (Q >= 2 * gxs + 2 || R >= 2 * gys + 2) return;
  const float* up =
      g_up + size_t(c) * g.PW * g.PH + size_t(8 * y0) * g.PW + 8 * x0;
  float s = 0.0f;
  for (int j = 0; j < 3; ++j) {
    const int r = R - 1 - j;
    if (r < 0 || r >= 2 * gys) continue;
    for (int iy = 0; iy < 4; ++iy) {
      const float* row = up + size_t(4 * r + iy) * g.PW;
      float hsum = 0.0f;
      for (int i = 0; i < 3; ++i) {
        const int q = Q - 1 - i;
        if (q < 0 || q >= 2 * gxs) continue;
        for (int ix = 0; ix < 4; ++ix) {
          hsum += c_t.ub4[i][ix] * row[4 * q + ix];
        }
      }
      s += c_t.ub4[j][iy] * hsum;
    }
  }
  g_pred[gi * kG2GroupFloats + c * kG2 * kG2 + R * kG2 + Q] = s;
}

// Per first block and channel: DC2x2FromLowFrequencies transposed into the
// LF corner (HF prediction), then the LLF coefficients' gradient is zeroed
// (they are overwritten by values from DC).
__global__ void k_adj_lf(Geo g, DevFrame f, const AdjJac* J, int predict_hf,
                         const float* g_pred, float* g_coef) {
  const int bx = blockIdx.x * blockDim.x + threadIdx.x;
  const int by = blockIdx.y * blockDim.y + threadIdx.y;
  const int c = blockIdx.z;
  if (bx >= g.Bx || by >= g.By) return;
  const int a = f.acs[by * g.Bx + bx];
  if (a & 0xF) return;
  const int type = a >> 4, cov = Covered(type), n = 8 * cov, m = 2 * cov;
  const int chunk = 64 * cov;
  float* base = g_coef + c * size_t(g.ac_stride) * g.By +
                size_t(by) * g.ac_stride + size_t(bx) * 64;
  auto at = [&](int i) -> float& {
    return base[(i / chunk) * size_t(g.ac_stride) + i % chunk];
  };
  if (predict_hf) {
    const int gi = (by >> 6) * g.Gx + (bx >> 6);
    const int lbx = bx & 63, lby = by & 63;
    const float* gp = g_pred + gi * kG2GroupFloats + c * kG2 * kG2 +
                      2 * (lby + 1) * kG2 + 2 * (lbx + 1);
    float cell[64];
    for (int r = 0; r < m * m; ++r) cell[r] = gp[(r / m) * kG2 + r % m];
    for (int u = 0; u < m * m; ++u) {
      float sum = 0.0f;
      for (int r = 0; r < m * m; ++r) sum += J->j2[type][r][u] * cell[r];
      at((u / m) * n + u % m) += sum;
    }
  }
  for (int y = 0; y < cov; ++y)
    for (int x = 0; x < cov; ++x) at(y * n + x) = 0.0f;
}

// Quant field: every coefficient of a cell scales with 1 / qf, so
// d L / d qf += -sum(g * ac) / qf (FP64 sum). One warp per cell, two
// coefficients per lane and channel (a cell per thread read 192 strided
// values in turn: 54 us at 1024x1024, now 6.5).
constexpr int kAdjQfCells = 8;  // warps per CTA
__global__ void __launch_bounds__(32 * kAdjQfCells)
    k_adj_qf(Geo g, DevFrame f, const float* ac0, const float* g_coef,
             float* g_qf) {
  const int cell = blockIdx.x * kAdjQfCells + (threadIdx.x >> 5);
  if (cell >= g.Bx * g.By) return;
  const int lane = threadIdx.x & 31;
  const int bx = cell % g.Bx, by = cell / g.Bx;
  const size_t plane_ac = size_t(g.ac_stride) * g.By;
  const size_t o = size_t(by) * g.ac_stride + size_t(bx) * 64 + 2 * lane;
  double s = 0.0;
#pragma unroll
  for (int c = 0; c < 3; ++c) {
    const float2 u =
        *reinterpret_cast<const float2*>(g_coef + c * plane_ac + o);
    const float2 v = *reinterpret_cast<const float2*>(ac0 + c * plane_ac + o);
    s += double(u.x) * double(v.x);
    s += double(u.y) * double(v.y);
  }
  for (int off = 16; off; off >>= 1) s += __shfl_xor_sync(~0u, s, off);
  if (lane) return;
  double q = double(f.qf[cell]);
  if (f.clamp_scale) q /= double(f.clamp_scale[cell]);
  g_qf[cell] += float(-s / q);
}

}  // namespace
}  // namespace pikgpu

namespace {

// The backward launches; the forward pass (with the stages it reads) has
// run on ctx->stream.
int LaunchAdjoint(pikgpu_ctx* ctx, const float* target) {
  const Geo& g = ctx->g;
  const FrameScalars& s = ctx->s;
  cudaStream_t st = ctx->stream;
  const size_t npx = size_t(g.PW) * g.PH;
  const size_t nac = size_t(g.ac_stride) * g.By;
  const int nb = g.Bx * g.By;
  DevFrame f{};
  f.acs = P<uint8_t>(ctx->acs);
  f.qf = P<int32_t>(ctx->qf);
  f.dq_cf = P<uint8_t>(ctx->dq_cf);
  f.dq_map = P<uint8_t>(ctx->dq_map);
  f.table = P<float>(ctx->table);
  f.offsets = P<uint32_t>(ctx->offsets);
  f.idct = P<float>(ctx->idct);
  f.clamp_scale = ctx->use_clamp_scale ? P<float>(ctx->clamp_scale) : nullptr;
  const AdjJac* J = P<AdjJac>(ctx->adj_jac);
  float* ga = P<float>(ctx->adj_a);  // g_pre, then g_filt
  float* gb = P<float>(ctx->adj_b);  // g_cur, then g_up
  float* gc = P<float>(ctx->adj_c);  // g_idct
  float* g_coef = P<float>(ctx->adj_coef);
  float* g_qf = P<float>(ctx->adj_qf);
  const uint32_t* L[kNumClasses];
  int n[kNumClasses];
  for (int k = 0; k < kNumClasses; ++k) {
    L[k] = P<uint32_t>(ctx->list[k]);
    n[k] = int(ctx->lists[k].size());
  }
  const Adj8Lists lists8 = {{L[kC4], L[kCSmall]}, {n[kC4], n[kCSmall]}};

  k_adj_loss<<<kAdjLossBlocks, kAdjThreads, 0, st>>>(
      P<float>(ctx->dbg_pre), target, g.W, g.H, g.PW, g.PH, ga,
      P<double>(ctx->adj_partial));
  k_adj_sum<<<1, 32, 0, st>>>(P<double>(ctx->adj_partial), kAdjLossBlocks,
                              P<double>(ctx->adj_partial) + kAdjLossBlocks);
  ctx->launches += 2;
  const float* g_cur = ga;
  if (s.gaborish) {
    dim3 b(32, 8), gr(Blocks(g.PW / 4, 32), Blocks(g.PH, 8), 3);
    k_adj_gab<<<gr, b, 0, st>>>(ga, g.PW, g.PH, s.gaborish, gb);
    ++ctx->launches;
    g_cur = gb;
  }
  CUDA_TRY(ctx, cudaMemsetAsync(g_qf, 0, sizeof(float) * nb, st));
  const float* g_idct = g_cur;
  if (s.have_ar) {
    // Guide bytes of the forward pass (the override, or MakeGuide again).
    const uint8_t* guide = P<uint8_t>(ctx->guide_ovr);
    if (!ctx->use_guide_ovr) {
      dim3 b(32, 8), gr(Blocks(g.PW / 4 + 3, 32), Blocks(g.PH + 12, 8), 3);
      k_export_guide<<<gr, b, 0, st>>>(
          f.idct, s.use_sharpened ? 0 : s.gaborish, g.PW, g.PH,
          P<uint32_t>(ctx->mm), P<uint8_t>(ctx->adj_guide));
      ++ctx->launches;
      guide = P<uint8_t>(ctx->adj_guide);
    }
    const int32_t* sig = P<int32_t>(ctx->sigma);
    const uint8_t* tape = P<uint8_t>(ctx->adj_tape);
    const float* epf = P<float>(ctx->dbg_epf);
    const float* sum_w = P<float>(ctx->adj_sw);
    // g_filt goes to ga (g_pre is dead once g_cur exists; without
    // gaborish g_cur is ga itself, so g_filt then takes gb).
    float* g_filt = s.gaborish ? ga : gb;
    if (n[kC8]) {
      k_adj_ar_dct8<<<Blocks(n[kC8], SquareArBlocks<8>()), kSquareArThreads, 0,
                      st>>>(
          g, f, s, L[kC8], n[kC8], sig, tape, epf, sum_w, g_cur, g_filt, gc,
          g_qf);
      ++ctx->launches;
    }
    if (n[kC4] + n[kCSmall]) {
      k_adj_ar8<<<Blocks(n[kC4] + n[kCSmall], kAdj8Blocks), kAdjThreads, 0,
                  st>>>(g, f, s, J, lists8, sig, tape, epf, sum_w, g_cur,
                        g_filt, gc, g_qf);
      ++ctx->launches;
    }
    if (n[kC16]) {
      k_adj_ar_sq<16><<<n[kC16], kAdjThreads, 0, st>>>(
          g, f, s, L[kC16], n[kC16], sig, tape, epf, sum_w, g_cur, g_filt, gc,
          g_qf);
      ++ctx->launches;
    }
    if (n[kC32]) {
      k_adj_ar_sq<32><<<n[kC32], kAdjThreads, 0, st>>>(
          g, f, s, L[kC32], n[kC32], sig, tape, epf, sum_w, g_cur, g_filt, gc,
          g_qf);
      ++ctx->launches;
    }
    dim3 gr(Blocks(g.PW, kEpfW), Blocks(g.PH, kAdjEpfH));
    k_adj_epf<<<gr, kAdjEpfThreads, kAdjEpfSmemBytes, st>>>(
        g.PW, g.PH, guide, sig, g_filt, gc);
    k_adj_epf_border<<<Blocks(AdjBandPixels(g.PW, g.PH), kAdjBand),
                       64 * kAdjBand, 0, st>>>(g.PW, g.PH, guide, sig, g_filt,
                                              gc);
    ctx->launches += 2;
    g_idct = gc;
  }
  // g_up: the upsampled-prediction gradient (zero outside HF blocks), in
  // whichever plane buffer g_idct does not occupy.
  float* g_up = g_idct == gb ? gc : gb;
  if (s.predict_hf) {
    CUDA_TRY(ctx, cudaMemsetAsync(g_up, 0, sizeof(float) * 3 * npx, st));
  }
  if (n[kC8]) {
    k_adj_topix_rows<8><<<Blocks(3 * n[kC8], kSquareThreads / 8),
                          kSquareThreads, 0, st>>>(
        g, f, L[kC8], n[kC8], s.predict_hf, g_idct, g_coef, g_up);
    ++ctx->launches;
  }
  if (n[kC4] + n[kCSmall]) {
    k_adj_topix8<<<Blocks(n[kC4] + n[kCSmall], kAdj8Blocks), kAdjThreads, 0,
                   st>>>(g, f, J, lists8, s.predict_hf, g_idct, g_coef, g_up);
    ++ctx->launches;
  }
  if (n[kC16]) {
    k_adj_topix_rows<16><<<Blocks(3 * n[kC16], kSquareThreads / 16),
                           kSquareThreads, 0, st>>>(
        g, f, L[kC16], n[kC16], s.predict_hf, g_idct, g_coef, g_up);
    ++ctx->launches;
  }
  if (n[kC32]) {
    k_adj_topix_sq<32><<<n[kC32], kAdjThreads, 0, st>>>(
        g, f, L[kC32], n[kC32], s.predict_hf, g_idct, g_coef, g_up);
    ++ctx->launches;
  }
  const int ng = g.Gx * g.Gy;
  if (s.predict_hf) {
    dim3 b(16, 16), gr(Blocks(2 * 64, 16), Blocks(2 * 64, 16), 3 * ng);
    k_adj_upsample<<<gr, b, 0, st>>>(g, g_up, P<float>(ctx->adj_pred));
    ++ctx->launches;
  }
  {
    dim3 b(32, 8), gr(Blocks(g.Bx, 32), Blocks(g.By, 8), 3);
    k_adj_lf<<<gr, b, 0, st>>>(g, f, J, s.predict_hf, P<float>(ctx->adj_pred),
                               g_coef);
    ++ctx->launches;
  }
  const float* ac0 =
      ctx->use_dq_ovr ? P<float>(ctx->dq_ovr) : P<float>(ctx->dbg_dequant);
  k_adj_qf<<<Blocks(nb, kAdjQfCells), 32 * kAdjQfCells, 0, st>>>(
      g, f, ac0, g_coef, g_qf);
  ++ctx->launches;
  (void)nac;
  CUDA_TRY(ctx, cudaGetLastError());
  return PIKGPU_OK;
}

}  // namespace

extern "C" {

int pikgpu_frame_set_dequantized_ac(pikgpu_ctx* ctx, const float* ac,
                                    int on_device) {
  if (!ctx) return PIKGPU_ERR_INVALID_ARG;
  PIKGPU_NOT_PENDING(ctx);
  if (!ctx->have_frame) return Fail(ctx, PIKGPU_ERR_STATE, "no frame");
  ++ctx->generation;
  ctx->use_dq_ovr = ac != nullptr;
  if (!ac) return PIKGPU_OK;
  const Geo& g = ctx->g;
  const size_t bytes = sizeof(float) * 3 * size_t(g.ac_stride) * g.By;
  int rc;
  if ((rc = Ensure(ctx, &ctx->dq_ovr, bytes))) return rc;
  CUDA_TRY(ctx, cudaSetDevice(ctx->device));
  CUDA_TRY(ctx, cudaMemcpyAsync(ctx->dq_ovr.p, ac, bytes,
                                on_device ? cudaMemcpyDeviceToDevice
                                          : cudaMemcpyHostToDevice,
                                ctx->stream));
  CUDA_TRY(ctx, cudaStreamSynchronize(ctx->stream));
  return PIKGPU_OK;
}

int pikgpu_frame_set_clamp_scale(pikgpu_ctx* ctx, const float* scale,
                                 int on_device) {
  if (!ctx) return PIKGPU_ERR_INVALID_ARG;
  PIKGPU_NOT_PENDING(ctx);
  if (!ctx->have_frame) return Fail(ctx, PIKGPU_ERR_STATE, "no frame");
  ++ctx->generation;
  ctx->use_clamp_scale = scale != nullptr;
  if (!scale) return PIKGPU_OK;
  const size_t bytes = sizeof(float) * size_t(ctx->g.Bx) * ctx->g.By;
  int rc;
  if ((rc = Ensure(ctx, &ctx->clamp_scale, bytes))) return rc;
  CUDA_TRY(ctx, cudaSetDevice(ctx->device));
  CUDA_TRY(ctx, cudaMemcpyAsync(ctx->clamp_scale.p, scale, bytes,
                                on_device ? cudaMemcpyDeviceToDevice
                                          : cudaMemcpyHostToDevice,
                                ctx->stream));
  CUDA_TRY(ctx, cudaStreamSynchronize(ctx->stream));
  return PIKGPU_OK;
}

int pikgpu_set_clamp_decisions(pikgpu_ctx* ctx, const uint8_t* tape) {
  if (!ctx) return PIKGPU_ERR_INVALID_ARG;
  PIKGPU_NOT_PENDING(ctx);
  if (!ctx->have_frame) return Fail(ctx, PIKGPU_ERR_STATE, "no frame");
  ++ctx->generation;
  ctx->use_tape_in = false;
  if (!tape) return PIKGPU_OK;
  const size_t n = size_t(ctx->g.ac_stride) * ctx->g.By;
  for (size_t i = 0; i < n; ++i) {
    if (tape[i] > 4) {
      return Fail(ctx, PIKGPU_ERR_INVALID_ARG, "clamp tape code %u at %zu",
                  tape[i], i);
    }
  }
  int rc;
  if ((rc = Ensure(ctx, &ctx->tape_in, n))) return rc;
  CUDA_TRY(ctx, cudaSetDevice(ctx->device));
  CUDA_TRY(ctx, cudaMemcpy(ctx->tape_in.p, tape, n, cudaMemcpyHostToDevice));
  ctx->use_tape_in = true;
  return PIKGPU_OK;
}

int pikgpu_get_clamp_decisions(pikgpu_ctx* ctx, uint8_t* tape) {
  if (!ctx || !tape) return PIKGPU_ERR_INVALID_ARG;
  PIKGPU_NOT_PENDING(ctx);
  if (!ctx->have_result || !ctx->tape_valid) {
    return Fail(ctx, PIKGPU_ERR_STATE,
                "no clamp tape: needs a frame with the EPF and a forward pass "
                "with PIKGPU_OPT_KEEP_STAGES (set before frame_begin) or "
                "pikgpu_adjoint");
  }
  CUDA_TRY(ctx, cudaSetDevice(ctx->device));
  CUDA_TRY(ctx, cudaMemcpy(tape, ctx->adj_tape.p,
                           size_t(ctx->g.ac_stride) * ctx->g.By,
                           cudaMemcpyDeviceToHost));
  return PIKGPU_OK;
}

int pikgpu_adjoint(pikgpu_ctx* ctx, const float* target, double* loss,
                   float* grad_ac, float* grad_qf, int buffers_on_device) {
  if (!ctx) return PIKGPU_ERR_INVALID_ARG;
  PIKGPU_NOT_PENDING(ctx);
  if (!ctx->have_frame || !(ctx->have_ac || ctx->use_dq_ovr)) {
    return Fail(ctx, PIKGPU_ERR_STATE, "frame or AC not supplied");
  }
  if (!target) return Fail(ctx, PIKGPU_ERR_INVALID_ARG, "target is NULL");
  CUDA_TRY(ctx, cudaSetDevice(ctx->device));
  const Geo& g = ctx->g;
  const size_t npx = size_t(g.PW) * g.PH;
  const size_t nac = size_t(g.ac_stride) * g.By;
  const size_t nb = size_t(g.Bx) * g.By;
  const size_t ntg = 3 * size_t(g.W) * g.H;
  const int ng = g.Gx * g.Gy;
  int rc;
  if ((rc = Ensure(ctx, &ctx->adj_a, 4 * 3 * npx)) ||
      (rc = Ensure(ctx, &ctx->adj_b, 4 * 3 * npx)) ||
      (rc = Ensure(ctx, &ctx->adj_c, 4 * 3 * npx)) ||
      (rc = Ensure(ctx, &ctx->adj_coef, 4 * 3 * nac)) ||
      (rc = Ensure(ctx, &ctx->adj_pred, 4 * kG2GroupFloats * ng)) ||
      (rc = Ensure(ctx, &ctx->adj_qf, 4 * nb)) ||
      (rc = Ensure(ctx, &ctx->adj_guide,
                   3 * size_t(g.PW + 12) * (g.PH + 12))) ||
      (rc = Ensure(ctx, &ctx->adj_partial,
                   sizeof(double) * (kAdjLossBlocks + 1))) ||
      (rc = Ensure(ctx, &ctx->adj_jac, sizeof(AdjJac))) ||
      (rc = Ensure(ctx, &ctx->adj_tape, nac)) ||
      (rc = Ensure(ctx, &ctx->adj_sw, 4 * npx)) ||
      (rc = Ensure(ctx, &ctx->dbg_dequant, 4 * 3 * nac)) ||
      (rc = Ensure(ctx, &ctx->dbg_epf, 4 * 3 * npx)) ||
      (rc = Ensure(ctx, &ctx->dbg_pre, 4 * ntg))) {
    return rc;
  }
  cudaStream_t st = ctx->stream;
  if (!ctx->adj_jac_built) {
    CUDA_TRY(ctx, cudaFuncSetAttribute(
                      k_adj_epf, cudaFuncAttributeMaxDynamicSharedMemorySize,
                      int(kAdjEpfSmemBytes)));
    k_adj_build_jac<<<2 * kJTypes + 9, 64, 0, st>>>(P<AdjJac>(ctx->adj_jac));
    CUDA_TRY(ctx, cudaGetLastError());
    ctx->adj_jac_built = true;
  }
  const float* tgt = target;
  if (!buffers_on_device) {
    if ((rc = Ensure(ctx, &ctx->adj_target, 4 * ntg))) return rc;
    CUDA_TRY(ctx, cudaMemcpyAsync(ctx->adj_target.p, target, 4 * ntg,
                                  cudaMemcpyHostToDevice, st));
    tgt = P<float>(ctx->adj_target);
  }
  // Forward pass, keeping the dequantised AC, the EPF output and pre_opsin.
  // The clamp kernels also record their branches (the clamp tape).
  const bool keep = ctx->keep_stages;
  ctx->keep_stages = ctx->record_tape = true;
  rc = LaunchAll(ctx, nullptr, 0, nullptr, 0);
  ctx->keep_stages = keep;
  ctx->record_tape = false;
  if (rc != PIKGPU_OK) return rc;
  if ((rc = LaunchAdjoint(ctx, tgt)) != PIKGPU_OK) return rc;
  const cudaMemcpyKind kind =
      buffers_on_device ? cudaMemcpyDeviceToDevice : cudaMemcpyDeviceToHost;
  if (grad_ac) {
    CUDA_TRY(ctx, cudaMemcpyAsync(grad_ac, ctx->adj_coef.p, 4 * 3 * nac, kind,
                                  st));
  }
  if (grad_qf) {
    CUDA_TRY(ctx, cudaMemcpyAsync(grad_qf, ctx->adj_qf.p, 4 * nb, kind, st));
  }
  if (loss) {
    CUDA_TRY(ctx, cudaMemcpyAsync(
                      loss, P<double>(ctx->adj_partial) + kAdjLossBlocks,
                      sizeof(double), kind, st));
  }
  CUDA_TRY(ctx, cudaStreamSynchronize(st));
  if (const int code = TakeTimeout(ctx)) {
    return Fail(ctx, PIKGPU_ERR_CUDA, "%s", WaitTimeoutMessage(code));
  }
  ctx->have_result = true;
  return PIKGPU_OK;
}

}  // extern "C"
