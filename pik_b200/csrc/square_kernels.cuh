// Square DCT blocks (8x8, 16x16) with one thread per row of the
// N x N block: a "unit" of N lanes holds one block (and channel) in
// registers, the transform matrices are compile-time operands from
// __constant__ memory, and the transpose between the two separable passes
// goes through a padded shared-memory tile with __syncwarp only. Every
// output is the same sequential sum (index 0..N-1, separate multiply and
// add) as the row-major formulation, so results are bit-identical to it.
// Included by recon_kernels.cu.
#pragma once

namespace pikgpu {
namespace square {

// A row times the transform matrix `m` (in constant memory): o[k] =
// sum_i M[k][i] v[i], two outputs' sums in one instruction: three issue slots
// for two rounded products and sums instead of four, and the FP32 pipe is the
// bound. 16x16 blocks of a 4K frame: inverse 141 -> 128 us, clamp 66 -> 57.
template <int N>
__device__ __forceinline__ void MatRow(const float* m, const float (&v)[N],
                                       float (&o)[N]) {
#pragma unroll
  for (int k = 0; k < N; k += 2) {
    float s0 = 0.f, s1 = 0.f;
#pragma unroll
    for (int i = 0; i < N; ++i) {
      Add2(s0, s1, v[i] * m[k * N + i], v[i] * m[(k + 1) * N + i]);
    }
    o[k] = s0;
    o[k + 1] = s1;
  }
}
// tsIDCT pass: t[v] = sum_l c[l] A[v][l], on coefficient row c (row =
// horizontal frequency k), then on the columns of its output.
template <int N>
__device__ __forceinline__ void IdctRow(const float (&c)[N], float (&t)[N]) {
  MatRow<N>(c_t.idct + MatOffset(N), c, t);
}
// tsDCT pass 1 on pixel row p (row y): t[k] = sum_x B[k][x] p[x].
template <int N>
__device__ __forceinline__ void DctRow(const float (&p)[N], float (&t)[N]) {
  MatRow<N>(c_t.dct + MatOffset(N), p, t);
}
// tsDCT pass 2 on q[y] = tmp[k][y]: o[l] = (sum_y q[y] B[l][y]) / N^2.
template <int N>
__device__ __forceinline__ void DctCol(const float (&q)[N], float (&o)[N]) {
  DctRow<N>(q, o);
#pragma unroll
  for (int l = 0; l < N; ++l) o[l] *= 1.0f / float(N * N);
}

// Writes `v` as row r of the unit's tile (stride N + 1) ...
template <int N>
__device__ __forceinline__ void PutRow(float* tile, int r, const float (&v)[N]) {
#pragma unroll
  for (int i = 0; i < N; ++i) tile[r * (N + 1) + i] = v[i];
}
template <int N>
__device__ __forceinline__ void PutCol(float* tile, int r, const float (&v)[N]) {
#pragma unroll
  for (int i = 0; i < N; ++i) tile[i * (N + 1) + r] = v[i];
}
template <int N>
__device__ __forceinline__ void GetRow(const float* tile, int r, float (&v)[N]) {
#pragma unroll
  for (int i = 0; i < N; ++i) v[i] = tile[r * (N + 1) + i];
}
template <int N>
__device__ __forceinline__ void GetCol(const float* tile, int r, float (&v)[N]) {
#pragma unroll
  for (int i = 0; i < N; ++i) v[i] = tile[i * (N + 1) + r];
}

// Pointer to row r of the block's coefficients in the frame layout: row r
// of the N x N matrix lives in block row (by + r / 8) at column offset
// bx * 64 + (r % 8) * N (GatherCoefficients layout, pik/ac_strategy.h:255-272).
__device__ __forceinline__ size_t CoefRowOffset(const Geo& g, int bx, int by,
                                                int n, int r) {
  return size_t(by + r / 8) * g.ac_stride + size_t(bx) * 64 + (r % 8) * n;
}

}  // namespace square

constexpr int kSquareThreads = 128;

// HF prediction + AddBlockExceptLFAndLLFTo + IDCT for square DCT blocks
// (UpSample4x4BlurDCT, pik/ac_predictions.cc:263-374; TransformToPixels,
// pik/ac_strategy.cc:674-848). One unit per (block, channel).
template <int N>
__global__ void __launch_bounds__(kSquareThreads)
    k_square_idct_rows(Geo g, DevFrame f, const uint32_t* list, int count,
                       int predict_hf) {
  PdlLaunchDependents();
  PdlTail pdl_tail;
  using namespace square;
  constexpr int UPW = 32 / N;  // units per warp
  constexpr int cov = N / 8;
  __shared__ float s_tile[kSquareThreads / N][N * (N + 1)];
  const int lane = threadIdx.x & 31;
  const int warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int unit = lane / N, r = lane % N;
  const int item = warp * UPW + unit;
  if (warp * UPW >= 3 * count) return;  // warp-uniform
  const bool active = item < 3 * count;
  float* tile = s_tile[threadIdx.x / N];
  const int b = active ? item / 3 : 0, c = active ? item % 3 : 0;
  const uint32_t pk = list[b];
  const int bx = pk & 0xFFFF, by = pk >> 16;
  const size_t plane_ac = size_t(g.ac_stride) * g.By;
  const float* crow = f.ac + c * plane_ac + CoefRowOffset(g, bx, by, N, r);
  float X[N];
#pragma unroll
  for (int i = 0; i < N; i += 4) {
    const float4 v = *reinterpret_cast<const float4*>(crow + i);
    X[i] = v.x, X[i + 1] = v.y, X[i + 2] = v.z, X[i + 3] = v.w;
  }
  if (predict_hf) {
    // DCT_NOHF shares the 8x8 class; its prediction is computed but not
    // added, keeping the warp's control flow uniform.
    const bool hf = PredictHFOf(f.acs[by * g.Bx + bx] >> 4);
    const int gi = (by >> 6) * g.Gx + (bx >> 6);
    const float* pred = f.pred2x2_g + gi * kG2GroupFloats + c * kG2 * kG2;
    const int X0 = (bx & 63) * 8, Y = (by & 63) * 8 + r;
    float P[N], T[N];
    UpsampleRow<N>(pred, X0, Y, P);
    DctRow<N>(P, T);
    PutCol<N>(tile, r, T);  // tmp[k][y = r]
    __syncwarp();
    GetRow<N>(tile, r, P);  // tmp[k = r][y]
    DctCol<N>(P, T);        // predicted coefficients row k = r
    __syncwarp();
#pragma unroll
    for (int l = 0; l < N; ++l) {
      if (hf && !(r < 2 * cov && l < 2 * cov)) X[l] += T[l];
    }
  }
  float T[N];
  IdctRow<N>(X, T);
  PutRow<N>(tile, r, T);  // tmp[k = r][v]
  __syncwarp();
  GetCol<N>(tile, r, X);  // column v = r
  IdctRow<N>(X, T);       // pixel row v = r
  if (active) {
    float* out = f.idct + c * size_t(g.PW) * g.PH +
                 size_t(by * 8 + r) * g.PW + bx * 8;
#pragma unroll
    for (int i = 0; i < N; i += 4) {
      *reinterpret_cast<float4*>(out + i) =
          make_float4(T[i], T[i + 1], T[i + 2], T[i + 3]);
    }
  }
}

// What the EPF and the clamp have to do, once the guide's range is known.
// One thread per block of all the classes:
//  * the sigma of its cells (SigmaFromQuant): `ovr` (the verification
//    override) if set; else `fixed` if >= 0 (the fixed-sigma EPF,
//    pik/epf_target.cc:1342-1386); else from the cell's quant field, strategy
//    and LUT;
//  * the block into its class's active list (counter k) if some cell is
//    filtered (sigma >= kMinSigma); for the others the clamp stage is an
//    exact no-op because the filtered block equals the original;
//  * its region (kRegionW x kRegionH pixels; no block crosses one) into the
//    EPF's list, once, if it is active or every region is kept.
struct EpfPlan {
  const int32_t* ovr;
  int fixed;
  int keep_all;
  int32_t* sigma;
  uint32_t* region;       // 0 / 1 per region
  uint32_t* region_list;  // the regions set, *region_count of them
  int* region_count;
};
__global__ void __launch_bounds__(256)
    k_epf_plan(Geo g, DevFrame f, const uint32_t* mm, EpfPlan p,
               ClassLists cl, int* counters) {
  PdlLaunchDependents();  // the EPF may start on free SMs
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  int k = 0;
  while (k < kMaxClasses && i >= cl.n[k]) i -= cl.n[k++];
  const bool on = k < kMaxClasses;
  uint32_t pk = 0;
  int cov = 0, cell0 = 0;
  float scale = 1.0f, most = 0.f;
  if (on) {
    // The inputs do not wait for the guide's range, and a sigma grows with
    // its unscaled value: the largest tells whether the block is filtered.
    pk = cl.list[k][i];
    cell0 = int(pk >> 16) * g.Bx + int(pk & 0xFFFF);
    const int type = f.acs[cell0] >> 4;
    cov = Covered(type);
    scale = ARQuantScaleOf(type);
    for (int y = 0; y < cov; ++y) {
      for (int x = 0; x < cov; ++x) {
        const int cell = cell0 + y * g.Bx + x;
        most = fmaxf(most,
                     UnscaledSigma(float(f.qf[cell]), scale, f.lut[cell]));
      }
    }
  }
  PdlWait();  // the min/max pass
  float amin, mul, stretch;
  GuideParams(mm, &amin, &mul, &stretch);
  bool any = on && (p.fixed >= 0 ? p.fixed : ScaledSigma(most, stretch)) >=
                       kMinSigma;
  if (p.ovr) {
    any = false;
    for (int y = 0; y < cov; ++y)
      for (int x = 0; x < cov; ++x)
        any |= p.ovr[cell0 + y * g.Bx + x] >= kMinSigma;
  }
  const int bx = pk & 0xFFFF, by = pk >> 16;
  if (on && (any || p.keep_all)) {
    const int rw = (g.PW + kRegionW - 1) / kRegionW;
    const int r = by / (kRegionH / 8) * rw + bx / (kRegionW / 8);
    if (p.region[r] == 0 && atomicExch(&p.region[r], 1u) == 0u) {
      p.region_list[atomicAdd(p.region_count, 1)] = r;
    }
  }
  // One atomic per warp and class: the lanes of a class take consecutive
  // slots after the first of them reserves them all.
  const int lane = threadIdx.x & 31;
  for (int kk = 0; kk < kMaxClasses; ++kk) {
    const uint32_t m = __ballot_sync(0xFFFFFFFFu, any && k == kk);
    if (!m) continue;
    const int leader = __ffs(m) - 1;
    int base = 0;
    if (lane == leader) base = atomicAdd(&counters[kk], __popc(m));
    base = __shfl_sync(0xFFFFFFFFu, base, leader);
    if (any && k == kk) {
      cl.active[kk][base + __popc(m & ((1u << lane) - 1))] = pk;
    }
  }
  for (int y = 0; y < cov; ++y) {
    for (int x = 0; x < cov; ++x) {
      const int cell = cell0 + y * g.Bx + x;
      p.sigma[cell] =
          p.ovr          ? p.ovr[cell]
          : p.fixed >= 0 ? p.fixed
                         : ScaledSigma(UnscaledSigma(float(f.qf[cell]), scale,
                                                     f.lut[cell]),
                                       stretch);
    }
  }
}

// Clamp intervals of N consecutive coefficients from the dequantisation
// matrix at `dm` (16-byte loads where its place in the table allows them).
template <int N>
__device__ __forceinline__ void LoadIntervals(const float* dm, float scale,
                                              float (&v)[N]) {
  if ((reinterpret_cast<uintptr_t>(dm) & 15) == 0) {
#pragma unroll
    for (int i = 0; i < N; i += 4) {
      const float4 q = *reinterpret_cast<const float4*>(dm + i);
      v[i] = q.x * scale, v[i + 1] = q.y * scale;
      v[i + 2] = q.z * scale, v[i + 3] = q.w * scale;
    }
  } else {
#pragma unroll
    for (int i = 0; i < N; ++i) v[i] = dm[i] * scale;
  }
}

// AdaptiveReconstruction clamp for square DCT blocks
// (pik/adaptive_reconstruction.cc:128-244, 334-471): a warp per channel of
// 32 / N blocks, the channels' ratios meeting in shared memory. With the
// three channels in one warp instead (three times the registers and a third
// of the warps) the clamp of a 256x256 frame of 16x16 blocks took 27 us
// against 9, of a 3840x2160 one 103 against 65. `count` is read from device
// memory (the compacted list of k_epf_plan).
constexpr int kSquareArGroups = 2;  // warps per channel in a CTA
constexpr int kSquareArThreads = 96 * kSquareArGroups;
template <int N>
__host__ __device__ constexpr int SquareArBlocks() {  // blocks per CTA
  return kSquareArGroups * 32 / N;
}
template <int N>
__global__ void __launch_bounds__(kSquareArThreads)
    k_square_ar_rows(Geo g, DevFrame f, FrameScalars s, const uint32_t* list,
                     const int* count_ptr) {
  PdlLaunchDependents();
  PdlTail pdl_tail;
  using namespace square;
  constexpr int UPW = 32 / N;
  constexpr int cov = N / 8, tile_size = N * (N + 1);
  __shared__ float s_tile[kSquareArGroups][3][UPW][tile_size];
  __shared__ float s_ratio[kSquareArGroups][3][UPW][tile_size];
  const int count = *count_ptr;
  if (int(blockIdx.x) * SquareArBlocks<N>() >= count) return;  // whole CTA
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int c = warp % 3, grp = warp / 3;
  const int unit = lane / N, r = lane % N;
  const int item = (blockIdx.x * kSquareArGroups + grp) * UPW + unit;
  const bool active = item < count;
  float* tile = s_tile[grp][c][unit];
  const uint32_t pk = list[active ? item : 0];
  const int bx = pk & 0xFFFF, by = pk >> 16;
  const size_t row = c * size_t(g.PW) * g.PH + size_t(by * 8 + r) * g.PW +
                     bx * 8;
  float X[N], D[N], Y[N];
#pragma unroll
  for (int x = 0; x < N; x += 4) {
    const float4 a = *reinterpret_cast<const float4*>(f.filt + row + x);
    const float4 o = *reinterpret_cast<const float4*>(f.idct + row + x);
    X[x] = o.x, X[x + 1] = o.y, X[x + 2] = o.z, X[x + 3] = o.w;
    D[x] = a.x - o.x, D[x + 1] = a.y - o.y;
    D[x + 2] = a.z - o.z, D[x + 3] = a.w - o.w;
  }
  const int type = f.acs[by * g.Bx + bx] >> 4;
  const ArBlockInfo info = ArInfo(g, f, s, bx, by, type);
  const float* dm = c == 0 ? info.dm[0] : c == 1 ? info.dm[1] : info.dm[2];
  DctRow<N>(D, Y);
  PutCol<N>(tile, r, Y);
  __syncwarp();
  GetRow<N>(tile, r, D);
  DctCol<N>(D, Y);
  __syncwarp();
  // This channel's clamp ratios of coefficient row k = r.
  float* ratio = s_ratio[grp][0][unit] + r * (N + 1);
  constexpr int channel = UPW * tile_size;
  LoadIntervals<N>(dm + r * N, info.inv_quant_ac, D);
  if (r < cov) {
#pragma unroll
    for (int l = 0; l < cov; ++l) D[l] = LlfScale(type, l, r) * s.mul_dc[c];
  }
#pragma unroll
  for (int l = 0; l < N; ++l) ratio[c * channel + l] = ClampRatio(Y[l], D[l]);
  __syncthreads();
  const size_t tape_row = CoefOffset(g, bx, by, cov, r * N);
  uint8_t* tape =
      f.clamp_tape && active && c == 0 ? f.clamp_tape + tape_row : nullptr;
  const uint8_t* tin =
      f.clamp_tape_in && active ? f.clamp_tape_in + tape_row : nullptr;
#pragma unroll
  for (int l = 0; l < N; ++l) {
    // The minimum over the channels.
    const float rt0 = ratio[l], rt1 = ratio[channel + l],
                rt2 = ratio[2 * channel + l];
    float mr = 1.0f;
    int arg = -1;
    if (rt0 < mr) mr = rt0, arg = 0;
    if (rt1 < mr) mr = rt1, arg = 1;
    if (rt2 < mr) mr = rt2, arg = 2;
    uint8_t code = arg < 0 ? 0 : mr == 0.0f ? 4 : uint8_t(arg + 1);
    if (tin) {
      code = tin[l];
      mr = TapeRatio(code, rt0, rt1, rt2);
    }
    if (tape) tape[l] = code;
    Y[l] = Y[l] * mr;
  }
  IdctRow<N>(Y, D);
  PutRow<N>(tile, r, D);
  __syncwarp();
  GetCol<N>(tile, r, Y);
  IdctRow<N>(Y, D);
  if (active) {
#pragma unroll
    for (int x = 0; x < N; x += 4) {
      *reinterpret_cast<float4*>(f.filt + row + x) =
          make_float4(D[x] + X[x], D[x + 1] + X[x + 1], D[x + 2] + X[x + 2],
                      D[x + 3] + X[x + 3]);
    }
  }
}

// ---------------------------------------------------------------------------
// DCT32X32 in the plain FP32 form. Four warps take one block and channel:
// lane r of every warp holds row r (or column r) of the 32 x 32 matrix in
// registers and warp w forms the pass's outputs 8 w .. 8 w + 7 of it, with
// the transform matrix read as 16-byte broadcasts from shared memory (fully
// unrolled rows with constant operands, as for 16x16, would be 130 KB of
// code). The transposes between the passes go through two padded tiles, each
// written again only after the barrier that follows its last reads. Every
// output is the sequential sum (index 0..31, separate multiply and add) of
// the row-major formulation, so results are bit-identical to it.
//
// Bound by the FP32 pipe and the issue slots of the row and matrix reads: at
// 3001x2003 with 89% of the area in such blocks the inverse's 8192 rounded
// operations per lane, block and channel take 0.11 ms at one per clock. A CTA
// per block with both operands of every product in shared memory took 0.565
// ms there (clamp 0.544); this split takes 0.221 (0.265), with scalar instead
// of packed products 0.244 (0.291), and 9 us instead of 49 on a 256x256 frame
// of mixed blocks. One warp per item, or per two items, without barriers:
// 0.248 and 0.223 ms there (scalar products), but 18 and 31 us on small
// frames, and 72 instead of 46 us at 1000x1000, where its longer turns leave
// the last wave empty.
namespace square32 {

constexpr int kN = 32;
constexpr int kStride = kN + 1;
constexpr int kTile = kN * kStride;
constexpr int kOut = 8;  // outputs per lane and pass
constexpr int kArThreads = 3 * kSquareThreads;

// The forward or inverse matrix of the tables, row-major.
__device__ __forceinline__ void LoadMat(float* m, const float* table) {
  const float4* src = reinterpret_cast<const float4*>(table + MatOffset(kN));
  for (int i = threadIdx.x; i < kN * kN / 4; i += blockDim.x) {
    reinterpret_cast<float4*>(m)[i] = src[i];
  }
}

// Rows 8 w .. 8 w + 7 of the matrix times the lane's vector.
__device__ __forceinline__ void Pass(const float* m, int w,
                                     const float (&v)[kN], float (&o)[kOut]) {
#pragma unroll
  for (int h = 0; h < kOut; h += 4) {
    const float* row = m + (kOut * w + h) * kN;
#pragma unroll
    for (int u = 0; u < 4; ++u) o[h + u] = 0.f;
#pragma unroll
    for (int i = 0; i < kN; i += 4) {
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        const float4 c = *reinterpret_cast<const float4*>(row + u * kN + i);
        float p[4];
        Mul2(p[0], p[1], v[i], v[i + 1], c.x, c.y);
        Mul2(p[2], p[3], v[i + 2], v[i + 3], c.z, c.w);
#pragma unroll
        for (int q = 0; q < 4; ++q) o[h + u] += p[q];
      }
    }
  }
}

__device__ __forceinline__ void Row(const float* t, int r, float (&v)[kN]) {
#pragma unroll
  for (int i = 0; i < kN; ++i) v[i] = t[r * kStride + i];
}
__device__ __forceinline__ void Col(const float* t, int r, float (&v)[kN]) {
#pragma unroll
  for (int i = 0; i < kN; ++i) v[i] = t[i * kStride + r];
}
__device__ __forceinline__ void PutRow(float* t, int r, int w,
                                       const float (&o)[kOut]) {
#pragma unroll
  for (int i = 0; i < kOut; ++i) t[r * kStride + kOut * w + i] = o[i];
}
__device__ __forceinline__ void PutCol(float* t, int r, int w,
                                       const float (&o)[kOut]) {
#pragma unroll
  for (int i = 0; i < kOut; ++i) t[(kOut * w + i) * kStride + r] = o[i];
}
// Eight floats at a 16-byte aligned address.
__device__ __forceinline__ void Load(const float* p, float (&v)[kOut]) {
  const float4 a = *reinterpret_cast<const float4*>(p);
  const float4 b = *reinterpret_cast<const float4*>(p + 4);
  v[0] = a.x, v[1] = a.y, v[2] = a.z, v[3] = a.w;
  v[4] = b.x, v[5] = b.y, v[6] = b.z, v[7] = b.w;
}
__device__ __forceinline__ void Store(float* p, const float (&v)[kOut]) {
  *reinterpret_cast<float4*>(p) = make_float4(v[0], v[1], v[2], v[3]);
  *reinterpret_cast<float4*>(p + 4) = make_float4(v[4], v[5], v[6], v[7]);
}

// tsDCT of the pixel rows in t0: coefficients (r, 8 w ..) in `o`.
__device__ __forceinline__ void Forward(const float* b, const float* t0,
                                        float* t1, int r, int w,
                                        float (&o)[kOut]) {
  float v[kN];
  __syncthreads();
  Row(t0, r, v);
  Pass(b, w, v, o);
  PutCol(t1, r, w, o);
  __syncthreads();
  Row(t1, r, v);
  Pass(b, w, v, o);
#pragma unroll
  for (int i = 0; i < kOut; ++i) o[i] = o[i] * (1.0f / float(kN * kN));
}
// tsIDCT of the coefficient rows in t0: pixels (r, 8 w ..) in `o`.
__device__ __forceinline__ void Inverse(const float* a, const float* t0,
                                        float* t1, int r, int w,
                                        float (&o)[kOut]) {
  float v[kN];
  __syncthreads();
  Row(t0, r, v);
  Pass(a, w, v, o);
  PutRow(t1, r, w, o);
  __syncthreads();
  Col(t1, r, v);
  Pass(a, w, v, o);
}

}  // namespace square32

// HF prediction + AddBlockExceptLFAndLLFTo + IDCT, a CTA per (block, channel).
__global__ void __launch_bounds__(kSquareThreads)
    k_square32_idct(Geo g, DevFrame f, const uint32_t* list, int predict_hf) {
  PdlLaunchDependents();
  PdlTail pdl_tail;
  using namespace square32;
  __shared__ __align__(16) float a[kN * kN], b[kN * kN];
  __shared__ float t0[kTile], t1[kTile];
  const int r = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int c = blockIdx.x % 3;
  const uint32_t pk = list[blockIdx.x / 3];
  const int bx = pk & 0xFFFF, by = pk >> 16;
  float x[kOut], o[kOut];
  Load(f.ac + c * size_t(g.ac_stride) * g.By +
           square::CoefRowOffset(g, bx, by, kN, r) + kOut * w,
       x);
  LoadMat(a, g_t.idct);
  if (predict_hf) {
    LoadMat(b, g_t.dct);
    const int gi = (by >> 6) * g.Gx + (bx >> 6);
    const float* pred = f.pred2x2_g + gi * kG2GroupFloats + c * kG2 * kG2;
    UpsampleRow<kOut>(pred, (bx & 63) * 8 + kOut * w, (by & 63) * 8 + r, o);
    PutRow(t0, r, w, o);
    Forward(b, t0, t1, r, w, o);
    if (r >= 8 || w >= 1) {  // all but the 8 x 8 low frequencies
#pragma unroll
      for (int i = 0; i < kOut; ++i) x[i] += o[i];
    }
  }
  PutRow(t0, r, w, x);
  Inverse(a, t0, t1, r, w, o);
  Store(f.idct + c * size_t(g.PW) * g.PH + size_t(by * 8 + r) * g.PW + bx * 8 +
            kOut * w,
        o);
}

// AdaptiveReconstruction clamp of DCT32X32 blocks
// (pik/adaptive_reconstruction.cc:128-244, 334-471): a CTA per block, four
// warps per channel; the channels' ratios meet in shared memory. `count` is
// read from device memory (k_epf_plan).
__global__ void __launch_bounds__(square32::kArThreads, 3)
    k_square32_ar(Geo g, DevFrame f, FrameScalars s, const uint32_t* list,
                  const int* count_ptr) {
  PdlLaunchDependents();
  PdlTail pdl_tail;
  using namespace square32;
  constexpr int cov = kN / 8;
  __shared__ __align__(16) float a[kN * kN], b[kN * kN];
  __shared__ float t0[3][kTile], t1[3][kTile];
  if (int(blockIdx.x) >= *count_ptr) return;  // whole CTA
  const int r = threadIdx.x & 31, w = (threadIdx.x >> 5) & 3;
  const int c = threadIdx.x / kSquareThreads;
  const uint32_t pk = list[blockIdx.x];
  const int bx = pk & 0xFFFF, by = pk >> 16;
  const size_t row = c * size_t(g.PW) * g.PH + size_t(by * 8 + r) * g.PW +
                     bx * 8 + kOut * w;
  float x[kOut], y[kOut], o[kOut];
  Load(f.filt + row, y);
  Load(f.idct + row, x);
  LoadMat(a, g_t.idct);
  LoadMat(b, g_t.dct);
  const ArBlockInfo info = ArInfo(g, f, s, bx, by, kDCT32X32);
  const float* dm = c == 0 ? info.dm[0] : c == 1 ? info.dm[1] : info.dm[2];
  const int e0 = r * kN + kOut * w;
#pragma unroll
  for (int i = 0; i < kOut; ++i) y[i] = y[i] - x[i];
  PutRow(t0[c], r, w, y);
  Forward(b, t0[c], t1[c], r, w, y);
  // This channel's ratios, then the minimum over the channels.
  LoadIntervals<kOut>(dm + e0, info.inv_quant_ac, o);
  if (r < cov && w == 0) {
#pragma unroll
    for (int i = 0; i < cov; ++i) o[i] = c_t.ar_llf32[r][i] * s.mul_dc[c];
  }
#pragma unroll
  for (int i = 0; i < kOut; ++i) o[i] = ClampRatio(y[i], o[i]);
  PutRow(t0[c], r, w, o);
  __syncthreads();
  const size_t to = CoefOffset(g, bx, by, cov, e0);
#pragma unroll
  for (int i = 0; i < kOut; ++i) {
    const int p = r * kStride + kOut * w + i;
    const float r0 = t0[0][p], r1 = t0[1][p], r2 = t0[2][p];
    float mr = 1.0f;
    int arg = -1;
    if (r0 < mr) mr = r0, arg = 0;
    if (r1 < mr) mr = r1, arg = 1;
    if (r2 < mr) mr = r2, arg = 2;
    if (f.clamp_tape || f.clamp_tape_in) {
      uint8_t code = arg < 0 ? 0 : mr == 0.0f ? 4 : uint8_t(arg + 1);
      if (f.clamp_tape_in) {
        code = f.clamp_tape_in[to + i];
        mr = TapeRatio(code, r0, r1, r2);
      }
      if (f.clamp_tape && c == 0) f.clamp_tape[to + i] = code;
    }
    y[i] = y[i] * mr;
  }
  PutRow(t1[c], r, w, y);
  Inverse(a, t1[c], t0[c], r, w, o);
#pragma unroll
  for (int i = 0; i < kOut; ++i) o[i] = o[i] + x[i];
  Store(f.filt + row, o);
}

}  // namespace pikgpu
