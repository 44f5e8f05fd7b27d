// Segment-parallel decode for the training / offline path, plain FP32
// (kernel templates; each decoder variant is instantiated in its own
// translation unit, decode_v<width>c<channels>.cu).
//
//   decode_fwd_plain  gather + integrate + mlp1 + mlp2 + sigmoid per segment
//   decode_bwd_plain  recompute + backprop through the MLPs and the integral:
//                     feature-grid gradient (vector atomics) and MLP weight
//                     gradient (register accumulators)
//
// Reference semantics: model/diver.py:159-180 (decode), utils/integrator.py:
// 62-112 (integral).
//
// Both kernels are bound by FP32 FMA issue, so everything is laid out to feed
// FMAs from few shared-memory loads and to need no barrier wider than a warp
// in the layer chain.  A warp owns a tile of SEGS (32 or 16) segments.  Its
// activations are feature-major, [feature][segment] with rows of SEGS + 4
// floats: a layer is a register-tiled product in which lane (tx, ty) =
// (lane % 8, lane / 8) computes outputs tx + 8 m of its SEGS / 4 consecutive
// segments, one 16-byte load per 4 segments and one per 4 outputs for each
// input feature (10.7 or more FMAs per load; one thread per segment with
// broadcast weights, as these kernels were before, is 3.6).  The rows' padding
// makes every access of the product, of its result's store and of the weight
// gradients (8 lanes on 8 consecutive rows) free of bank conflicts beyond
// the 16-byte minimum.  Every output is the same chain of FMAs, inputs in
// order from its bias, whatever the tiling: results do not depend on it.
// Measured on a GB300 against one thread per segment (128-thread CTAs, the
// backward's with one CTA of 2 or 4 warps per SM and its weight gradients in
// shared memory): a 2035-ray DIVeR32 training step on a 160^3 grid, backward
// 1068 -> 362 us, forward 196 -> 115 us; a 1024-ray DIVeR64 step over 64
// channels on a 192^3 grid, backward 2853 -> 600 us.  Packed FMAs since: 338
// and 107 us; with the forward's record (REC_SEGS) 237 and 124.
#pragma once
#include "common.cuh"
#include "integrate.cuh"
#include "mlp.cuh"
#include "tc.cuh"

#include <algorithm>

namespace dv {

constexpr int MAX_LAYERS = 5;

struct DecodeArgs {
  const float* grid;
  int nvx, nvy, nvz;
  const float* seg;        // [S][6]
  const int* seg_ray;      // [S]
  long long S;             // segment count, or capacity when S_dev is set
  const int64_t* S_dev;    // optional device-held count (clamped to S)
  const int64_t* offsets;  // [B+1]
  int B;
  const float* params;     // packed plain layout
  int n_params;            // multiple of 4
  int w_off[MAX_LAYERS];
  int b_off[MAX_LAYERS];
  const float* dirs;       // [B][3]
  float* pe_feat;          // [B][28]   PE values
  float* pe_out;           // [B][W]    b + PE @ Wt(pe rows) of mlp2's first layer
  float4* out4;            // [S] (sigma_raw, r, g, b)
  const float4* d4;        // [S] (dL/dsigma_raw, dL/dr, dL/dg, dL/db)
  float* grad_grid;        // accumulated
  float* grad_params;      // accumulated, packed layout
  int white_back;
  float* rgb;              // [B][3]
  float* t_final;          // [B] or null
  float* reg_sum;          // [B] or null: sum of log(1 + sigma^2 / 0.5)
  const float* g_rgb;      // [B][3] dL/drgb
  float reg_coef;          // l_s / (B * M), or l_s / B with reg_scale = 1 / M
  const float* reg_scale;  // optional device factor on reg_coef
  float* acts;             // optional record of the forward's activations (REC_FLOATS a tile)
  float* alpha_map;        // occupancy extraction: [N][N][N] max of segment weights
  int occ_n, occ_pad;
};

// Layer indices: 0 .. D1-1 hidden layers of mlp1 (first: C -> W), D1: mlp1
// output (W -> W+1, sigma and the hidden feature), D1+1: mlp2 first
// (W+27 -> W), D1+2: mlp2 output (W -> 3).

// Weights in shared memory (floats).  Every hidden layer is [in][LDW] with
// LDW = W + 4 and its W outputs permuted (wpos) so that the 4 outputs
// tx + 8 i (i = 0..3) of a lane are one float4; the padding keeps loads down a
// column (8 lanes on 8 consecutive input rows, the backward) free of bank
// conflicts too, so one copy serves both directions.
template <int C, int W, int D1>
struct PlainWeights {
  static constexpr int LDW = W + 4;
  static constexpr int l0 = 0;                                   // C -> W
  static constexpr int l1 = l0 + C * LDW;                        // W -> W (D1 = 2)
  static constexpr int wh = l1 + (D1 == 2 ? W * LDW : 0);        // mlp1 output, hidden part
  static constexpr int w2 = wh + W * LDW;                        // mlp2 first layer, hidden rows
  static constexpr int sig = w2 + W * LDW;                       // mlp1 output, density column [W]
  static constexpr int w3 = sig + W;                             // [W][4]
  static constexpr int b0 = w3 + 4 * W;
  static constexpr int b1 = b0 + W;
  static constexpr int bh = b1 + W;
  static constexpr int b3 = bh + W;                              // rgb, then the density bias
  static constexpr int size = b3 + 4;
};

__host__ __device__ constexpr int wpos(int j) { return (j & ~31) + (j & 7) * 4 + ((j & 31) >> 3); }

template <int C, int W, int D1>
__device__ __forceinline__ void stage_weights(const DecodeArgs& a, float* sw) {
  using P = PlainWeights<C, W, D1>;
  const int t = threadIdx.x, n = blockDim.x;
  for (int i = t; i < C * W; i += n) sw[P::l0 + (i / W) * P::LDW + wpos(i % W)] = __ldg(a.params + a.w_off[0] + i);
  if (D1 == 2)
    for (int i = t; i < W * W; i += n) sw[P::l1 + (i / W) * P::LDW + wpos(i % W)] = __ldg(a.params + a.w_off[1] + i);
  for (int i = t; i < W * W; i += n) {
    const int k = i / W, j = i % W;
    sw[P::wh + k * P::LDW + wpos(j)] = __ldg(a.params + a.w_off[D1] + k * (W + 4) + 1 + j);
    sw[P::w2 + k * P::LDW + wpos(j)] = __ldg(a.params + a.w_off[D1 + 1] + i);
  }
  for (int i = t; i < W; i += n) {
    sw[P::sig + i] = __ldg(a.params + a.w_off[D1] + i * (W + 4));
    sw[P::b0 + i] = __ldg(a.params + a.b_off[0] + i);
    if (D1 == 2) sw[P::b1 + i] = __ldg(a.params + a.b_off[1] + i);
    sw[P::bh + i] = __ldg(a.params + a.b_off[D1] + 1 + i);
  }
  for (int i = t; i < 4 * W; i += n) sw[P::w3 + i] = __ldg(a.params + a.w_off[D1 + 2] + i);
  if (t < 3) sw[P::b3 + t] = __ldg(a.params + a.b_off[D1 + 2] + t);
  if (t == 3) sw[P::b3 + 3] = __ldg(a.params + a.b_off[D1]);
}

// Corner weights and rows of a segment, computed once by one lane and read by
// the lanes that gather (and scatter) its channels: w[8], then the lower
// corner's row and the row steps to the upper corner along x, y and z (0
// where it is clamped).  Rows fit 32 bits: 2^32 rows of 32 channels are twice
// the device's memory.
constexpr int COEF = 12;

template <int SEGS>
__device__ __forceinline__ void put_coefs(const DecodeArgs& a, long long S, long long s0, float* coef) {
  const int lane = threadIdx.x & 31;
  if (lane < SEGS && s0 + lane < S) {
    const float* sg = a.seg + (s0 + lane) * 6;
    const SegCorner sc = segment_corners(__ldg(sg), __ldg(sg + 1), __ldg(sg + 2), __ldg(sg + 3), __ldg(sg + 4),
                                         __ldg(sg + 5), a.nvx, a.nvy, a.nvz);
    float4* c = reinterpret_cast<float4*>(coef + lane * COEF);
    c[0] = make_float4(sc.w[0], sc.w[1], sc.w[2], sc.w[3]);
    c[1] = make_float4(sc.w[4], sc.w[5], sc.w[6], sc.w[7]);
    reinterpret_cast<uint4*>(c)[2] =
        make_uint4(((unsigned)sc.z * a.nvy + sc.y) * a.nvx + sc.x, sc.x1 - sc.x, (sc.y1 - sc.y) * a.nvx,
                   (unsigned)(sc.z1 - sc.z) * a.nvx * a.nvy);
  }
}

__device__ __forceinline__ unsigned coef_row(const uint4 m, int j) {
  return m.x + ((j & 1) ? m.y : 0u) + ((j & 2) ? m.z : 0u) + ((j & 4) ? m.w : 0u);
}

// Feature rows of the tile: C/4 lanes per segment, each integrating 4 channels
// (coalesced corner rows), written feature-major.  The 4 channels go out in an
// order that rotates with the channel quad, so that the quads, 4 rows apart,
// fall into different banks.
template <int C, int SEGS>
__device__ __forceinline__ void gather_warp(const DecodeArgs& a, long long S, long long s0, const float* coef, float* X) {
  constexpr int TPS = C / 4, SPP = 32 / TPS, LD = SEGS + 4;
  const int lane = threadIdx.x & 31, q = lane % TPS;
#pragma unroll 1
  for (int p = 0; p < SEGS / SPP; ++p) {
    const int ls = p * SPP + lane / TPS;
    float4 f = make_float4(0.f, 0.f, 0.f, 0.f);
    if (s0 + ls < S) {
      const float4 wa = *reinterpret_cast<const float4*>(coef + ls * COEF);
      const float4 wb = *reinterpret_cast<const float4*>(coef + ls * COEF + 4);
      const uint4 m = *reinterpret_cast<const uint4*>(coef + ls * COEF + 8);
      const float w[8] = {wa.x, wa.y, wa.z, wa.w, wb.x, wb.y, wb.z, wb.w};
      float4 v[8];
#pragma unroll
      for (int j = 0; j < 8; ++j) v[j] = ldg4(a.grid + (long long)coef_row(m, j) * C + 4 * q);
#pragma unroll
      for (int j = 0; j < 8; ++j) fma4(f, w[j], v[j]);
    }
    const int rot = (q >> 1) & 3;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int c = (i + rot) & 3;
      X[(4 * q + c) * LD + ls] = c < 2 ? (c == 0 ? f.x : f.y) : (c == 2 ? f.z : f.w);
    }
  }
}

template <int N>
__device__ __forceinline__ void load_segs(const float* p, float* v) {
#pragma unroll
  for (int i = 0; i < N; i += 4) {
    const float4 x = *reinterpret_cast<const float4*>(p + i);
    v[i] = x.x;
    v[i + 1] = x.y;
    v[i + 2] = x.z;
    v[i + 3] = x.w;
  }
}

// Accumulators of two consecutive segments as one packed pair.  The products
// below run on packed FMAs, both halves with the same weight: half the issue
// slots for the same rounding (2035-ray DIVeR32 step: backward 358 -> 341 us,
// forward 115 -> 108 us).
template <int M, int SPT>
struct AccPairs {
  unsigned long long v[M][SPT / 2];
  __device__ __forceinline__ explicit AccPairs(const float (&a)[M][SPT]) {
#pragma unroll
    for (int m = 0; m < M; ++m)
#pragma unroll
      for (int s = 0; s < SPT; s += 2) v[m][s / 2] = f32x2(a[m][s], a[m][s + 1]);
  }
  __device__ __forceinline__ void to(float (&a)[M][SPT]) const {
#pragma unroll
    for (int m = 0; m < M; ++m)
#pragma unroll
      for (int s = 0; s < SPT; s += 2) {
        const float2 f = f32x2_get(v[m][s / 2]);
        a[m][s] = f.x;
        a[m][s + 1] = f.y;
      }
  }
  __device__ __forceinline__ void fma(int m, const unsigned long long (&x)[SPT / 2], float w) {
    const unsigned long long ww = f32x2(w, w);
#pragma unroll
    for (int s = 0; s < SPT / 2; ++s) v[m][s] = fma_f32x2(x[s], ww, v[m][s]);
  }
};

template <int N>
__device__ __forceinline__ void load_pairs(const float* p, unsigned long long (&v)[N / 2]) {
#pragma unroll
  for (int i = 0; i < N; i += 4) {
    const float4 x = *reinterpret_cast<const float4*>(p + i);
    v[i / 2] = f32x2(x.x, x.y);
    v[i / 2 + 1] = f32x2(x.z, x.w);
  }
}

// acc[m][s] += sum over k of X[k][segment s] * wl[k][output tx + 8 m].
template <int K, int W, int SEGS>
__device__ __forceinline__ void layer_fwd(const float* X, const float* wl, float (&acc)[W / 8][SEGS / 4]) {
  constexpr int SPT = SEGS / 4, LD = SEGS + 4, LDW = W + 4;
  const int lane = threadIdx.x & 31, tx = lane & 7, ty = lane >> 3;
  const float* xp = X + SPT * ty;
  const float* wp = wl + 4 * tx;
  AccPairs<W / 8, SPT> c(acc);
#pragma unroll 4
  for (int k = 0; k < K; ++k) {
    unsigned long long x[SPT / 2];
    load_pairs<SPT>(xp + k * LD, x);
#pragma unroll
    for (int h = 0; h < W / 32; ++h) {
      const float4 w = *reinterpret_cast<const float4*>(wp + k * LDW + 32 * h);
      c.fma(4 * h, x, w.x);
      c.fma(4 * h + 1, x, w.y);
      c.fma(4 * h + 2, x, w.z);
      c.fma(4 * h + 3, x, w.w);
    }
  }
  c.to(acc);
}

template <int M, int SPT>
__device__ __forceinline__ void set_acc(float (&acc)[M][SPT], const float* bias) {
  const int tx = threadIdx.x & 7;
#pragma unroll
  for (int m = 0; m < M; ++m) {
    const float b = bias ? bias[tx + 8 * m] : 0.f;
#pragma unroll
    for (int s = 0; s < SPT; ++s) acc[m][s] = b;
  }
}

// Writes the lane's outputs into the feature-major tile (after every lane of
// the warp has read what it replaces, and before any reads the new rows).
template <int M, int SPT, bool RELU>
__device__ __forceinline__ void put_acc(float* X, const float (&acc)[M][SPT]) {
  constexpr int LD = 4 * SPT + 4;
  const int lane = threadIdx.x & 31, tx = lane & 7, ty = lane >> 3;
  __syncwarp();
#pragma unroll
  for (int m = 0; m < M; ++m) {
    float v[SPT];
#pragma unroll
    for (int s = 0; s < SPT; ++s) v[s] = RELU ? fmaxf(acc[m][s], 0.f) : acc[m][s];
#pragma unroll
    for (int s = 0; s < SPT; s += 4)
      *reinterpret_cast<float4*>(X + (tx + 8 * m) * LD + SPT * ty + s) = make_float4(v[s], v[s + 1], v[s + 2], v[s + 3]);
  }
  __syncwarp();
}

// Adds each segment's per-ray term (bias + PE part of mlp2's first layer).
// ray: lane i holds segment i's ray; a tile inside one ray loads it once.
template <int W, int SPT>
__device__ __forceinline__ void add_ray_term(const DecodeArgs& a, int ray, float (&acc)[W / 8][SPT]) {
  const int lane = threadIdx.x & 31, tx = lane & 7, ty = lane >> 3;
  const int r0 = __shfl_sync(0xffffffffu, ray, 0);
  if (__all_sync(0xffffffffu, ray == r0)) {
#pragma unroll
    for (int m = 0; m < W / 8; ++m) {
      const float p = __ldg(a.pe_out + (long long)r0 * W + tx + 8 * m);
#pragma unroll
      for (int s = 0; s < SPT; ++s) acc[m][s] += p;
    }
  } else {
#pragma unroll
    for (int s = 0; s < SPT; ++s) {
      const int r = __shfl_sync(0xffffffffu, ray, SPT * ty + s);
#pragma unroll
      for (int m = 0; m < W / 8; ++m) acc[m][s] += __ldg(a.pe_out + (long long)r * W + tx + 8 * m);
    }
  }
}

// Ray of this lane's segment; lanes without one get the tile's first ray.
template <int SEGS>
__device__ __forceinline__ int tile_ray(const DecodeArgs& a, long long S, long long s0) {
  const int lane = threadIdx.x & 31;
  const int r0 = __ldg(a.seg_ray + s0);
  return lane < SEGS && s0 + lane < S ? __ldg(a.seg_ray + s0 + lane) : r0;
}

// Density (raw) and colour logits of the lane's segment from its columns of
// the last mlp1 activation (AL) / the last mlp2 activation (A4).
template <int W, int LD>
__device__ __forceinline__ float density(const float* sig, float bias, const float* AL, int seg) {
  float v = bias;
#pragma unroll 4
  for (int k = 0; k < W; k += 4) {
    const float4 w = *reinterpret_cast<const float4*>(sig + k);
    v = fmaf(AL[k * LD + seg], w.x, v);
    v = fmaf(AL[(k + 1) * LD + seg], w.y, v);
    v = fmaf(AL[(k + 2) * LD + seg], w.z, v);
    v = fmaf(AL[(k + 3) * LD + seg], w.w, v);
  }
  return v;
}

template <int W, int LD>
__device__ __forceinline__ float3 colour(const float* w3, const float* b3, const float* A4, int seg) {
  float3 o = make_float3(b3[0], b3[1], b3[2]);
#pragma unroll 8
  for (int k = 0; k < W; ++k) {
    const float x = A4[k * LD + seg];
    const float4 w = *reinterpret_cast<const float4*>(w3 + 4 * k);
    o.x = fmaf(x, w.x, o.x);
    o.y = fmaf(x, w.y, o.y);
    o.z = fmaf(x, w.z, o.z);
  }
  return make_float3(sigmoidf_acc(o.x), sigmoidf_acc(o.y), sigmoidf_acc(o.z));
}

// A training forward's record for the backward: per tile of REC_SEGS segments,
// the features and every relu activation as they lie in a warp's shared memory,
// rows of REC_LD.  The backward reads it in place of gathering and recomputing
// (a third of its FMAs, and the gather's latency).  Measured, a 2035-ray DIVeR32
// step on a 160^3 grid: backward 338 -> 237 us, forward 107 -> 124 us.
constexpr int REC_SEGS = 32, REC_LD = REC_SEGS + 4;
template <int C, int W, int D1>
constexpr int REC_FLOATS = (C + (D1 + 1) * W) * REC_LD;

// Copies `rows` rows of the warp's tile X out (its next writer calls
// saved_rows first).
__device__ __forceinline__ void save_rows(float* dst, const float* X, int rows) {
  tc::fence_async_smem();
  __syncwarp();
  if ((threadIdx.x & 31) == 0) {
    tc::bulk_store(dst, X, (uint32_t)(rows * REC_LD * 4));
    tc::bulk_commit();
  }
}
__device__ __forceinline__ void saved_rows() {
  if ((threadIdx.x & 31) == 0) tc::bulk_wait_read();
  __syncwarp();
}

// Shared memory of decode_fwd_plain (floats): weights, then per warp its
// activation tile and its segments' coefficients.
template <int C, int W, int D1, int SEGS>
struct FwdSmem {
  static constexpr int X = (C > W ? C : W) * (SEGS + 4);
  static constexpr int warp = X + SEGS * COEF;
};

// Warps take tiles independently (tile = block + grid * warp slot, so a
// launch with few tiles spreads over all SMs); nothing in the loop is wider
// than a warp.
template <int C, int W, int D1, int SEGS, int WARPS, int CTAS, bool SAVE>
__global__ void __launch_bounds__(32 * WARPS, CTAS) decode_fwd_plain(const DecodeArgs a) {
  using P = PlainWeights<C, W, D1>;
  using L = FwdSmem<C, W, D1, SEGS>;
  constexpr int LD = SEGS + 4;
  extern __shared__ __align__(16) float smem[];
  float* sw = smem;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  float* X = smem + P::size + warp * L::warp;
  float* coef = X + L::X;
  stage_weights<C, W, D1>(a, sw);
  __syncthreads();
  const long long S = segment_total(a.S, a.S_dev);
  const long long tiles = (S + SEGS - 1) / SEGS;
  for (long long tile = blockIdx.x + (long long)gridDim.x * warp; tile < tiles; tile += (long long)gridDim.x * WARPS) {
    const long long s0 = tile * SEGS;
    put_coefs<SEGS>(a, S, s0, coef);
    __syncwarp();
    gather_warp<C, SEGS>(a, S, s0, coef, X);
    float* rec = a.acts;
    if constexpr (SAVE) {
      static_assert(SEGS == REC_SEGS, "the record's tile");
      rec += tile * REC_FLOATS<C, W, D1>;
      save_rows(rec, X, C);
    } else {
      __syncwarp();
    }
    float acc[W / 8][SEGS / 4];
    set_acc(acc, sw + P::b0);
    layer_fwd<C, W, SEGS>(X, sw + P::l0, acc);
    if constexpr (SAVE) saved_rows();
    put_acc<W / 8, SEGS / 4, true>(X, acc);
    if constexpr (SAVE) save_rows(rec + C * LD, X, W);
    if constexpr (D1 == 2) {
      set_acc(acc, sw + P::b1);
      layer_fwd<W, W, SEGS>(X, sw + P::l1, acc);
      if constexpr (SAVE) saved_rows();
      put_acc<W / 8, SEGS / 4, true>(X, acc);
      if constexpr (SAVE) save_rows(rec + (C + W) * LD, X, W);
    }
    const float sigma = lane < SEGS ? density<W, LD>(sw + P::sig, sw[P::b3 + 3], X, lane) : 0.f;
    set_acc(acc, sw + P::bh);
    layer_fwd<W, W, SEGS>(X, sw + P::wh, acc);
    if constexpr (SAVE) saved_rows();
    put_acc<W / 8, SEGS / 4, false>(X, acc);
    set_acc(acc, nullptr);
    layer_fwd<W, W, SEGS>(X, sw + P::w2, acc);
    add_ray_term<W>(a, tile_ray<SEGS>(a, S, s0), acc);
    put_acc<W / 8, SEGS / 4, true>(X, acc);
    if constexpr (SAVE) save_rows(rec + (C + D1 * W) * LD, X, W);
    if (lane < SEGS && s0 + lane < S) {
      const float3 c = colour<W, LD>(sw + P::w3, sw + P::b3, X, lane);
      a.out4[s0 + lane] = make_float4(sigma, c.x, c.y, c.z);
    }
    if constexpr (SAVE) saved_rows();
    __syncwarp();  // the next gather overwrites the tile
  }
  if (SAVE && lane == 0) tc::bulk_wait_all();
}

// ---- backward ----------------------------------------------------------------

// acc[m][s] += sum over outputs j of wl[tx + 8 m][j] * D[j][segment s]: the
// gradient of a layer's inputs tx + 8 m.
template <int K, int W, int SEGS>
__device__ __forceinline__ void layer_bwd(const float* D, const float* wl, float (&acc)[K / 8][SEGS / 4]) {
  constexpr int SPT = SEGS / 4, LD = SEGS + 4, LDW = W + 4;
  const int lane = threadIdx.x & 31, tx = lane & 7, ty = lane >> 3;
  const float* dp = D + SPT * ty;
  const float* wp = wl + tx * LDW;
  AccPairs<K / 8, SPT> c(acc);
#pragma unroll
  for (int h = 0; h < W / 32; ++h)
#pragma unroll 2
    for (int g = 0; g < 8; ++g) {  // outputs 32 h + g + 8 i: 4 consecutive weights
      unsigned long long d[4][SPT / 2];
#pragma unroll
      for (int i = 0; i < 4; ++i) load_pairs<SPT>(dp + (32 * h + 8 * i + g) * LD, d[i]);
#pragma unroll
      for (int m = 0; m < K / 8; ++m) {
        const float4 w = *reinterpret_cast<const float4*>(wp + 8 * m * LDW + 32 * h + 4 * g);
        c.fma(m, d[0], w.x);
        c.fma(m, d[1], w.y);
        c.fma(m, d[2], w.z);
        c.fma(m, d[3], w.w);
      }
    }
  c.to(acc);
}

// The record of the SEGS segments from s0 on (all or half of one of its
// tiles) into the warp's shared memory; zeros past the last segment, where the
// record ends.
template <int ROWS, int SEGS>
__device__ __forceinline__ void load_record(float* dst, const float* rec, long long s0, long long S) {
  constexpr int Q = SEGS / 4, LD = SEGS + 4;
  const float* src = rec + s0 / REC_SEGS * (ROWS * REC_LD) + s0 % REC_SEGS;
  for (int i = threadIdx.x & 31; i < ROWS * Q; i += 32) {
    float* d = dst + i / Q * LD + i % Q * 4;
    if (s0 < S)
      asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(tc::smem_u32(d)),
                   "l"(src + i / Q * REC_LD + i % Q * 4)
                   : "memory");
    else
      *reinterpret_cast<float4*>(d) = make_float4(0.f, 0.f, 0.f, 0.f);
  }
  asm volatile("cp.async.wait_all;" ::: "memory");
  __syncwarp();
}

// Writes the input gradients over the activation they belong to, zero where
// that relu activation is zero.
template <int M, int SPT>
__device__ __forceinline__ void put_masked(float* X, const float (&acc)[M][SPT]) {
  constexpr int LD = 4 * SPT + 4;
  const int lane = threadIdx.x & 31, tx = lane & 7, ty = lane >> 3;
  __syncwarp();
#pragma unroll
  for (int m = 0; m < M; ++m)
#pragma unroll
    for (int s = 0; s < SPT; s += 4) {
      float4* x = reinterpret_cast<float4*>(X + (tx + 8 * m) * LD + SPT * ty + s);
      const float4 r = *x;
      *x = make_float4(r.x > 0.f ? acc[m][s] : 0.f, r.y > 0.f ? acc[m][s + 1] : 0.f, r.z > 0.f ? acc[m][s + 2] : 0.f,
                       r.w > 0.f ? acc[m][s + 3] : 0.f);
    }
  __syncwarp();
}

// acc[m][n] += sum over a tile's segments of act[ti + 8 m] * del[tj + 4 n]
// (act, del: the first rows of the block), ti = lane % 8, tj = lane / 8.
template <int NI, int NJ, int SEGS>
__device__ __forceinline__ void weight_grad(const float* act, const float* del, float (&acc)[NI][NJ]) {
  constexpr int LD = SEGS + 4;
  const int lane = threadIdx.x & 31;
  const float* ap = act + (lane & 7) * LD;
  const float* dp = del + (lane >> 3) * LD;
#pragma unroll 1
  for (int c = 0; c < SEGS; c += 4) {
    float4 x[NI];
#pragma unroll
    for (int m = 0; m < NI; ++m) x[m] = *reinterpret_cast<const float4*>(ap + 8 * m * LD + c);
#pragma unroll
    for (int n = 0; n < NJ; ++n) {
      const float4 d = *reinterpret_cast<const float4*>(dp + 4 * n * LD + c);
#pragma unroll
      for (int m = 0; m < NI; ++m) {
        acc[m][n] = fmaf(x[m].x, d.x, acc[m][n]);
        acc[m][n] = fmaf(x[m].y, d.y, acc[m][n]);
        acc[m][n] = fmaf(x[m].z, d.z, acc[m][n]);
        acc[m][n] = fmaf(x[m].w, d.w, acc[m][n]);
      }
    }
  }
}

template <int SEGS>
__device__ __forceinline__ float row_dot(const float* x, const float* y) {
  float v = 0.f;
#pragma unroll
  for (int c = 0; c < SEGS; c += 4) {
    const float4 p = *reinterpret_cast<const float4*>(x + c), q = *reinterpret_cast<const float4*>(y + c);
    v = fmaf(p.x, q.x, fmaf(p.y, q.y, fmaf(p.z, q.z, fmaf(p.w, q.w, v))));
  }
  return v;
}

// Sum of the row's entries whose bit in `m` is set.
template <int SEGS>
__device__ __forceinline__ float row_sum(const float* x, unsigned m) {
  float v = 0.f;
#pragma unroll
  for (int c = 0; c < SEGS; c += 4) {
    const float4 p = *reinterpret_cast<const float4*>(x + c);
    v += ((m >> c) & 1u ? p.x : 0.f) + ((m >> c) & 2u ? p.y : 0.f) + (((m >> c) & 4u ? p.z : 0.f) + ((m >> c) & 8u ? p.w : 0.f));
  }
  return v;
}

// Scatter of the tile's feature gradient (feature-major rows of X) into the
// corner rows: lane (run, q) takes channel quad q of a run of consecutive
// segments.  Consecutive segments of a ray usually sit in face-adjacent
// voxels: the four corner rows they share are added in registers and reach
// memory with one vector atomic instead of two.  A merge needs both voxels
// whole (upper corners not clamped) and lower corners one row step apart
// along one axis, so the merged rows are the same rows.
template <int C, int SEGS>
__device__ __forceinline__ void scatter_warp(const DecodeArgs& a, long long S, long long s0, const float* coef,
                                             const float* X) {
  constexpr int TPS = C / 4, HRUN = SEGS / (32 / TPS), LD = SEGS + 4;
  const int lane = threadIdx.x & 31, q = lane % TPS, first = (lane / TPS) * HRUN;
  const int rot = (q >> 1) & 3;
  float4 pend[8];
  uint4 pm = make_uint4(0u, 0u, 0u, 0u);
  bool have = false, pwhole = false;
  float* grid = a.grad_grid + 4 * q;
#pragma unroll 1
  for (int k = 0; k < HRUN; ++k) {
    const int ls = first + k;
    if (s0 + ls >= S) break;
    const float4 wa = *reinterpret_cast<const float4*>(coef + ls * COEF);
    const float4 wb = *reinterpret_cast<const float4*>(coef + ls * COEF + 4);
    const uint4 m = *reinterpret_cast<const uint4*>(coef + ls * COEF + 8);
    const float w[8] = {wa.x, wa.y, wa.z, wa.w, wb.x, wb.y, wb.z, wb.w};
    float g[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int c = (i + rot) & 3;
      const float v = X[(4 * q + c) * LD + ls];
#pragma unroll
      for (int u = 0; u < 4; ++u) g[u] = c == u ? v : g[u];
    }
    const bool whole = m.y != 0u && m.z != 0u && m.w != 0u;
    int axis = -1;
    bool up = false;
    if (have && whole && pwhole) {
      const unsigned d = m.x - pm.x, e = pm.x - m.x;
      if (d == m.y || e == m.y) axis = 0;
      if (d == m.z || e == m.z) axis = 1;
      if (d == m.w || e == m.w) axis = 2;
      up = d < e;
    }
    if (have) {
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        const bool shared = axis >= 0 && ((j >> axis) & 1) == (up ? 1 : 0);
        if (!shared) red_add4(grid + (long long)coef_row(pm, j) * C, pend[j]);
      }
    }
    float4 nx[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      float4 c = make_float4(w[j] * g[0], w[j] * g[1], w[j] * g[2], w[j] * g[3]);
      if (axis >= 0 && ((j >> axis) & 1) == (up ? 0 : 1)) {
        const float4 o = axis == 0 ? pend[j ^ 1] : (axis == 1 ? pend[j ^ 2] : pend[j ^ 4]);
        c.x += o.x;
        c.y += o.y;
        c.z += o.z;
        c.w += o.w;
      }
      nx[j] = c;
    }
#pragma unroll
    for (int j = 0; j < 8; ++j) pend[j] = nx[j];
    pm = m;
    pwhole = whole;
    have = true;
  }
  if (have) {
#pragma unroll
    for (int j = 0; j < 8; ++j) red_add4(grid + (long long)coef_row(pm, j) * C, pend[j]);
  }
}

// Shared memory of decode_bwd_plain (floats): weights, the folded layer, then
// per warp the activations (each overwritten by the gradient of its
// pre-activation), 4 rows (3 logit gradients, dL/dsigma) and coefficients.
// The flush reuses the warps' part for the gradients of the CTA.
template <int C, int W, int D1, int SEGS, int WARPS>
struct BwdSmem {
  using P = PlainWeights<C, W, D1>;
  static constexpr int LD = SEGS + 4;
  static constexpr int wf = P::size;  // [W][LDW]
  static constexpr int warps = wf + W * P::LDW;
  static constexpr int X0 = 0, A1 = X0 + C * LD, A2 = A1 + W * LD, A4 = A1 + D1 * W * LD, DS = A4 + W * LD;
  static constexpr int AL = D1 == 2 ? A2 : A1;  // last mlp1 activation
  static constexpr int coef = DS + 4 * LD;
  static constexpr int warp = coef + SEGS * COEF;
  static constexpr int size = warps + WARPS * warp;
  // flush, from `warps` on: the packed gradients with the folded layer in place of its two factors
  static constexpr int g0 = 0, g1 = g0 + C * W, gf = g1 + (D1 == 2 ? W * W : 0), gpe = gf + W * P::LDW;
  static constexpr int gs = gpe + PE_DIM * W, g3 = gs + W, gb0 = g3 + 4 * W, gb1 = gb0 + W, gb4 = gb1 + W;
  static constexpr int gb3 = gb4 + W, flush = gb3 + 4;
  static_assert(flush <= WARPS * warp, "the flush fits the warps' part");
};

// mlp1's output layer has no activation, so its hidden part WH and mlp2's
// first layer W2 act as one matrix WF = WH W2: with AL the activation before
// and delta the gradient after both,
//   dL/dAL  = delta WF^T (+ the density column),    GF = AL^T delta,
//   dL/dW2  = hidden^T delta = WH^T GF + bh (sum delta)^T,
//   dL/dWH  = AL^T (delta W2^T) = GF W2^T,   dL/dbh = W2 (sum delta),
// so the backward needs one product each way and one weight gradient less
// per segment; GF becomes the two gradients once per CTA.  The forward
// recompute keeps the two layers: its relu decisions are decode_fwd_plain's.
// dL/dW2's rounding stands against its two parts: where the hidden layer is r
// times smaller than WH^T A2 and bh, its relative error is about 5e-7 r
// (measured: r = 1 3e-7 to 1e-6, r = 26 5e-6 to 1.5e-5, r = 207 4e-5 to 1e-4;
// default initialisation has r below 1).
// The PE rows of mlp2's first layer see the same input along a ray: delta is
// summed over the tile's segments of a ray before the outer product.
//
// Weight gradients stay in registers for the CTA's life.  DIST false
// (DIVeR32): every warp accumulates all of them over its own segments.  DIST
// true (DIVeR64, 14 k gradients): warp w accumulates a block of each layer over
// the segments of all warps, so the warps step through the layers together.
template <int C, int W, int D1, int SEGS, int WARPS, bool DIST, bool SAVED>
__global__ void __launch_bounds__(32 * WARPS, 1) decode_bwd_plain(const DecodeArgs a) {
  using P = PlainWeights<C, W, D1>;
  using L = BwdSmem<C, W, D1, SEGS, WARPS>;
  constexpr int LD = L::LD, LDW = P::LDW, SPT = SEGS / 4, RW = W / 32;
  static_assert(!DIST || (WARPS == 8 && D1 == 1), "block assignment of the distributed weight gradients");
  // gradient blocks: all of [K][W] per warp, or 1/8 of it
  constexpr int NJ0 = DIST ? (C == 64 ? 4 : 2) : 8, NJF = DIST ? 4 : 8;
  extern __shared__ __align__(16) float smem[];
  float* sw = smem;
  float* wf = smem + L::wf;
  const int t = threadIdx.x, lane = t & 31, warp = t >> 5, tx = lane & 7, ty = lane >> 3;
  float* mine = smem + L::warps + warp * L::warp;
  float *X0 = mine + L::X0, *A1 = mine + L::A1, *AL = mine + L::AL, *A4 = mine + L::A4, *DS = mine + L::DS;
  float* coef = mine + L::coef;
  stage_weights<C, W, D1>(a, sw);
  __syncthreads();
  // WF, W / 4 thread columns (4 outputs each), each thread several inputs
  {
    constexpr int COLS = W / 4, ROWS = 32 * WARPS / COLS, RI = (W + ROWS - 1) / ROWS;
    const int c = t % COLS, r = t / COLS;
    float4 f[RI];
#pragma unroll
    for (int i = 0; i < RI; ++i) f[i] = make_float4(0.f, 0.f, 0.f, 0.f);
    for (int h = 0; h < W; ++h) {
      const float4 w = *reinterpret_cast<const float4*>(sw + P::w2 + h * LDW + 4 * c);
#pragma unroll
      for (int i = 0; i < RI; ++i)
        if (r + i * ROWS < W) fma4(f[i], sw[P::wh + (r + i * ROWS) * LDW + wpos(h)], w);
    }
#pragma unroll
    for (int i = 0; i < RI; ++i)
      if (r + i * ROWS < W) *reinterpret_cast<float4*>(wf + (r + i * ROWS) * LDW + 4 * c) = f[i];
  }
  __syncthreads();

  const int i0 = (DIST && C == 64) ? 32 * (warp & 1) : 0, j0 = DIST ? (C == 64 ? 16 * (warp >> 1) : 8 * warp) : 0;
  const int iF = DIST ? 32 * (warp & 1) : 0, jF = DIST ? 16 * (warp >> 1) : 0;
  float G0[4][NJ0] = {}, G1[D1 == 2 ? 4 : 1][8] = {}, GF[4][NJF] = {};
  float GPE[RW][PE_DIM] = {}, GS[RW] = {}, G3[RW][3] = {}, B0[RW] = {}, B1[RW] = {}, B4[RW] = {}, B3 = 0.f;

  const long long S = segment_total(a.S, a.S_dev);
  const long long span = DIST ? SEGS * WARPS : SEGS;  // segments per step of this loop
  const long long tiles = (S + span - 1) / span;
  const long long step = DIST ? gridDim.x : (long long)gridDim.x * WARPS;
  for (long long tile = blockIdx.x + (DIST ? 0 : (long long)gridDim.x * warp); tile < tiles; tile += step) {
    const long long s0 = tile * span + (DIST ? SEGS * warp : 0);
    put_coefs<SEGS>(a, S, s0, coef);
    __syncwarp();
    const int ray = s0 < S ? tile_ray<SEGS>(a, S, s0) : 0;
    if constexpr (SAVED) {
      static_assert(L::A1 == C * LD && L::DS == (C + (D1 + 1) * W) * LD && REC_SEGS % SEGS == 0, "the record's rows");
      load_record<C + (D1 + 1) * W, SEGS>(mine, a.acts, s0, S);
      // the next step's record on its way to L2 (DIVeR32: 247 -> 237 us)
      const long long sn = s0 + step * span;
      if (sn < S) {
        const float* rec = a.acts + sn / REC_SEGS * REC_FLOATS<C, W, D1>;
        for (int i = 32 * lane; i < REC_FLOATS<C, W, D1>; i += 32 * 32)
          asm volatile("prefetch.global.L2 [%0];" ::"l"(rec + i));
      }
    } else {
      gather_warp<C, SEGS>(a, S, s0, coef, X0);
      __syncwarp();
      // forward, keeping the activations
      float acc[W / 8][SPT];
      set_acc(acc, sw + P::b0);
      layer_fwd<C, W, SEGS>(X0, sw + P::l0, acc);
      put_acc<W / 8, SPT, true>(A1, acc);
      if constexpr (D1 == 2) {
        set_acc(acc, sw + P::b1);
        layer_fwd<W, W, SEGS>(A1, sw + P::l1, acc);
        put_acc<W / 8, SPT, true>(AL, acc);
      }
      set_acc(acc, sw + P::bh);
      layer_fwd<W, W, SEGS>(AL, sw + P::wh, acc);
      put_acc<W / 8, SPT, false>(A4, acc);
      set_acc(acc, nullptr);
      layer_fwd<W, W, SEGS>(A4, sw + P::w2, acc);
      add_ray_term<W>(a, ray, acc);
      put_acc<W / 8, SPT, true>(A4, acc);
    }
    // gradients of the logits and of sigma (zero past the last segment)
    if (lane < SEGS) {
      const long long s = s0 + lane;
      const float4 g = s < S ? a.d4[s] : make_float4(0.f, 0.f, 0.f, 0.f);
      const float3 c = colour<W, LD>(sw + P::w3, sw + P::b3, A4, lane);
      DS[lane] = g.y * c.x * (1.f - c.x);
      DS[LD + lane] = g.z * c.y * (1.f - c.y);
      DS[2 * LD + lane] = g.w * c.z * (1.f - c.z);
      DS[3 * LD + lane] = g.x;
    }
    __syncwarp();
    B3 += row_sum<SEGS>(DS + (lane & 3) * LD, 0xffffffffu);
#pragma unroll
    for (int r = 0; r < RW; ++r) {
#pragma unroll
      for (int c = 0; c < 3; ++c) G3[r][c] += row_dot<SEGS>(A4 + (lane + 32 * r) * LD, DS + c * LD);
      GS[r] += row_dot<SEGS>(AL + (lane + 32 * r) * LD, DS + 3 * LD);
    }
    // delta of mlp2's first layer, over its activation
    {
      float d[3][SPT], acc[W / 8][SPT];
#pragma unroll
      for (int c = 0; c < 3; ++c) load_segs<SPT>(DS + c * LD + SPT * ty, d[c]);
#pragma unroll
      for (int m = 0; m < W / 8; ++m) {
        const float4 w = *reinterpret_cast<const float4*>(sw + P::w3 + 4 * (tx + 8 * m));
#pragma unroll
        for (int s = 0; s < SPT; ++s) acc[m][s] = fmaf(w.z, d[2][s], fmaf(w.y, d[1][s], w.x * d[0][s]));
      }
      put_masked(A4, acc);
    }
    // its bias and PE rows: delta summed per ray
    for (unsigned left = SEGS == 32 ? 0xffffffffu : (1u << SEGS) - 1u; left != 0u;) {
      const int r = __shfl_sync(0xffffffffu, ray, __ffs(left) - 1);
      const unsigned m = __ballot_sync(0xffffffffu, ray == r) & left;
      left &= ~m;
      float v[RW];
#pragma unroll
      for (int u = 0; u < RW; ++u) {
        v[u] = row_sum<SEGS>(A4 + (lane + 32 * u) * LD, m);
        B4[u] += v[u];
      }
      const float* pe = a.pe_feat + (long long)r * PE_PAD;
#pragma unroll
      for (int k = 0; k < PE_DIM; ++k) {
        const float p = __ldg(pe + k);
#pragma unroll
        for (int u = 0; u < RW; ++u) GPE[u][k] = fmaf(p, v[u], GPE[u][k]);
      }
    }
    // folded layer
    if constexpr (DIST) {
      __syncthreads();
#pragma unroll 1
      for (int w = 0; w < WARPS; ++w) {
        const float* o = smem + L::warps + w * L::warp;
        weight_grad<4, NJF, SEGS>(o + L::AL + iF * LD, o + L::A4 + jF * LD, GF);
      }
      __syncthreads();
    } else {
      weight_grad<4, NJF, SEGS>(AL, A4, GF);
    }
    {
      float d[SPT], acc[W / 8][SPT];
      load_segs<SPT>(DS + 3 * LD + SPT * ty, d);
#pragma unroll
      for (int m = 0; m < W / 8; ++m) {
        const float w = sw[P::sig + tx + 8 * m];
#pragma unroll
        for (int s = 0; s < SPT; ++s) acc[m][s] = w * d[s];
      }
      layer_bwd<W, W, SEGS>(A4, wf, acc);
      put_masked(AL, acc);
    }
    // mlp1's second hidden layer
    if constexpr (D1 == 2) {
      B1[0] += row_sum<SEGS>(AL + lane * LD, 0xffffffffu);
      weight_grad<4, 8, SEGS>(A1, AL, G1);
      float acc[W / 8][SPT] = {};
      layer_bwd<W, W, SEGS>(AL, sw + P::l1, acc);
      put_masked(A1, acc);
    }
    // first layer
#pragma unroll
    for (int u = 0; u < RW; ++u) B0[u] += row_sum<SEGS>(A1 + (lane + 32 * u) * LD, 0xffffffffu);
    if constexpr (DIST) {
      __syncthreads();
#pragma unroll 1
      for (int w = 0; w < WARPS; ++w) {
        const float* o = smem + L::warps + w * L::warp;
        weight_grad<4, NJ0, SEGS>(o + L::X0 + i0 * LD, o + L::A1 + j0 * LD, G0);
      }
      __syncthreads();
    } else {
      weight_grad<4, NJ0, SEGS>(X0, A1, G0);
    }
    {
      float acc[C / 8][SPT] = {};
      layer_bwd<C, W, SEGS>(A1, sw + P::l0, acc);
      put_acc<C / 8, SPT, false>(X0, acc);
    }
    scatter_warp<C, SEGS>(a, S, s0, coef, X0);
    __syncwarp();  // the next gather overwrites the tile and its coefficients
  }

  // flush: the CTA's gradients into shared memory, warp by warp
  __syncthreads();
  float* fl = smem + L::warps;
  for (int i = t; i < L::flush; i += 32 * WARPS) fl[i] = 0.f;
  __syncthreads();
#pragma unroll 1
  for (int w = 0; w < WARPS; ++w) {
    if (warp == w) {
#pragma unroll
      for (int m = 0; m < 4; ++m) {
#pragma unroll
        for (int n = 0; n < NJ0; ++n) fl[L::g0 + (i0 + tx + 8 * m) * W + j0 + ty + 4 * n] += G0[m][n];
#pragma unroll
        for (int n = 0; n < NJF; ++n) fl[L::gf + (iF + tx + 8 * m) * LDW + wpos(jF + ty + 4 * n)] += GF[m][n];
        if constexpr (D1 == 2) {
#pragma unroll
          for (int n = 0; n < 8; ++n) fl[L::g1 + (tx + 8 * m) * W + ty + 4 * n] += G1[m][n];
        }
      }
#pragma unroll
      for (int u = 0; u < RW; ++u) {
        const int j = lane + 32 * u;
#pragma unroll
        for (int k = 0; k < PE_DIM; ++k) fl[L::gpe + k * W + j] += GPE[u][k];
        fl[L::gs + j] += GS[u];
#pragma unroll
        for (int c = 0; c < 3; ++c) fl[L::g3 + 4 * j + c] += G3[u][c];
        fl[L::gb0 + j] += B0[u];
        if (D1 == 2) fl[L::gb1 + j] += B1[u];
        fl[L::gb4 + j] += B4[u];
      }
      if (lane < 4) fl[L::gb3 + lane] += B3;
    }
    __syncthreads();
  }
  float* gp = a.grad_params;
  constexpr int NT = 32 * WARPS;
  for (int i = t; i < C * W; i += NT) atomicAdd(gp + a.w_off[0] + i, fl[L::g0 + i]);
  if (D1 == 2)
    for (int i = t; i < W * W; i += NT) atomicAdd(gp + a.w_off[1] + i, fl[L::g1 + i]);
  for (int i = t; i < PE_DIM * W; i += NT) atomicAdd(gp + a.w_off[D1 + 1] + W * W + i, fl[L::gpe + i]);
  for (int i = t; i < W; i += NT) {
    atomicAdd(gp + a.w_off[D1] + i * (W + 4), fl[L::gs + i]);
    atomicAdd(gp + a.b_off[0] + i, fl[L::gb0 + i]);
    if (D1 == 2) atomicAdd(gp + a.b_off[1] + i, fl[L::gb1 + i]);
    atomicAdd(gp + a.b_off[D1 + 1] + i, fl[L::gb4 + i]);
    float bh = 0.f;  // dL/dbh = W2 (sum delta)
    for (int j = 0; j < W; ++j) bh = fmaf(sw[P::w2 + i * LDW + wpos(j)], fl[L::gb4 + j], bh);
    atomicAdd(gp + a.b_off[D1] + 1 + i, bh);
  }
  for (int i = t; i < 4 * W; i += NT)
    if ((i & 3) < 3) atomicAdd(gp + a.w_off[D1 + 2] + i, fl[L::g3 + i]);
  if (t < 3) atomicAdd(gp + a.b_off[D1 + 2] + t, fl[L::gb3 + t]);
  if (t == 3) atomicAdd(gp + a.b_off[D1], fl[L::gb3 + 3]);
  // dL/dWH[i][h] = sum_j GF[i][j] W2[h][j]: a thread takes 4 x 4 entries, rows
  // and columns W / 4 apart
  constexpr int Q = W / 4;
  for (int e = t; e < Q * Q; e += NT) {
    const int i = e / Q, h = e % Q;
    float v[4][4] = {};
    for (int j = 0; j < W; j += 4) {
      float4 x[4];
#pragma unroll
      for (int m = 0; m < 4; ++m) x[m] = *reinterpret_cast<const float4*>(fl + L::gf + (i + Q * m) * LDW + j);
#pragma unroll
      for (int n = 0; n < 4; ++n) {
        const float4 y = *reinterpret_cast<const float4*>(sw + P::w2 + (h + Q * n) * LDW + j);
#pragma unroll
        for (int m = 0; m < 4; ++m) v[m][n] = fmaf(x[m].x, y.x, fmaf(x[m].y, y.y, fmaf(x[m].z, y.z, fmaf(x[m].w, y.w, v[m][n]))));
      }
    }
#pragma unroll
    for (int m = 0; m < 4; ++m)
#pragma unroll
      for (int n = 0; n < 4; ++n) atomicAdd(gp + a.w_off[D1] + (i + Q * m) * (W + 4) + 1 + h + Q * n, v[m][n]);
  }
  // dL/dW2[h][j] = sum_i WH[i][h] GF[i][j] + bh[h] (sum delta)[j], 4 consecutive positions of each
  for (int e = t; e < Q * Q; e += NT) {
    const int hp = 4 * (e / Q), jp = 4 * (e % Q);
    float v[4][4];
    // position p holds entry (p & ~31) + (p & 31) / 4 + 8 (p % 4)
    const int h = (hp & ~31) + ((hp & 31) >> 2), j = (jp & ~31) + ((jp & 31) >> 2);
#pragma unroll
    for (int m = 0; m < 4; ++m)
#pragma unroll
      for (int n = 0; n < 4; ++n) v[m][n] = sw[P::bh + h + 8 * m] * fl[L::gb4 + j + 8 * n];
    for (int i = 0; i < W; ++i) {
      const float4 x = *reinterpret_cast<const float4*>(sw + P::wh + i * LDW + hp);
      const float4 y = *reinterpret_cast<const float4*>(fl + L::gf + i * LDW + jp);
      const float xs[4] = {x.x, x.y, x.z, x.w}, ys[4] = {y.x, y.y, y.z, y.w};
#pragma unroll
      for (int m = 0; m < 4; ++m)
#pragma unroll
        for (int n = 0; n < 4; ++n) v[m][n] = fmaf(xs[m], ys[n], v[m][n]);
    }
#pragma unroll
    for (int m = 0; m < 4; ++m)
#pragma unroll
      for (int n = 0; n < 4; ++n) atomicAdd(gp + a.w_off[D1 + 1] + (h + 8 * m) * W + j + 8 * n, v[m][n]);
  }
}

// Blocks of a launch: every SM gets work before any gets a second tile per warp slot.
template <int C, int W, int D1, int SEGS, int WARPS, int CTAS>
int launch_decode_fwd(const DecodeArgs& a, cudaStream_t st, int sms) {
  const size_t smem =
      (size_t)(PlainWeights<C, W, D1>::size + WARPS * FwdSmem<C, W, D1, SEGS>::warp) * sizeof(float);
  auto k = a.acts ? decode_fwd_plain<C, W, D1, SEGS, WARPS, CTAS, true> : decode_fwd_plain<C, W, D1, SEGS, WARPS, CTAS, false>;
  if (cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) != cudaSuccess) return DV_ERR_CUDA;
  const long long tiles = (a.S + SEGS - 1) / SEGS;
  const long long grid = std::min<long long>({tiles, (long long)sms * CTAS, std::max<long long>(sms, (tiles + WARPS - 1) / WARPS)});
  k<<<(unsigned)grid, 32 * WARPS, smem, st>>>(a);
  DV_TRY_LAUNCH();
  return DV_OK;
}

template <int C, int W, int D1, int SEGS, bool DIST>
int launch_decode_bwd(const DecodeArgs& a, cudaStream_t st, int sms) {
  constexpr int WARPS = 8;
  const size_t smem = (size_t)BwdSmem<C, W, D1, SEGS, WARPS>::size * sizeof(float);
  auto k = a.acts ? decode_bwd_plain<C, W, D1, SEGS, WARPS, DIST, true> : decode_bwd_plain<C, W, D1, SEGS, WARPS, DIST, false>;
  if (cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) != cudaSuccess) return DV_ERR_CUDA;
  const long long tiles = (a.S + SEGS - 1) / SEGS;
  const long long grid = std::min<long long>(DIST ? (tiles + WARPS - 1) / WARPS : tiles, sms);
  k<<<(unsigned)grid, 32 * WARPS, smem, st>>>(a);
  DV_TRY_LAUNCH();
  return DV_OK;
}

// Per-variant entry points, one translation unit each.
int decode_fwd_v32c32(const DecodeArgs& a, cudaStream_t st, int sms);
int decode_bwd_v32c32(const DecodeArgs& a, cudaStream_t st, int sms);
int decode_fwd_v64c32(const DecodeArgs& a, cudaStream_t st, int sms);
int decode_bwd_v64c32(const DecodeArgs& a, cudaStream_t st, int sms);
int decode_fwd_v64c64(const DecodeArgs& a, cudaStream_t st, int sms);
int decode_bwd_v64c64(const DecodeArgs& a, cudaStream_t st, int sms);

}  // namespace dv
