// Tensor-core (tcgen05) decoder forward for the training / offline path.
//
// One CTA = 128 threads = one tile of 128 segments = the 128 TMEM lanes of
// an M=128 MMA.  Per tile:
//   gather  C/4 threads per segment read the 8 corner rows (coalesced float4),
//           integrate in FP32 and write the feature row as BF16/FP16 straight
//           into the K-major A operand tile in shared memory
//   layers  each Linear layer is one chain of K/16 tcgen05.mma (A and B from
//           shared memory, FP32 accumulators in TMEM), committed to an
//           mbarrier; thread t then reads its row (TMEM lane t), adds the bias,
//           applies ReLU and writes the next A tile row
//   output  sigma (FP32) and sigmoid(rgb) per segment
// Issue slots and the L1's wavefronts bound it more than the tensor core does
// (ncu on the form before: 67 % of issue slots, 69 % of LSU wavefronts, 5 %
// tensor), so a segment's corners are computed once, additions and the
// integral's FMAs go in packed pairs, biases come in 16-byte loads and ReLU is
// taken on rounded pairs.  Measured against one thread per 8 channels doing
// all of it: 800x800 frame of the 256^3 scene, BF16 10.5 -> 8.8 ms; DIVeR64 over
// 64 channels, 399x401, FP16 5.2 -> 3.8 ms; split, 65,792 rays of the wide grid
// 647 -> 509 us.  Then, single-term forms without a save record: activations
// in TMEM and a swizzled feature tile (LSU wavefronts 2244 -> 1670 per tile) and
// tiles taken dynamically: frame 8.8 -> 6.2 ms, DIVeR64 view 3.8 -> 3.1 ms.
// What is left of a frame's tile (8 CTAs per SM): half of its time gathers at
// four fifths of the LSU pipe, a fifth waits for the five MMA chains.
// The decoder's weights (all layers, B operands in the same K-major layout)
// and biases stay in shared memory for the CTA's lifetime; the grid is
// persistent over tiles and sized so TMEM never oversubscribes.
// Reference semantics: model/diver.py:159-180 (mlp1, PE, mlp2, sigmoid).
#include "common.cuh"
#include "integrate.cuh"
#include "mlp.cuh"
#include "tc.cuh"

#include <cuda_bf16.h>
#include <cuda_fp16.h>

#include <algorithm>

namespace dv {

constexpr int TC_MAX_LAYERS = 5;

struct TcLayer {
  int b_off;     // byte offset of the layer's B image in the weight blob
  int K, N;      // padded: K % 16 == 0, N % 16 == 0
  int bias_off;  // float offset of the layer's bias (N entries)
  int s_bias;    // its offset in shared memory (a multiple of 16)
  int s_off;     // split form: byte offset of the layer's [3 x N][K] image (terms side by side) in shared memory
};

struct TcArgs {
  const float* grid;
  const uint16_t* grid16;  // optional BF16/FP16 copy of the grid (same layout); used when non-null
  int nvx, nvy, nvz;
  const float* seg;
  const int* seg_ray;
  long long S;           // segment count, or capacity when S_dev is set
  const int64_t* S_dev;  // optional device-held count (clamped to S)
  const float* pe_out;  // [B][W]: bias + PE part of mlp2's first layer (FP32)
  float4* out4;
  const uint8_t* wblob;
  int wbytes;  // bytes of one term's weight images (multiple of 16); TERMS terms follow each other
  const float* bias;
  int nbias;   // biases in shared memory
  TcLayer L[TC_MAX_LAYERS];
  int* err;    // set to 1 if an MMA completion wait timed out
  int steal;   // one CTA was launched per tile, and running ones take over those not yet started
  uint8_t* save;       // optional: every layer's input tile, per 128-segment tile (training)
  int save_off[TC_MAX_LAYERS];  // byte offset of layer l's input tile inside a tile's record; negative: not saved
  int save_bytes;      // bytes per tile record (sum of 256 * K over the layers)
};

// Address of term i of element (r, c) of an A tile with K columns.  One term:
// a [128][K] K-major tile at sA.  Three terms: terms 0 and 1 side by side in
// one [128][2K] tile at sA (columns i * K + c; the two-term copy of the layer
// input that the training backward reads back, saved with one bulk copy),
// term 2 in a [128][K] tile of its own at sA + 2 * tstride.
template <int TERMS>
__device__ __forceinline__ uint8_t* a_term(uint8_t* sA, uint32_t tstride, int r, int c, int K, int i) {
  if constexpr (TERMS == 1) return sA + tc::kmajor_offset(r, c, K);
  return i < 2 ? sA + tc::kmajor_offset(r, i * K + c, 2 * K) : sA + 2 * tstride + tc::kmajor_offset(r, c, K);
}

// Corner weights and rows of this thread's segment, s0 + threadIdx.x: the
// weights, the lower corner's row and the row steps to the upper corners
// (0 where clamped).  Computed once per segment and handed to the C/4 or C/8
// threads that gather its channels, all in the same warp (computed by each of
// them, this was a third of the kernel's instructions).  Rows fit 32 bits: 2^32
// rows of 32 channels are twice the device's memory.
struct Corners {
  float w[8];
  uint32_t row, dx, dy, dz;
};

// This thread's segment record.
struct Seg6 {
  float p[6];
};

__device__ __forceinline__ Seg6 load_seg(const TcArgs& a, long long S, long long s) {
  Seg6 r{};
  if (s < S) {
#pragma unroll
    for (int i = 0; i < 6; ++i) r.p[i] = __ldg(a.seg + s * 6 + i);
  }
  return r;
}

__device__ __forceinline__ Corners corners_of(const TcArgs& a, bool valid, const Seg6& g) {
  Corners c{};
  if (valid) {
    const SegCorner sc = segment_corners(g.p[0], g.p[1], g.p[2], g.p[3], g.p[4], g.p[5], a.nvx, a.nvy, a.nvz);
#pragma unroll
    for (int j = 0; j < 8; ++j) c.w[j] = sc.w[j];
    c.row = ((uint32_t)sc.z * a.nvy + sc.y) * a.nvx + sc.x;
    c.dx = sc.x1 - sc.x;
    c.dy = (uint32_t)(sc.y1 - sc.y) * a.nvx;
    c.dz = (uint32_t)(sc.z1 - sc.z) * a.nvx * a.nvy;
  }
  return c;
}

// The 8 corner rows (BYTES each) at byte q of a row.
template <int BYTES>
__device__ __forceinline__ void load_corners(const uint8_t* grid, uint32_t row, uint32_t dx, uint32_t dy, uint32_t dz,
                                             uint4* v) {
  const uint8_t* p = grid + (unsigned long long)row * BYTES;
  const uint32_t x = dx * BYTES;
  const uint8_t* py = p + (unsigned long long)dy * BYTES;
  const uint8_t* pz = p + (unsigned long long)dz * BYTES;
  const uint8_t* pw = py + (unsigned long long)dz * BYTES;
  const uint8_t* r[4] = {p, py, pz, pw};
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    v[2 * j] = __ldg(reinterpret_cast<const uint4*>(r[j]));
    v[2 * j + 1] = __ldg(reinterpret_cast<const uint4*>(r[j] + x));
  }
}

// A 16-bit pair as two FP32 values.
template <int BF16>
__device__ __forceinline__ unsigned long long unpack2(uint32_t x) {
  if (BF16) return f32x2(__uint_as_float(x << 16), __uint_as_float(x & 0xffff0000u));
  const float2 f = __half22float2(*reinterpret_cast<const __half2*>(&x));
  return f32x2(f.x, f.y);
}

constexpr int COEF = 12;  // floats of a segment's Corners in shared memory

__device__ __forceinline__ void put_corners(float* coef, const Corners& c) {
  float4* d = reinterpret_cast<float4*>(coef + threadIdx.x * COEF);
  d[0] = make_float4(c.w[0], c.w[1], c.w[2], c.w[3]);
  d[1] = make_float4(c.w[4], c.w[5], c.w[6], c.w[7]);
  reinterpret_cast<uint4*>(d)[2] = make_uint4(c.row, c.dx, c.dy, c.dz);
  __syncwarp();
}

// Single-term gather: TPS threads per segment, each integrating 16 bytes of
// every corner row (4 channels of the FP32 grid, or 8 of its 16-bit copy) in
// FP32, and writing the feature row's 16-bit operand.  U passes' loads are in
// flight per thread.
template <int C, int BF16, bool G16, bool SWZ, int U>
__device__ __forceinline__ void gather_tile(const TcArgs& a, long long S, long long s0, const Seg6& g, uint8_t* sA, float* coef) {
  constexpr int CH = G16 ? 8 : 4, TPS = C / CH, SPP = 32 / TPS, BYTES = C * (G16 ? 2 : 4);
  const int lane = threadIdx.x & 31, q = lane % TPS, first = (threadIdx.x & ~31) + lane / TPS;
  const Corners own = corners_of(a, s0 + threadIdx.x < S, g);
  put_corners(coef, own);
  // training (a save record): the rows of the later passes on their way while the first waits; a
  // training batch's come from DRAM (captured 4096-ray BF16 step of a 256^3 scene, 1038 -> 1012 us)
  if (!G16 && !SWZ && a.save != nullptr && s0 + threadIdx.x < S)
    prefetch_rows<C * 4>(a.grid, own.row, own.dx, own.dy, own.dz);
  const uint8_t* grid = (G16 ? reinterpret_cast<const uint8_t*>(a.grid16) : reinterpret_cast<const uint8_t*>(a.grid)) + 16 * q;
#pragma unroll 1
  for (int p = 0; p < TPS; p += U) {
    uint4 v[U][8];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const uint4 m = *reinterpret_cast<const uint4*>(coef + (first + (p + u) * SPP) * COEF + 8);
      load_corners<BYTES>(grid, m.x, m.y, m.z, m.w, v[u]);  // past the last segment: row 0, weights 0
    }
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int ls = first + (p + u) * SPP;
      const float4 wa = *reinterpret_cast<const float4*>(coef + ls * COEF);
      const float4 wb = *reinterpret_cast<const float4*>(coef + ls * COEF + 4);
      const float w[8] = {wa.x, wa.y, wa.z, wa.w, wb.x, wb.y, wb.z, wb.w};
      unsigned long long f[CH / 2];
#pragma unroll
      for (int k = 0; k < CH / 2; ++k) f[k] = 0ull;
      const bool in = s0 + ls < S;
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        const unsigned long long ww = f32x2(w[j], w[j]);
        const uint4 x = v[u][j];
        if (G16) {
          f[0] = fma_f32x2(ww, unpack2<BF16>(x.x), f[0]);
          f[1] = fma_f32x2(ww, unpack2<BF16>(x.y), f[1]);
          f[CH / 2 - 2] = fma_f32x2(ww, unpack2<BF16>(x.z), f[CH / 2 - 2]);
          f[CH / 2 - 1] = fma_f32x2(ww, unpack2<BF16>(x.w), f[CH / 2 - 1]);
        } else {
          f[0] = fma_f32x2(ww, f32x2(__uint_as_float(x.x), __uint_as_float(x.y)), f[0]);
          f[1] = fma_f32x2(ww, f32x2(__uint_as_float(x.z), __uint_as_float(x.w)), f[1]);
        }
      }
      uint32_t o[CH / 2];
#pragma unroll
      for (int k = 0; k < CH / 2; ++k) {
        const float2 r = f32x2_get(f[k]);
        o[k] = in ? tc::pack2<BF16>(r.x, r.y) : 0u;
      }
      uint8_t* dst = sA + (SWZ ? tc::swizzled_offset<C>(ls, CH * q) : tc::kmajor_offset(ls, CH * q, C));
      if (G16)
        *reinterpret_cast<uint4*>(dst) = make_uint4(o[0], o[1], o[CH / 2 - 2], o[CH / 2 - 1]);
      else
        *reinterpret_cast<uint2*>(dst) = make_uint2(o[0], o[1]);
    }
  }
}

// The split form's gather (FP32 grid, three operand terms): two passes at a
// time, so each thread has 16 corner-row loads in flight.  Its kernel runs 4
// CTAs per SM (its shared memory), so the registers this takes cost no
// residency, and the corners go from lane to lane by shuffles, as shared
// memory is what is short.
template <int C, int TERMS>
__device__ __forceinline__ void gather_tile_split(const TcArgs& a, long long S, long long s0, const Seg6& g,
                                                  uint8_t* sA, uint32_t tstride) {
  constexpr int TPS = C / 4, SPP = 32 / TPS;
  static_assert(TPS % 2 == 0, "passes are taken in pairs");
  const int lane = threadIdx.x & 31, warp0 = threadIdx.x & ~31, q = lane % TPS;
  const Corners c = corners_of(a, s0 + threadIdx.x < S, g);
  const uint8_t* grid = reinterpret_cast<const uint8_t*>(a.grid) + 16 * q;
  const uint32_t flags = (c.dx ? 1u : 0u) | (c.dy ? 2u : 0u) | (c.dz ? 4u : 0u);
#pragma unroll 1
  for (int p = 0; p < TPS; p += 2) {
    uint4 v[2][8];
#pragma unroll
    for (int u = 0; u < 2; ++u) {
      const int src = (p + u) * SPP + lane / TPS;
      const uint32_t row = __shfl_sync(0xffffffffu, c.row, src), m = __shfl_sync(0xffffffffu, flags, src);
      load_corners<C * 4>(grid, row, m & 1u, (m & 2u) ? a.nvx : 0, (m & 4u) ? (uint32_t)a.nvx * a.nvy : 0, v[u]);
    }
#pragma unroll
    for (int u = 0; u < 2; ++u) {
      const int src = (p + u) * SPP + lane / TPS, ls = warp0 + src;
      unsigned long long f[2] = {0ull, 0ull};
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        const float w = __shfl_sync(0xffffffffu, c.w[j], src);
        const uint4 x = v[u][j];
        f[0] = fma_f32x2(f32x2(w, w), f32x2(__uint_as_float(x.x), __uint_as_float(x.y)), f[0]);
        f[1] = fma_f32x2(f32x2(w, w), f32x2(__uint_as_float(x.z), __uint_as_float(x.w)), f[1]);
      }
      const bool in = s0 + ls < S;
      const float2 lo = f32x2_get(f[0]), hi = f32x2_get(f[1]);
      uint32_t x[TERMS], y[TERMS];
      tc::split_pair<TERMS>(in ? lo.x : 0.f, in ? lo.y : 0.f, x);
      tc::split_pair<TERMS>(in ? hi.x : 0.f, in ? hi.y : 0.f, y);
#pragma unroll
      for (int i = 0; i < TERMS; ++i)
        *reinterpret_cast<uint2*>(a_term<TERMS>(sA, tstride, ls, 4 * q, C, i)) = make_uint2(x[i], y[i]);
    }
  }
}

// Issues one layer's MMA chain (thread 0) and waits for it (all threads).
// With TERMS = 3 the A tile and the weight images are three BF16 terms each
// and the chain sums the six products whose term indices add up to at most 2
// (FP32-grade products) in four MMAs per 16 columns of K: A0 and A1 against
// the weight terms [W0|W1] side by side (N = 2N), A0 x W2 into columns
// N..2N-1 and A2 x W0 into columns 0..N-1; the layer's output is the sum of
// the two column blocks (acc_row / acc_row4).  A tcgen05.mma costs about the
// same at N = 2N as at N, so this is two MMAs fewer per K step.  With `save`, thread 0 also copies the layer's input
// tile (the A operand, 256 * K bytes; with TERMS = 3 the [128][2K] tile of its
// first two terms, a two-term split of the same values) to global memory by a
// bulk async copy and, before the caller's barrier lets anyone overwrite A,
// waits until that copy has read it.
template <int BF16, int TERMS>
__device__ __forceinline__ bool tc_layer(const TcLayer& L, const uint8_t* sB, const uint8_t* sA, uint32_t tstride,
                                         uint32_t tmem, uint64_t* bar, uint32_t& phase,
                                         uint8_t* save = nullptr) {
  if (threadIdx.x == 0) {
    tc::fence_after_sync();
    if (save != nullptr) {
      tc::bulk_store(save, sA, (uint32_t)L.K * 256u * (TERMS > 1 ? 2u : 1u));
      tc::bulk_commit();
    }
    const uint32_t sbo = (uint32_t)(L.K / 8) * 128;
    if constexpr (TERMS == 1) {
      const uint32_t idesc = tc::idesc_f16(128, L.N, BF16);
      const uint32_t a0 = tc::smem_u32(sA), b0 = tc::smem_u32(sB + L.b_off);
      for (int k = 0; k < L.K / 16; ++k)
        tc::mma_f16(tmem, tc::smem_desc(a0 + k * 256, 128, sbo), tc::smem_desc(b0 + k * 256, 128, sbo), idesc,
                    k > 0 ? 1u : 0u);
    } else {
      // A terms (a_term's layout): 0 and 1 are K-column slices of the [128][2K] tile, 2 its own tile
      const uint64_t a0 = tc::smem_desc(tc::smem_u32(sA), 128, 2 * sbo);
      const uint64_t a1 = tc::desc_plus(a0, (uint32_t)(L.K / 8) * 128);
      const uint64_t a2 = tc::smem_desc(tc::smem_u32(sA + 2 * tstride), 128, sbo);
      // weights [W0|W1|W2] along N (rows): [W0|W1] is the first 2N rows, W0 the first N
      const uint64_t b01 = tc::smem_desc(tc::smem_u32(sB + L.s_off), 128, sbo);
      const uint64_t b2 = tc::desc_plus(b01, (uint32_t)(2 * L.N * L.K * 2));
      const uint32_t i2 = tc::idesc_f16(128, 2 * L.N, 1), i1 = tc::idesc_f16(128, L.N, 1);
      for (int k = 0; k < L.K / 16; ++k) {
        const uint32_t o = (uint32_t)k * 256;
        tc::mma_f16(tmem, tc::desc_plus(a0, o), tc::desc_plus(b01, o), i2, k > 0 ? 1u : 0u);
        tc::mma_f16(tmem, tc::desc_plus(a1, o), tc::desc_plus(b01, o), i2, 1u);
        tc::mma_f16(tmem + L.N, tc::desc_plus(a0, o), tc::desc_plus(b2, o), i1, 1u);
        tc::mma_f16(tmem, tc::desc_plus(a2, o), tc::desc_plus(b01, o), i1, 1u);
      }
    }
    tc::mma_commit(bar);
  }
  const bool done = tc::mbar_wait_bounded(bar, phase);
  phase ^= 1u;
  tc::fence_after_sync();
  if (save != nullptr && threadIdx.x == 0) tc::bulk_wait_read();
  return done;
}

// A layer of the single-term form without a save record: A is the swizzled
// feature tile in shared memory (FIRST) or the activations in TMEM columns
// from `acol`, B as above.
template <int K, bool FIRST>
__device__ __forceinline__ bool tc_layer_ts(const TcLayer& L, const uint8_t* sB, const uint8_t* sA, uint32_t tmem,
                                            uint32_t acol, int bf16, uint64_t* bar, uint32_t& phase) {
  if (threadIdx.x == 0) {
    tc::fence_after_sync();
    const uint32_t idesc = tc::idesc_f16(128, L.N, bf16);
    const uint64_t b0 = tc::smem_desc(tc::smem_u32(sB + L.b_off), 128, (K / 8) * 128);
    const uint64_t a0 = tc::swizzled_desc<K>(tc::smem_u32(sA));
#pragma unroll
    for (int k = 0; k < K / 16; ++k) {
      if (FIRST)
        tc::mma_f16(tmem, tc::desc_plus(a0, k * 32), tc::desc_plus(b0, k * 256), idesc, k > 0 ? 1u : 0u);
      else
        tc::mma_f16_ts(tmem, tmem + acol + 8 * k, tc::desc_plus(b0, k * 256), idesc, k > 0 ? 1u : 0u);
    }
    tc::mma_commit(bar);
  }
  const bool done = tc::mbar_wait_bounded(bar, phase);
  phase ^= 1u;
  tc::fence_after_sync();
  return done;
}

// Epilogue columns per pass: 32, or 16 for the split form, whose rows are the
// sum of two TMEM column blocks (registers: its kernel runs 4 CTAs per SM).
template <int TERMS>
constexpr int EPI_COLS = TERMS == 1 ? 32 : 16;

// This thread's row of a layer's output, EPI_COLS columns from taddr; with
// TERMS = 3 the sum of tc_layer's two column blocks (the second n columns on).
template <int TERMS>
__device__ __forceinline__ void acc_row(uint32_t taddr, int n, float* v) {
  if constexpr (TERMS == 1) {
    tc::ld_32x32b_x32(taddr, v);
    tc::ld_wait();
  } else {
    float u[16];
    tc::ld_32x32b_x16(taddr, v);
    tc::ld_32x32b_x16(taddr + n, u);
    tc::ld_wait();
#pragma unroll
    for (int i = 0; i < 16; ++i) v[i] += u[i];
  }
}

// Same for 4 columns.
template <int TERMS>
__device__ __forceinline__ void acc_row4(uint32_t taddr, int n, float* v) {
  tc::ld_32x32b_x4(taddr, v);
  if constexpr (TERMS > 1) {
    float u[4];
    tc::ld_32x32b_x4(taddr + n, u);
    tc::ld_wait();
#pragma unroll
    for (int i = 0; i < 4; ++i) v[i] += u[i];
  } else {
    tc::ld_wait();
  }
}

// Adds n (a multiple of 4) values at p (16-byte aligned) to v.
template <int n>
__device__ __forceinline__ void add_row(float* v, const float* p) {
#pragma unroll
  for (int i = 0; i < n; i += 4) {
    const float4 b = *reinterpret_cast<const float4*>(p + i);
    const float2 x = f32x2_get(add_f32x2(f32x2(v[i], v[i + 1]), f32x2(b.x, b.y)));
    const float2 y = f32x2_get(add_f32x2(f32x2(v[i + 2], v[i + 3]), f32x2(b.z, b.w)));
    v[i] = x.x;
    v[i + 1] = x.y;
    v[i + 2] = y.x;
    v[i + 3] = y.y;
  }
}

// 16-bit pair of max(a, 0), max(b, 0) (NaN gives 0, like fmaxf): rounding is
// monotone, so the maximum is taken on the rounded pair, one instruction.
template <int BF16>
__device__ __forceinline__ uint32_t pack2_relu(float a, float b) {
  uint32_t r = tc::pack2<BF16>(a, b);
  if (BF16)
    asm("max.bf16x2 %0, %0, %1;" : "+r"(r) : "r"(0u));
  else
    asm("max.f16x2 %0, %0, %1;" : "+r"(r) : "r"(0u));
  return r;
}

// Writes EPI_COLS values (columns c0.. of the next layer's input) of row t,
// through ReLU if RELU, as TERMS operand terms (a_term's layout).
template <int BF16, int TERMS, bool RELU>
__device__ __forceinline__ void store_row(uint8_t* sA, uint32_t tstride, int t, int c0, int K, float* v) {
#pragma unroll
  for (int j = 0; j < EPI_COLS<TERMS> / 8; ++j) {
    if constexpr (TERMS == 1) {
      uint32_t w[4];
#pragma unroll
      for (int i = 0; i < 4; ++i)
        w[i] = RELU ? pack2_relu<BF16>(v[8 * j + 2 * i], v[8 * j + 2 * i + 1])
                    : tc::pack2<BF16>(v[8 * j + 2 * i], v[8 * j + 2 * i + 1]);
      *reinterpret_cast<uint4*>(a_term<1>(sA, tstride, t, c0 + 8 * j, K, 0)) = make_uint4(w[0], w[1], w[2], w[3]);
    } else {
      uint32_t x[TERMS], y[TERMS], z[TERMS], u[TERMS];
      if (RELU) {
#pragma unroll
        for (int i = 0; i < 8; ++i) v[8 * j + i] = fmaxf(v[8 * j + i], 0.f);
      }
      tc::split_pair<TERMS>(v[8 * j + 0], v[8 * j + 1], x);
      tc::split_pair<TERMS>(v[8 * j + 2], v[8 * j + 3], y);
      tc::split_pair<TERMS>(v[8 * j + 4], v[8 * j + 5], z);
      tc::split_pair<TERMS>(v[8 * j + 6], v[8 * j + 7], u);
#pragma unroll
      for (int i = 0; i < TERMS; ++i)
        *reinterpret_cast<uint4*>(a_term<TERMS>(sA, tstride, t, c0 + 8 * j, K, i)) = make_uint4(x[i], y[i], z[i], u[i]);
    }
  }
}

// The same 32 values of row t into TMEM columns (two per column).
template <int BF16, bool RELU>
__device__ __forceinline__ void put_row_ts(uint32_t taddr, const float* v) {
  uint32_t w[16];
#pragma unroll
  for (int i = 0; i < 16; ++i)
    w[i] = RELU ? pack2_relu<BF16>(v[2 * i], v[2 * i + 1]) : tc::pack2<BF16>(v[2 * i], v[2 * i + 1]);
  tc::st_32x32b_x16(taddr, w);
}

__device__ __forceinline__ void sync_for_mma_ts() {
  tc::st_wait();
  tc::fence_before_sync();
  __syncthreads();
}

__device__ __forceinline__ void sync_for_mma() {
  tc::fence_before_sync();
  tc::fence_async_smem();
  __syncthreads();
}

// NCOLS: TMEM columns (>= widest N, power of two >= 32).  TERMS: operand
// terms (1: BF16 or FP16 operands; 3: FP32 values as three BF16 terms, six
// products per layer, FP32-grade; BF16 only and read from the FP32 grid).
// Registers per thread are capped to the residency the other resources allow:
// 8 CTAs per SM for the single-term forms (TMEM), 4 for the DIVeR32 split
// form (shared memory; its two-pass gather would otherwise take 3).
template <int C, int W, int D1, int BF16, int NCOLS, int TERMS, bool TS>
__global__ void __launch_bounds__(128, TERMS == 1 ? (W == 32 ? 8 : 4) : ((C == 32 && W == 32) ? 4 : 1)) decode_fwd_tc(const TcArgs a) {
  constexpr int KMAX = C > W ? C : W;
  constexpr uint32_t TSTRIDE = 128 * KMAX * 2;  // bytes between the A tile's terms
  extern __shared__ __align__(1024) uint8_t smem[];
  uint8_t* sA = smem;  // on a 1024-byte boundary (its swizzle)
  uint8_t* sB = smem + TERMS * TSTRIDE;
  float* sBias = reinterpret_cast<float*>(sB + TERMS * a.wbytes);
  float* coef = sBias + a.nbias;
  uint8_t* answer = reinterpret_cast<uint8_t*>(coef + (TERMS == 1 ? 128 * COEF : 0));  // 16 bytes
  uint64_t* bar = reinterpret_cast<uint64_t*>(answer + 16);
  uint64_t* bar_next = bar + 1;
  uint32_t* tslot = reinterpret_cast<uint32_t*>(bar + 2);
  const int t = threadIdx.x, warp = t >> 5;
  if constexpr (TERMS == 1) {
    for (int i = t; i < a.wbytes / 16; i += 128)
      reinterpret_cast<uint4*>(sB)[i] = __ldg(reinterpret_cast<const uint4*>(a.wblob) + i);
  } else {
    // the images regrouped layer by layer, the three terms side by side along N
#pragma unroll 1
    for (int l = 0; l < D1 + 3; ++l) {
      const TcLayer& L = a.L[l];
      const int img16 = L.N * L.K * 2 / 16;
      for (int i = t; i < 3 * img16; i += 128) {
        const int j = i / img16, o = i % img16;
        reinterpret_cast<uint4*>(sB + L.s_off)[i] =
            __ldg(reinterpret_cast<const uint4*>(a.wblob + (size_t)j * a.wbytes + L.b_off) + o);
      }
    }
  }
#pragma unroll 1
  for (int l = 0; l < D1 + 3; ++l)
    for (int i = t; i < a.L[l].N; i += 128) sBias[a.L[l].s_bias + i] = __ldg(a.bias + a.L[l].bias_off + i);
  if (t == 0) {
    tc::mbar_init(bar, 1);
    tc::mbar_init(bar_next, 1);
    tc::fence_mbar_init();
  }
  if (warp == 0) {
    tc::tmem_alloc(tslot, NCOLS);
    tc::tmem_relinquish();
  }
  sync_for_mma();
  tc::fence_after_sync();
  const uint32_t tmem = *tslot;
  const uint32_t trow = tmem + ((uint32_t)(warp * 32) << 16);  // this warp's TMEM lanes
  uint32_t phase = 0;
  bool ok = true;
  const bool saving = a.save != nullptr;
  const long long S = segment_total(a.S, a.S_dev);
  const long long tiles = (S + 127) / 128;
  // the next tile's segment is loaded while this one's last layer runs, where
  // registers allow it (the single-term DIVeR32 forms have none to spare)
  constexpr bool AHEAD = TERMS > 1 || W > 32;
  Seg6 seg{};
  if (AHEAD) seg = load_seg(a, S, (long long)blockIdx.x * 128 + t);
  uint32_t phase_next = 0;
  long long next = 0;
  for (long long tile = blockIdx.x; tile < tiles && ok; tile = next) {
    const long long s0 = tile * 128;
    const long long s = s0 + t;
    next = tile + gridDim.x;
    if (a.steal && t == 0) {
      tc::fence_async_smem();  // the last answer was read (the tile's end barrier) before this one is written
      tc::clc_request(answer, bar_next);
    }
    const bool valid = s < S;
    uint8_t* rec = saving ? a.save + tile * (long long)a.save_bytes : nullptr;
    constexpr int EC = EPI_COLS<TERMS>;
    constexpr uint32_t ACOL = NCOLS - W / 2;  // TS: the activations' columns, behind the widest layer's output
    float v[EC];
    // A layer's MMAs, then its wait; a wait that gave up is seen by all at the
    // tile's end.  While the layer's input is being copied out nobody may
    // overwrite it, which takes a barrier.
#define DV_LAYER(l, first)                                                                                       \
  do {                                                                                                           \
    if constexpr (TS) {                                                                                          \
      ok &= tc_layer_ts<first ? C : W, first>(a.L[l], sB, sA, tmem, ACOL, BF16, bar, phase);                     \
    } else {                                                                                                     \
      const bool copy = saving && a.save_off[l] >= 0;                                                            \
      ok &= tc_layer<BF16, TERMS>(a.L[l], sB, sA, TSTRIDE, tmem, bar, phase,                                     \
                                  copy ? rec + a.save_off[l] : nullptr);                                         \
      if (copy) __syncthreads();                                                                                 \
    }                                                                                                            \
  } while (0)
    // Its output plus `bias`, through ReLU if asked, as the next layer's input.
#define DV_EPILOGUE(l, bias, relu)                                     \
  do {                                                                 \
    _Pragma("unroll") for (int c0 = 0; c0 < W; c0 += EC) {             \
      acc_row<TERMS>(trow + c0, a.L[l].N, v);                          \
      add_row<EC>(v, (bias) + c0);                                     \
      if constexpr (TS)                                                \
        put_row_ts<BF16, relu>(trow + ACOL + c0 / 2, v);               \
      else                                                             \
        store_row<BF16, TERMS, relu>(sA, TSTRIDE, t, c0, W, v);        \
    }                                                                  \
    if constexpr (TS)                                                  \
      sync_for_mma_ts();                                               \
    else                                                               \
      sync_for_mma();                                                  \
  } while (0)
    if (!AHEAD) seg = load_seg(a, S, s);
    if constexpr (TERMS > 1) {
      gather_tile_split<C, TERMS>(a, S, s0, seg, sA, TSTRIDE);
    } else {
      constexpr int U = W == 32 ? 1 : 2;  // 8 CTAs per SM leave 64 registers a thread, 4 leave 128
      if (a.grid16)
        gather_tile<C, BF16, true, TS, U>(a, S, s0, seg, sA, coef);
      else
        gather_tile<C, BF16, false, TS, U>(a, S, s0, seg, sA, coef);
    }
    sync_for_mma();
    // mlp1 hidden layers: D = relu(A W^T + b)
    DV_LAYER(0, true);
    DV_EPILOGUE(0, sBias + a.L[0].s_bias, true);
    if constexpr (D1 == 2) {
      DV_LAYER(1, false);
      DV_EPILOGUE(1, sBias + a.L[1].s_bias, true);
    }
    // mlp1 output: columns 0..W-1 hidden (no activation), column W sigma
    const float* po = a.pe_out + (long long)(valid ? __ldg(a.seg_ray + s) : 0) * W;
    DV_LAYER(D1, false);
    float sigma;
    {
      float sv[4];
      acc_row4<TERMS>(trow + W, a.L[D1].N, sv);
      sigma = sv[0] + sBias[a.L[D1].s_bias + W];
    }
    DV_EPILOGUE(D1, sBias + a.L[D1].s_bias, false);
    // mlp2 first layer: relu(hidden W^T + per-ray (bias + PE term))
    asm volatile("prefetch.global.L1 [%0];" ::"l"(po));  // on its way while the layer runs
    DV_LAYER(D1 + 1, false);
    DV_EPILOGUE(D1 + 1, po, true);
    // mlp2 output: 3 logits -> sigmoid
    if (a.steal) {
      ok &= tc::mbar_wait_bounded(bar_next, phase_next);
      phase_next ^= 1u;
      const int got = ok ? tc::clc_answer(answer) : -1;
      next = got < 0 ? tiles : got;
    }
    if (AHEAD) seg = load_seg(a, S, next * 128 + t);
    DV_LAYER(D1 + 2, false);
    // a training batch's rays lie apart, so most of its rows come from DRAM: ask for the next tile's
    // (captured 4096-ray step of the 256^3 scene, 304 -> 280 us); a frame's neighbouring rays share
    // theirs, and there it only costs (65,792 rays of the wide grid, 730 -> 745 us a pass)
    if (TERMS > 1 && saving && next * 128 + t < S) {
      const Corners c = corners_of(a, true, seg);
      prefetch_rows<C * 4>(a.grid, c.row, c.dx, c.dy, c.dz);
    }
#undef DV_LAYER
#undef DV_EPILOGUE
    {
      float o[4];
      acc_row4<TERMS>(trow, a.L[D1 + 2].N, o);
      const float* bo = sBias + a.L[D1 + 2].s_bias;
      if (valid && ok)
        a.out4[s] = make_float4(sigma, sigmoidf_acc(o[0] + bo[0]), sigmoidf_acc(o[1] + bo[1]),
                                sigmoidf_acc(o[2] + bo[2]));
    }
    tc::fence_before_sync();
    ok = __syncthreads_and(ok);  // the next gather overwrites A
  }
  if (!ok && t == 0 && a.err) atomicExch(a.err, 1);
  if (saving && t == 0) tc::bulk_wait_all();
  tc::fence_before_sync();
  __syncthreads();
  tc::fence_after_sync();
  if (warp == 0) tc::tmem_dealloc(tmem, NCOLS);
}

// The persistent grid holds as many CTAs per SM as registers, shared memory
// and TMEM (512 columns) allow together (the occupancy API under-reports
// kernels that allocate TMEM).
template <int C, int W, int D1, int BF16, int TERMS, bool TS>
int launch_decode_fwd_tc_as(TcArgs a, cudaStream_t st) {
  // split form: two column blocks of the widest N
  constexpr int NCOLS = TERMS > 1 ? (W == 32 ? 128 : 256) : (W == 32 ? 64 : 128);
  constexpr int KMAX = C > W ? C : W;
  const size_t smem = (size_t)TERMS * a.wbytes + (size_t)a.nbias * 4 + (size_t)TERMS * 128 * KMAX * 2 +
                      (TERMS == 1 ? 128 * COEF * 4 : 0) + 48;
  auto k = decode_fwd_tc<C, W, D1, BF16, NCOLS, TERMS, TS>;
  if (cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) != cudaSuccess) return DV_ERR_CUDA;
  int dev = 0, sms = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  const tc::Residency res = tc::tmem_residency(reinterpret_cast<const void*>(k), smem, NCOLS, 128);
  if (res.dyn_smem != smem) {
    if (cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)res.dyn_smem) != cudaSuccess)
      return DV_ERR_CUDA;
    if (cudaFuncSetAttribute(k, cudaFuncAttributePreferredSharedMemoryCarveout, (int)cudaSharedmemCarveoutMaxShared) !=
        cudaSuccess)
      return DV_ERR_CUDA;
  }
  const long long tiles = (a.S + 127) / 128;
  const long long wave = (long long)sms * res.per_sm;
  // With the count on the host, one CTA per tile, of which the first wave takes
  // over the others' tiles as it goes: with a fixed share each, the slowest CTA
  // of an 800x800 frame ended 25 % after the mean.  With the count on the
  // device most of the capacity's tiles do not exist, and fixed shares of
  // those that do are what one wave can take.
  a.steal = a.S_dev == nullptr && tiles > wave && tiles < (1LL << 31);
  k<<<(unsigned)(a.steal ? tiles : std::min(tiles, wave)), 128, res.dyn_smem, st>>>(a);
  DV_TRY_LAUNCH();
  return DV_OK;
}

// Single-term forms without a save record keep the activations in TMEM; with
// one, every layer's input has to be in shared memory for its bulk copy, and
// the split form's three terms do not fit beside its two column blocks.
template <int C, int W, int D1, int BF16, int TERMS = 1>
int launch_decode_fwd_tc(const TcArgs& a, cudaStream_t st) {
  if constexpr (TERMS == 1) {
    bool fits = a.save == nullptr;
    for (int l = 0; l < D1 + 3; ++l) fits = fits && a.L[l].N <= W + 16;  // outputs in front of the activations' columns
    if (fits) return launch_decode_fwd_tc_as<C, W, D1, BF16, 1, true>(a, st);
  }
  return launch_decode_fwd_tc_as<C, W, D1, BF16, TERMS, false>(a, st);
}

// Exercises the bounded completion wait that every tensor-core kernel uses
// (tc::mbar_wait_bounded): one wait on an mbarrier that nobody arrives on
// must give up after `limit` polls and report it; one after an arrival must
// succeed.  status[0] = 1 if the unarrived wait timed out, status[1] = 0 if
// the arrived wait completed.
__global__ void wait_selftest_kernel(uint32_t limit, int* status) {
  __shared__ __align__(8) uint64_t bar[2];
  tc::mbar_init(&bar[0], 1);
  tc::mbar_init(&bar[1], 1);
  tc::fence_mbar_init();
  status[0] = tc::mbar_wait_bounded(&bar[0], 0, limit) ? 0 : 1;
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(tc::smem_u32(&bar[1])) : "memory");
  status[1] = tc::mbar_wait_bounded(&bar[1], 0, limit) ? 0 : 1;
}

// Weight image gather for a refresh after an optimizer step: out term t, entry
// i = term t of ext[index[i]], where ext[0] = 0 and ext[j] = params[j - 1].
// form 0: FP32 (biases), 1: BF16, 2: FP16, 3: three BF16 terms, each the
// round-to-nearest-even of what the previous ones left (the residuals are
// exact in FP32), term t at out + t * n * 2 bytes.
__global__ void tc_image_kernel(const float* __restrict__ params, long long n_params,
                                const int64_t* __restrict__ index, long long n, int form, void* out) {
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
    const long long j = index[i];
    const float x = (j > 0 && j <= n_params) ? params[j - 1] : 0.f;
    if (form == 0) {
      static_cast<float*>(out)[i] = x;
    } else if (form == 2) {
      static_cast<__half*>(out)[i] = __float2half_rn(x);
    } else {
      __nv_bfloat16* o = static_cast<__nv_bfloat16*>(out);
      float r = x;
      const int terms = form == 3 ? 3 : 1;
      for (int t = 0; t < terms; ++t) {
        const __nv_bfloat16 b = __float2bfloat16_rn(r);
        o[t * n + i] = b;
        r = __fsub_rn(r, __bfloat162float(b));
      }
    }
  }
}

}  // namespace dv

using namespace dv;

// Checks the arguments of a tensor-core forward launch and fills TcArgs;
// terms: operand terms (1, or 3 for the split-operand form; the save record
// then holds two terms of every layer input).
static int decode_fwd_tc_args(TcArgs& a, int kind, int channels, int terms, const void* wblob, int wbytes,
                              const float* bias, int nbias, const int* layers, int n_layers, const float* voxels,
                              const void* voxels16, int nvx, int nvy, int nvz, const float* seg, const int* seg_ray,
                              long long n_seg, const int64_t* n_seg_dev, const float* pe_out, float* out4, void* save,
                              long long save_capacity, int* err) {
  const int d1 = kind == 32 ? 2 : (kind == 64 ? 1 : -1);
  DV_CHECK(d1 > 0 && n_layers == d1 + 3 && n_layers <= TC_MAX_LAYERS, DV_ERR_ARG);
  DV_CHECK((kind == 32 && channels == 32) || (kind == 64 && (channels == 32 || channels == 64)), DV_ERR_UNSUPPORTED);
  DV_CHECK(wblob && bias && layers && voxels && seg && seg_ray && pe_out && out4, DV_ERR_ARG);
  DV_CHECK(wbytes > 0 && wbytes % 16 == 0 && nbias > 0 && nbias % 4 == 0, DV_ERR_ARG);
  DV_CHECK(((uintptr_t)wblob & 15) == 0 && ((uintptr_t)voxels & 15) == 0 && ((uintptr_t)out4 & 15) == 0, DV_ERR_ARG);
  DV_CHECK(voxels16 == nullptr || ((uintptr_t)voxels16 & 15) == 0, DV_ERR_ARG);
  a.grid = voxels;
  a.grid16 = reinterpret_cast<const uint16_t*>(voxels16);
  a.nvx = nvx;
  a.nvy = nvy;
  a.nvz = nvz;
  a.seg = seg;
  a.seg_ray = seg_ray;
  a.S = n_seg;
  a.S_dev = n_seg_dev;
  a.pe_out = pe_out;
  a.out4 = reinterpret_cast<float4*>(out4);
  a.wblob = reinterpret_cast<const uint8_t*>(wblob);
  a.wbytes = wbytes;
  a.bias = bias;
  a.nbias = nbias;
  a.err = err;
  const int W = kind;
  for (int l = 0; l < n_layers; ++l) {
    a.L[l].b_off = layers[4 * l];
    a.L[l].K = layers[4 * l + 1];
    a.L[l].N = layers[4 * l + 2];
    a.L[l].bias_off = layers[4 * l + 3];
    const TcLayer& L = a.L[l];
    // every operand must lie inside the blob, on a 16-byte boundary, with legal MMA shapes
    DV_CHECK(L.K % 16 == 0 && L.N % 16 == 0 && L.N >= 16 && L.N <= 256 && L.b_off % 16 == 0, DV_ERR_ARG);
    DV_CHECK((long long)L.b_off + (long long)L.N * L.K * 2 <= wbytes && L.bias_off + L.N <= nbias, DV_ERR_ARG);
    DV_CHECK(L.N <= (W == 32 ? 64 : 128), DV_ERR_ARG);
  }
  // biases layer by layer in shared memory (N is a multiple of 16, so every layer's are 16-byte aligned)
  a.nbias = 0;
  for (int l = 0; l < n_layers; ++l) {
    a.L[l].s_bias = a.nbias;
    a.nbias += a.L[l].N;
  }
  // the split form's images regrouped in shared memory, layer by layer
  {
    long long off = 0;
    for (int l = 0; l < n_layers; ++l) {
      a.L[l].s_off = (int)off;
      off += 3LL * a.L[l].N * a.L[l].K * 2;
    }
    DV_CHECK(terms == 1 || off <= 3LL * wbytes, DV_ERR_ARG);
  }
  // saved layer inputs: one record of sum(256 K) bytes (per saved term) per 128-segment tile
  if (save != nullptr) {
    const int saved_terms = terms > 1 ? 2 : 1;
    int off = 0;
    for (int l = 0; l < n_layers; ++l) {
      a.save_off[l] = off;
      off += 256 * a.L[l].K * saved_terms;
    }
    a.save = reinterpret_cast<uint8_t*>(save);
    a.save_bytes = off;
    DV_CHECK(((uintptr_t)save & 15) == 0, DV_ERR_ARG);
    DV_CHECK((n_seg + 127) / 128 * (long long)off <= save_capacity, DV_ERR_ARG);
  }
  // layer shapes the kernel assumes
  DV_CHECK(a.L[0].K == channels && a.L[0].N == W, DV_ERR_ARG);
  for (int l = 1; l < d1; ++l) DV_CHECK(a.L[l].K == W && a.L[l].N == W, DV_ERR_ARG);
  DV_CHECK(a.L[d1].K == W && a.L[d1].N >= W + 4, DV_ERR_ARG);
  DV_CHECK(a.L[d1 + 1].K == W && a.L[d1 + 1].N == W && a.L[d1 + 2].K == W && a.L[d1 + 2].N >= 16, DV_ERR_ARG);
  return DV_OK;
}

// The split-operand forward; folded: its record leaves out the input of mlp2's
// first layer, which the folded backward does not read (a fifth of the record:
// captured 4096-ray step of the 256^3 scene, 322 -> 304 us).
static int fwd_split(int kind, int channels, const void* wblob, int wbytes, const float* bias, int nbias,
                     const int* layers, int n_layers, const float* voxels, int nvx, int nvy, int nvz, const float* seg,
                     const int* seg_ray, long long n_seg, const int64_t* n_seg_dev, const float* pe_out, float* out4,
                     void* save, long long save_capacity, bool folded, int* err, void* stream) {
  DV_CHECK(n_seg >= 0, DV_ERR_ARG);
  if (n_seg == 0) return DV_OK;
  TcArgs a{};
  const int rc = decode_fwd_tc_args(a, kind, channels, 3, wblob, wbytes, bias, nbias, layers, n_layers, voxels,
                                    nullptr, nvx, nvy, nvz, seg, seg_ray, n_seg, n_seg_dev, pe_out, out4, save,
                                    save_capacity, err);
  if (rc != DV_OK) return rc;
  if (folded) a.save_off[n_layers - 2] = -1;
  cudaStream_t st = (cudaStream_t)stream;
  if (kind == 32) return launch_decode_fwd_tc<32, 32, 2, 1, 3>(a, st);
  if (channels == 32) return launch_decode_fwd_tc<32, 64, 1, 1, 3>(a, st);
  return launch_decode_fwd_tc<64, 64, 1, 1, 3>(a, st);
}

extern "C" {

int dv_decode_fwd_tc(int kind, int channels, int bf16, const void* wblob, int wbytes, const float* bias, int nbias,
                     const int* layers, int n_layers, const float* voxels, const void* voxels16, int nvx, int nvy,
                     int nvz, const float* seg, const int* seg_ray, long long n_seg, const int64_t* n_seg_dev,
                     const float* pe_out, float* out4, void* save, long long save_capacity, int* err,
                     void* stream) {
  DV_CHECK(n_seg >= 0 && (bf16 == 0 || bf16 == 1), DV_ERR_ARG);
  if (n_seg == 0) return DV_OK;
  TcArgs a{};
  const int rc = decode_fwd_tc_args(a, kind, channels, 1, wblob, wbytes, bias, nbias, layers, n_layers, voxels,
                                    voxels16, nvx, nvy, nvz, seg, seg_ray, n_seg, n_seg_dev, pe_out, out4, save,
                                    save_capacity, err);
  if (rc != DV_OK) return rc;
  cudaStream_t st = (cudaStream_t)stream;
  if (kind == 32) return bf16 ? launch_decode_fwd_tc<32, 32, 2, 1>(a, st) : launch_decode_fwd_tc<32, 32, 2, 0>(a, st);
  if (channels == 32)
    return bf16 ? launch_decode_fwd_tc<32, 64, 1, 1>(a, st) : launch_decode_fwd_tc<32, 64, 1, 0>(a, st);
  return bf16 ? launch_decode_fwd_tc<64, 64, 1, 1>(a, st) : launch_decode_fwd_tc<64, 64, 1, 0>(a, st);
}

int dv_decode_fwd_tc_split(int kind, int channels, const void* wblob, int wbytes, const float* bias, int nbias,
                           const int* layers, int n_layers, const float* voxels, int nvx, int nvy, int nvz,
                           const float* seg, const int* seg_ray, long long n_seg, const int64_t* n_seg_dev,
                           const float* pe_out, float* out4, void* save, long long save_capacity, int* err,
                           void* stream) {
  return fwd_split(kind, channels, wblob, wbytes, bias, nbias, layers, n_layers, voxels, nvx, nvy, nvz, seg, seg_ray, n_seg,
                   n_seg_dev, pe_out, out4, save, save_capacity, false, err, stream);
}

int dv_decode_fwd_tc_folded(int kind, int channels, const void* wblob, int wbytes, const float* bias, int nbias,
                            const int* layers, int n_layers, const float* voxels, int nvx, int nvy, int nvz,
                            const float* seg, const int* seg_ray, long long n_seg, const int64_t* n_seg_dev,
                            const float* pe_out, float* out4, void* save, long long save_capacity, int* err,
                            void* stream) {
  return fwd_split(kind, channels, wblob, wbytes, bias, nbias, layers, n_layers, voxels, nvx, nvy, nvz, seg, seg_ray, n_seg,
                   n_seg_dev, pe_out, out4, save, save_capacity, true, err, stream);
}

long long dv_decode_tc_split_save_bytes(int kind, int channels, long long n_seg) {
  const int d1 = kind == 32 ? 2 : (kind == 64 ? 1 : -1);
  if (d1 < 0 || n_seg < 0) return -1;
  const long long record = 2 * 256LL * (channels + (d1 + 2) * kind);
  return (n_seg + 127) / 128 * record;
}

int dv_wait_selftest(int limit, int* status, void* stream) {
  DV_CHECK(limit > 0 && limit <= (1 << 20) && status, DV_ERR_ARG);
  wait_selftest_kernel<<<1, 1, 0, (cudaStream_t)stream>>>((uint32_t)limit, status);
  DV_TRY_LAUNCH();
  return DV_OK;
}

long long dv_decode_tc_save_bytes(int kind, int channels, long long n_seg) {
  const int d1 = kind == 32 ? 2 : (kind == 64 ? 1 : -1);
  if (d1 < 0 || n_seg < 0) return -1;
  const long long record = 256LL * (channels + (d1 + 2) * kind);
  return (n_seg + 127) / 128 * record;
}

int dv_tc_image(const float* params, long long n_params, const int64_t* index, long long n, int form, void* out,
                void* stream) {
  DV_CHECK(n >= 0 && n_params >= 0 && form >= 0 && form <= 3, DV_ERR_ARG);
  if (n == 0) return DV_OK;
  DV_CHECK(index && out && (params || n_params == 0), DV_ERR_ARG);
  const unsigned blocks = (unsigned)std::min<long long>((n + 255) / 256, 4LL * 152);
  tc_image_kernel<<<blocks, 256, 0, (cudaStream_t)stream>>>(params, n_params, index, n, form, out);
  DV_TRY_LAUNCH();
  return DV_OK;
}

}  // extern "C"
