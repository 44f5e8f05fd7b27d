// Tensor-core (tcgen05) backward of the DIVeR32 decoder with split BF16
// operands: FP32-grade gradients from BF16 tensor cores.
//
// Every FP32 operand is carried as a sum of BF16 terms (tc::split_pair):
//   - delta propagation  dL/d input = delta @ W: delta and W as three terms
//     each, the six products whose term indices add up to at most 2;
//   - weight gradient    dW += delta^T @ activation: two terms each, all four
//     products (FP32 accumulators resident in TMEM for the CTA's life);
//   - bias gradient      dB += delta^T @ ones: the column sums of the two-term
//     delta, also accumulated in TMEM (the PE layer's from a column of ones in the
//     PE tile, which the weight-gradient MMA already reads).
// Products are accumulated in FP32 in TMEM, so the propagated deltas and the
// gradients keep about 2^-24 (propagation) and 2^-16 (weight gradients) of
// relative precision per product; emulating the kernel's arithmetic on the
// CPU gives gradients within a few 1e-7 (grid) and 1e-6 (weights) relative
// of an FP64 backward, where a single BF16 term gives 1e-2.
//
// A tcgen05.mma costs the tensor core about 46 clocks whatever its shape up
// to N = 64 (M = 64 or 128, K = 16), so the layout is chosen for few, wide
// MMAs:
//   - the delta tile is one [128][3 x 48] tile, term i in columns 48i..48i+47;
//     read transposed with M = 128 it puts delta terms 0 and 1 in accumulator
//     rows 0..47 and 48..95 of ONE MMA (rows 96..127 see term 2 and are never
//     read);
//   - the saved activations and the PE tile are [128][2 x 32] tiles, term j
//     in columns 32j..32j+31, so one MMA of N = 64 takes both terms;
//   - the propagation images sit layer by layer with the three weight terms
//     side by side along N: per 16 columns of K, delta_0 x [W0|W1] and
//     delta_1 x [W0|W1] (N = 64), delta_0 x W2 into columns 32..63 and
//     delta_2 x W0 into columns 0..31; the epilogue adds the two column blocks.
// Per 128-segment tile that is 32 propagation, 40 weight-gradient and 24
// bias-gradient MMAs with mlp1's output layer and mlp2's first taken as one
// (40, 48 and 32 layer by layer: see Cfg).
//
// The forward is not recomputed: dv_decode_fwd_tc_split saved, per tile of 128
// segments, every layer's input as a [128][2 x 32] two-term tile (X0, A1, A2,
// hidden, A4; 16 KiB each), and its FP32 out4 gives the colour logits'
// sigmoid.  The record is read into shared memory by bulk async copies, one
// per layer slot.
//
// One CTA per SM, 544 threads in three roles:
//   issuer   (warp 0) issues the MMAs and the record loads
//   chain    (256, warps 1-8) a thread owns one segment row r (TMEM lane r;
//            warps w and w + 4 share a lane quadrant) and half h of its
//            columns: it turns a layer's propagated delta into the next one's
//   scatter  (256) adds the finished tile's feature gradient to the grid
// A layer's propagation is issued and committed first; its gradient MMAs
// follow in the same queue and run while the chain forms the next delta, in
// the other of two delta tiles.  A propagation's commit also covers the
// gradient MMAs queued before it, which is what frees the delta tile and the
// record slot of the layer before.
// Shared memory (at most 226 KiB): the propagation images, the saved record in
// per-layer slots, the PE tile, two delta tiles, a tile of ones, the FP32
// staging rows of the feature gradient and the scatter's corners.  TMEM: all 512
// columns are allocated (64 working; folded 320 weight-gradient and 48
// bias-gradient columns, layer by layer 384 and 64: Cfg::DWCOL, Cfg::DBCOL).
// Measured, captured 4096-ray step of the 256^3 scene (1.26 M segments): 733 us
// with the chain doing the scatter in its waits and every MMA of a layer ahead
// of its epilogue, 625 us in this form with one thread issuing and stepping
// with the chain, 522 us with the issuer's warp running free of it, 513 us with
// the layer loops rolled (instruction cache), 490 us folded, 474 us with two
// staging tiles and the scatter's segments fetched a tile ahead, 424 us with
// the scatter's rows asked for ahead.  What is left is the scatter: folded,
// without its atomics, the kernel takes 330 us, and the atomics alone, rows not
// asked for, 290-310 us at any split of the segments (3.9 M distinct rows, 1.0
// GB read and written, at about half the copy rate).
// Reference semantics: the autograd backward of model/diver.py:159-180.
#include "common.cuh"
#include "integrate.cuh"
#include "mlp.cuh"
#include "tc.cuh"

#include <algorithm>

namespace dv {
namespace bws {

constexpr int C = 32, W = 32;
constexpr int CHAIN = 256;             // the layer chain's threads: two per segment row (warps 1-8)
constexpr int CHAIN_ALL = CHAIN + 32;  // chain and issuer warp
constexpr int SCATTER = 256;           // warps 9-16
constexpr int THREADS = CHAIN_ALL + SCATTER;
constexpr int FD = 48;              // delta columns per term (K of the widest propagation MMA)
constexpr int DW = 3 * FD;          // delta tile columns: the three terms side by side
constexpr int TILE = 128 * 32 * 2;  // one term of a [128][32] BF16 tile
constexpr int DTILE = 128 * FD * 2; // one term's share of the delta tile
constexpr int TMEM_COLS = 512;      // 64 working columns, the weight and the bias gradients
constexpr int PE_ONES = 27;         // the PE tile's column of ones (PE_DIM = 27 values before it)

// The layers that the chain steps through, last to first.
//
// Plain: the decoder's own five, 0 (C->W), 1 (W->W), 2 (W->W+1: sigma,
// hidden), 3 (W+27->W), 4 (W->3).
//
// Folded: mlp1's output layer has no activation, so its hidden part WH and
// mlp2's first layer W2 act as one matrix WF = WH W2, and the steps are
// 0 (C->W), 1 (W->W), 2 (A2 and PE -> sigma and mlp2's hidden), 3 (W->3): a
// fifth less of the MMAs, hand-overs and record bytes.  With delta the
// gradient after WF and GF = A2^T delta,
//   dL/dWH = GF W2^T,   dL/dW2 = WH^T GF + bh (sum delta)^T,   dL/dbh = W2 (sum delta),
// once per CTA.  The forward keeps the two layers, so its ReLU decisions stand.
// dL/dW2 is a sum of two parts in place of one over the hidden layer: where the
// hidden layer is r times smaller than its own two parts, WH^T A2 and bh, its
// error against 64 bits grows with r (measured relative L2, folded / layer by
// layer: r = 1 6e-6 / 7e-6, r = 26 6e-5 to 1.7e-4 / 5e-6 to 9e-6, r = 207 4e-4
// to 1.4e-3 / 4e-5 to 5e-5; default initialisation has r below 1).  Every other
// gradient is as good as layer by layer.
template <bool FOLD>
struct Cfg {
  static constexpr int NL = FOLD ? 4 : 5;
  // staging tiles, and whether the scatter group fetches the next tile's segments ahead (shared memory allows both folded)
  static constexpr int NST = FOLD ? 2 : 1;
  static constexpr bool AHEAD = FOLD;
  static constexpr int PEL = FOLD ? 2 : 3;  // the layer with the PE rows; its bias gradient is column 27 of its PE block
  __host__ __device__ static constexpr int REC(int l) { return FOLD && l == 3 ? 4 : l; }  // its input's tile in the record
  __host__ __device__ static constexpr int IN(int l) { return l == 0 ? C : (l == PEL ? W + PE_DIM : W); }
  __host__ __device__ static constexpr int OUT(int l) { return l == 2 ? W + 1 : (l == NL - 1 ? 3 : W); }
  __host__ __device__ static constexpr int OUT4(int l) { return pad4(OUT(l)); }
  __host__ __device__ static constexpr int NBLK(int l) { return l == PEL ? 2 : 1; }  // 32-column input blocks
  // weight gradient of layer l: per input block, 64 columns (activation terms 0 and 1)
  __host__ __device__ static constexpr int DWCOL(int l) { return 64 + 64 * l + (l > PEL ? 64 : 0); }
  // bias gradient of layer l != PEL (column 0 of 16)
  __host__ __device__ static constexpr int DBCOL(int l) { return 64 + 64 * (NL + 1) + 16 * (l < PEL ? l : l - 1); }
  __host__ __device__ static constexpr int KPROP(int l) { return l == NL - 1 ? 16 : (l == 2 ? W + 16 : W); }  // propagation K
  // propagation image of layer l in shared memory: [3 terms x 32 rows][KPROP(l)],
  // the three terms side by side along N, layers one after the other
  __host__ __device__ static constexpr int PIMG(int l) { return 32 * KPROP(l) * 2; }  // one term's bytes
  __host__ __device__ static constexpr int POFF(int l) {
    return 3 * 64 * (32 * l + (l > 2 ? 16 : 0) - (l >= NL ? 16 : 0));
  }
};

constexpr uint32_t RECORD = 5 * 2 * TILE;  // saved record of one tile: 5 layer inputs, [128][2 x 32] each
constexpr uint32_t ONES_BYTES = 128 * 16 * 2;  // a [128][16] BF16 tile of ones
constexpr int STAGE = 128 * (C + 4);           // floats of a tile's staging rows
constexpr int COEF = 12;                       // floats per segment: 8 corner weights, lower corner's row, row steps

struct Args {
  int nvx, nvy, nvz;
  const float* seg;
  const int* seg_ray;
  long long S;           // segment count, or capacity when S_dev is set
  const int64_t* S_dev;  // optional device-held count (clamped to S)
  const float* pe_feat;  // [B][28]
  const float4* d4;      // [S] (dL/dsigma, dL/drgb)
  const float4* out4;    // [S] (sigma, sigmoid rgb) of the forward
  const uint8_t* saved;  // RECORD bytes per tile
  float* grad_grid;
  float* grad_params;    // packed torch layout
  uint8_t* touched;      // optional: a byte per grid row, set at each segment's lower corner
  int w_off[5], b_off[5];  // of the decoder's own layers
  const uint8_t* wb;     // transposed weight images, three terms of wterm bytes
  int wterm;
  int b_img[5];          // byte offset of layer l's image inside a term
  const float* params;   // folded: the packed parameters
  int* err;
};

// Shared-memory layout (byte offsets).
template <bool FOLD>
struct Layout {
  using P = Cfg<FOLD>;
  uint32_t bb, rec, pe, d, ones, stage, coef, seg, bar;
  __host__ __device__ static Layout make() {
    Layout L;
    L.bb = 0;
    L.rec = (uint32_t)(P::POFF(P::NL) + 1023) / 1024 * 1024;
    L.pe = L.rec + P::NL * 2 * TILE;
    L.d = L.pe + 2 * TILE;
    L.ones = L.d + 2 * 3 * DTILE;
    L.stage = L.ones + ONES_BYTES;
    L.coef = L.stage + P::NST * STAGE * 4;
    L.seg = L.coef + 128 * COEF * 4;
    L.bar = L.seg + (P::AHEAD ? 128 * 6 * 4 : 0);
    return L;
  }
  // barriers: propagation, NL record slots, the last MMAs; then the TMEM address and the stop flag
  __host__ __device__ uint32_t bytes() const { return bar + 8 * (2 + P::NL) + 16; }
};

// Writes n values (multiple of 8) of row r, columns c0.., as three BF16 terms
// into the delta tile (term i in columns FD * i + c).
__device__ __forceinline__ void put3(uint8_t* D, int r, int c0, const float* v, int n) {
#pragma unroll
  for (int c = 0; c < n; c += 8) {
    uint32_t x[3], y[3], z[3], u[3];
    tc::split_pair<3>(v[c], v[c + 1], x);
    tc::split_pair<3>(v[c + 2], v[c + 3], y);
    tc::split_pair<3>(v[c + 4], v[c + 5], z);
    tc::split_pair<3>(v[c + 6], v[c + 7], u);
#pragma unroll
    for (int i = 0; i < 3; ++i)
      *reinterpret_cast<uint4*>(D + tc::kmajor_offset(r, FD * i + c0 + c, DW)) = make_uint4(x[i], y[i], z[i], u[i]);
  }
}

// Same with two terms into a [128][2 x 32] tile (term j in columns 32 j + c).
__device__ __forceinline__ void put2(uint8_t* tile, int r, int c0, const float* v, int n) {
#pragma unroll
  for (int c = 0; c < n; c += 8) {
    uint32_t x[2], y[2], z[2], u[2];
    tc::split_pair<2>(v[c], v[c + 1], x);
    tc::split_pair<2>(v[c + 2], v[c + 3], y);
    tc::split_pair<2>(v[c + 4], v[c + 5], z);
    tc::split_pair<2>(v[c + 6], v[c + 7], u);
#pragma unroll
    for (int j = 0; j < 2; ++j)
      *reinterpret_cast<uint4*>(tile + tc::kmajor_offset(r, 32 * j + c0 + c, 64)) = make_uint4(x[j], y[j], z[j], u[j]);
  }
}

// Zeroes v[i] where the activation (leading term of a [128][2 x 32] record
// tile, row r, columns c0..c0+n-1) is not positive: the ReLU derivative.  The
// leading BF16 term has the sign of the FP32 activation (and is zero only with it).
__device__ __forceinline__ void relu_mask(const uint8_t* tile, int r, int c0, float* v, int n) {
#pragma unroll
  for (int c = 0; c < n; c += 8) {
    const uint4 w = *reinterpret_cast<const uint4*>(tile + tc::kmajor_offset(r, c0 + c, 64));
    const uint32_t x[4] = {w.x, w.y, w.z, w.w};
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      if (!(tc::bf_lo(x[j]) > 0.f)) v[c + 2 * j] = 0.f;
      if (!(tc::bf_hi(x[j]) > 0.f)) v[c + 2 * j + 1] = 0.f;
    }
  }
}

// Propagation: TMEM columns [0, 32) + [32, 64) = delta [128][K] x W^T, for
// delta three terms of the delta tile (term i starting at column FD i) and
// the layer's image [3 x 32][K] (weight term j in rows 32j..32j+31): per 16
// columns of K, delta_0 x [W0|W1] and delta_1 x [W0|W1] into columns 0..63,
// delta_0 x W2 into 32..63 and delta_2 x W0 into 0..31.
__device__ __forceinline__ void mma_prop(uint32_t by, uint32_t tmem, const uint8_t* D, const uint8_t* img, int K) {
  constexpr uint32_t sboA = (DW / 8) * 128, term = (FD / 8) * 128;
  const uint64_t a0 = tc::smem_desc(tc::smem_u32(D), 128, sboA);
  const uint64_t b0 = tc::smem_desc(tc::smem_u32(img), 128, (uint32_t)(K / 8) * 128);
  const uint32_t i64 = tc::idesc_f16(128, 64, 1), i32 = tc::idesc_f16(128, 32, 1);
#pragma unroll 1
  for (int k = 0; k < K / 16; ++k) {
    const uint64_t ak = tc::desc_plus(a0, k * 256), bk = tc::desc_plus(b0, k * 256);
    tc::mma_f16_by(by, tmem, ak, bk, i64, k > 0 ? 1u : 0u);
    tc::mma_f16_by(by, tmem, tc::desc_plus(ak, term), bk, i64, 1u);
    tc::mma_f16_by(by, tmem + 32, ak, tc::desc_plus(bk, 2 * 32 * K * 2), i32, 1u);
    tc::mma_f16_by(by, tmem, tc::desc_plus(ak, 2 * term), bk, i32, 1u);
  }
}

// Transposed view of the delta tile as the A operand of the gradient MMAs:
// M = 128 rows = delta tile columns 0..127 (terms 0 and 1 in rows 0..47 and
// 48..95), K = 16 segments per MMA.
__device__ __forceinline__ uint64_t delta_t_desc(const uint8_t* D) {
  constexpr uint32_t lbo = (DW / 8) * 128;  // next 8 segments
  return tc::smem_desc(tc::smem_u32(D), lbo, 128);
}
constexpr uint32_t DELTA_T_K = 2 * (DW / 8) * 128;  // bytes per 16 segments of that view

// Weight gradient over the tile's 128 segments: TMEM dW[128][64] +=
// delta^T x act, act a [128][2 x 32] tile read transposed (N = 64: both terms).
__device__ __forceinline__ void mma_dw(uint32_t by, uint32_t tmem, const uint8_t* D, const uint8_t* act, bool accumulate) {
  const uint32_t idesc = tc::idesc_f16(128, 64, 1) | (1u << 15) | (1u << 16);
  constexpr uint32_t lboB = (64 / 8) * 128;
  const uint64_t a0 = delta_t_desc(D), b0 = tc::smem_desc(tc::smem_u32(act), lboB, 128);
#pragma unroll 1
  for (int k = 0; k < 8; ++k)
    tc::mma_f16_by(by, tmem, tc::desc_plus(a0, k * DELTA_T_K), tc::desc_plus(b0, k * 2 * lboB), idesc,
                (accumulate || k > 0) ? 1u : 0u);
}

// Bias gradient over the tile's 128 segments: TMEM dB[128][16] += delta^T x
// ones, every column the column sum of the delta (terms 0 and 1 in rows 0..47
// and 48..95; the ones are exact in BF16 and any reading of the all-ones tile
// is the same).
__device__ __forceinline__ void mma_db(uint32_t by, uint32_t tmem, const uint8_t* D, const uint8_t* ones, bool accumulate) {
  const uint32_t idesc = tc::idesc_f16(128, 16, 1) | (1u << 15) | (1u << 16);
  constexpr uint32_t lboB = (16 / 8) * 128;
  const uint64_t a0 = delta_t_desc(D), b0 = tc::smem_desc(tc::smem_u32(ones), lboB, 128);
#pragma unroll 1
  for (int k = 0; k < 8; ++k)
    tc::mma_f16_by(by, tmem, tc::desc_plus(a0, k * DELTA_T_K), tc::desc_plus(b0, k * 2 * lboB), idesc,
                (accumulate || k > 0) ? 1u : 0u);
}

// Named barriers (0 is __syncthreads): a delta in place (the chain arrives, the
// issuer waits); the whole chain with the issuer; the scatter group; the
// staging rows handed to it (the chain arrives, it waits) and taken by it (the
// other way round).
constexpr int BAR_DELTA = 1, BAR_CHAIN = 2, BAR_SCATTER = 3, BAR_STAGED = 4, BAR_STOP = 6, BAR_TAKEN = 7;  // STAGED and TAKEN: one per staging tile

__device__ __forceinline__ void named_sync(int id, int n) { asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(n) : "memory"); }
__device__ __forceinline__ void named_arrive(int id, int n) {
  __threadfence_block();
  asm volatile("bar.arrive %0, %1;" ::"r"(id), "r"(n) : "memory");
}
// AND of `v` over the n threads of named barrier `id` (all of them wait).
__device__ __forceinline__ bool named_and(int id, int n, bool v) {
  uint32_t r;
  asm volatile(
      "{\n .reg .pred p, q;\n setp.ne.u32 q, %1, 0;\n bar.red.and.pred p, %2, %3, q;\n selp.u32 %0, 1, 0, p;\n}\n"
      : "=r"(r)
      : "r"((uint32_t)v), "r"(id), "r"(n)
      : "memory");
  return r != 0;
}

// Asynchronous copy of one float into this thread's own shared memory, and the wait for all of this thread's.
__device__ __forceinline__ void cp_async4(float* dst, const float* src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(tc::smem_u32(dst)), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_all;" ::: "memory"); }

// Scatter of a finished tile's feature gradient into the corner rows of its
// segments: thread i takes channel quad q = i % 8 of the HRUN consecutive
// segments HRUN * (i / 8)...  Consecutive segments of a ray usually sit in
// face-adjacent voxels and share four corner rows: the shared corners'
// contributions are added in registers and reach memory with one atomic
// instead of two.  A merge needs both voxels whole (upper corners not
// clamped) and lower corners one row step apart along one axis, so the merged
// rows are the same rows.
constexpr int HRUN = 4;
static_assert((C / 4) * (128 / HRUN) == SCATTER, "one thread per (channel quad, run)");

// Corner weights and rows of the segment at sg (0 steps where the upper corner is
// clamped; rows fit 32 bits, 2^32 rows are twice the device's memory), and its
// row mark for the next step's sparse clear (dv_mark_corner_rows' rule).
__device__ __forceinline__ void put_coefs(const Args& a, float* coef, const float* sg) {
  const SegCorner sc = segment_corners(sg[0], sg[1], sg[2], sg[3], sg[4], sg[5], a.nvx, a.nvy, a.nvz);
  const uint32_t row = ((uint32_t)sc.z * a.nvy + sc.y) * a.nvx + sc.x;
  float4* c = reinterpret_cast<float4*>(coef);
  c[0] = make_float4(sc.w[0], sc.w[1], sc.w[2], sc.w[3]);
  c[1] = make_float4(sc.w[4], sc.w[5], sc.w[6], sc.w[7]);
  const uint32_t dx = sc.x1 - sc.x, dy = (uint32_t)(sc.y1 - sc.y) * a.nvx, dz = (uint32_t)(sc.z1 - sc.z) * a.nvx * a.nvy;
  reinterpret_cast<uint4*>(c)[2] = make_uint4(row, dx, dy, dz);
  // an atomic that misses L2 costs more than a load that does (474 -> 424 us; a tile earlier 436)
  prefetch_rows<C * 4>(a.grad_grid, row, dx, dy, dz);
  if (a.touched) a.touched[row] = 1;
}

__device__ __forceinline__ uint32_t coef_row(const uint4 m, int j) {
  return m.x + ((j & 1) ? m.y : 0u) + ((j & 2) ? m.z : 0u) + ((j & 4) ? m.w : 0u);
}

// n: segments of this thread's run (0..HRUN); st: its quad in the run's first
// staging row.
__device__ __forceinline__ void scatter_run(const Args& a, const float* coef, int n, const float* st, int q, int taken) {
  float4 pend[8];  // contributions of the previous segment's corners not yet in memory
  uint4 pm = make_uint4(0u, 0u, 0u, 0u);
  bool pwhole = false;
  float* grid = a.grad_grid + 4 * q;
#pragma unroll 1
  for (int k = 0; k < n; ++k) {
    const float4 g = *reinterpret_cast<const float4*>(st + k * (C + 4));
    const float4 wa = *reinterpret_cast<const float4*>(coef + k * COEF);
    const float4 wb = *reinterpret_cast<const float4*>(coef + k * COEF + 4);
    const uint4 m = *reinterpret_cast<const uint4*>(coef + k * COEF + 8);
    const float w[8] = {wa.x, wa.y, wa.z, wa.w, wb.x, wb.y, wb.z, wb.w};
    const bool whole = m.y != 0u && m.z != 0u && m.w != 0u;
    int axis = -1;
    bool up = false;
    if (k > 0 && whole && pwhole) {
      const uint32_t d = m.x - pm.x, e = pm.x - m.x;
      if (d == m.y || e == m.y) axis = 0;
      if (d == m.z || e == m.z) axis = 1;
      if (d == m.w || e == m.w) axis = 2;
      up = d < e;
    }
    if (k > 0) {  // the previous segment's corners off the shared face go to memory
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        const bool shared = axis >= 0 && ((j >> axis) & 1) == (up ? 1 : 0);
        if (!shared) red_add4(grid + (long long)coef_row(pm, j) * C, pend[j]);
      }
    }
    float4 nx[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      float4 c = make_float4(w[j] * g.x, w[j] * g.y, w[j] * g.z, w[j] * g.w);
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
  }
  named_arrive(taken, CHAIN + SCATTER);
  if (n > 0) {
#pragma unroll
    for (int j = 0; j < 8; ++j) red_add4(grid + (long long)coef_row(pm, j) * C, pend[j]);
  }
}

// The chain's side of a delta hand-over: its generic-proxy shared-memory
// writes before the tensor core's reads, its TMEM reads before the next MMAs'
// writes.
__device__ __forceinline__ void delta_ready() {
  tc::fence_before_sync();
  tc::fence_async_smem();
  named_arrive(BAR_DELTA, CHAIN_ALL);
}

// PE tile row r, columns 16h..16h+15 (PE_DIM = 27 values, then a one in
// column PE_ONES for the layer's bias gradient, zeros after), two terms.
__device__ __forceinline__ void load_pe(const Args& a, int ray, int h, float* v) {
  const float* pf = a.pe_feat + (long long)ray * PE_PAD + 16 * h;
#pragma unroll
  for (int i = 0; i < 16; ++i) v[i] = (16 * h + i < PE_DIM) ? __ldg(pf + i) : (16 * h + i == PE_ONES ? 1.f : 0.f);
}

// Delta of the colour logits (dL/drgb * sigmoid') into columns 0..15 of row r.
__device__ __forceinline__ void write_delta4(uint8_t* D, int r, float4 g, float4 oc) {
  float v[16];
#pragma unroll
  for (int i = 0; i < 16; ++i) v[i] = 0.f;
  v[0] = g.y * oc.y * (1.f - oc.y);
  v[1] = g.z * oc.z * (1.f - oc.z);
  v[2] = g.w * oc.w * (1.f - oc.w);
  put3(D, r, 0, v, 16);
}

// This thread's row of the propagation result, columns c..c+15 (taddr =
// lane base + c): the two column blocks of mma_prop added.
__device__ __forceinline__ void prop_row16(uint32_t taddr, float* v) {
  float b[16];
  tc::ld_32x32b_x16(taddr, v);
  tc::ld_32x32b_x16(taddr + 32, b);
  tc::ld_wait();
#pragma unroll
  for (int i = 0; i < 16; ++i) v[i] += b[i];
}

// Same for columns 0..31.
__device__ __forceinline__ void prop_row32(uint32_t taddr, float* v) {
  prop_row16(taddr, v);
  prop_row16(taddr + 16, v + 16);
}

// One tile per step of the persistent loop: the layer steps, each the
// propagation, its gradient MMAs and the epilogue that forms the next delta;
// the last stages the tile's feature gradient (FP32) for the scatter group
// (folded: in one of two staging tiles, so neither group waits for the other's
// slow tile; and the group's segments come a tile ahead).
// The saved record sits in a slot per layer step (four folded, five layer by
// layer), each with its own mbarrier: a
// slot is refilled with the next input of that layer once the MMAs that read
// it are done, so the loads run behind the steps in between.  What the chain
// reads from global memory for the next tile (ray, PE row, the first delta's
// inputs) is loaded before a wait and used after it.  Waits are bounded: a
// thread whose wait gave up goes on through the tile, and all stop at its end.
template <bool FOLD>
__global__ void __launch_bounds__(THREADS, 1) decode_bwd_tc_split_kernel(const Args a) {
  using P = Cfg<FOLD>;
  constexpr int NL = P::NL, PEL = P::PEL;
  static_assert(P::POFF(3) == P::POFF(2) + 3 * P::PIMG(2) && P::POFF(NL) == P::POFF(NL - 1) + 3 * P::PIMG(NL - 1),
                "images one after the other");
  static_assert(P::DBCOL(NL - 1) + 16 <= TMEM_COLS, "TMEM columns");
  extern __shared__ __align__(1024) uint8_t smem[];
  const Layout<FOLD> lay = Layout<FOLD>::make();
  uint8_t* Bb = smem + lay.bb;
  uint8_t* REC = smem + lay.rec;
  uint8_t* PE = smem + lay.pe;
  uint8_t* ONES = smem + lay.ones;
  float* stage = reinterpret_cast<float*>(smem + lay.stage);  // [128][C + 4] FP32
  float* coefs = reinterpret_cast<float*>(smem + lay.coef);   // [128][COEF]
  uint64_t* bar = reinterpret_cast<uint64_t*>(smem + lay.bar);
  uint64_t* bar_rec = bar + 1;  // [NL]: completion of slot l's record load
  uint64_t* bar_end = bar + 1 + NL;
  uint32_t* tslot = reinterpret_cast<uint32_t*>(bar + 2 + NL);
  volatile uint32_t* stop = tslot + 1;  // the chain gave up: nothing was staged

  const int t = threadIdx.x, warp = __shfl_sync(0xffffffffu, t >> 5, 0);
  const long long S = segment_total(a.S, a.S_dev);
  const long long tiles = (S + 127) / 128;

  // propagation images, regrouped layer by layer with the three terms side by side
#pragma unroll
  for (int l = 0; l < NL; ++l)
    for (int i = t; i < 3 * P::PIMG(l) / 16; i += THREADS) {
      const int j = i / (P::PIMG(l) / 16), o = i % (P::PIMG(l) / 16);
      reinterpret_cast<uint4*>(Bb + P::POFF(l))[i] =
          __ldg(reinterpret_cast<const uint4*>(a.wb + j * a.wterm + a.b_img[l]) + o);
    }
  for (int i = t; i < 2 * 3 * DTILE / 16; i += THREADS) reinterpret_cast<uint4*>(smem + lay.d)[i] = make_uint4(0, 0, 0, 0);
  for (int i = t; i < (int)ONES_BYTES / 16; i += THREADS)
    reinterpret_cast<uint4*>(ONES)[i] = make_uint4(0x3f803f80u, 0x3f803f80u, 0x3f803f80u, 0x3f803f80u);  // bf16 1.0
  if (t == 0) {
    tc::mbar_init(bar, 1);
    tc::mbar_init(bar_end, 1);
    for (int l = 0; l < NL; ++l) tc::mbar_init(bar_rec + l, 1);
    tc::fence_mbar_init();
    *stop = 0;
  }
  if (warp == 0) {
    tc::tmem_alloc(tslot, TMEM_COLS);
    tc::tmem_relinquish();
  }
  tc::fence_before_sync();
  tc::fence_async_smem();
  __syncthreads();
  tc::fence_after_sync();
  const uint32_t tmem = *tslot;

  bool ok = true, first = true;  // first: no tile done yet
  if (warp == 0) {
    // ---- issuer
    const uint32_t by = tc::elect_one();
    uint32_t phase_rec = 0;  // bit l = parity of slot l's next completion
    uint32_t pending = 0;    // slots with a load in flight
    uint32_t db = 0;         // the delta tile of the next step
    auto load_slot = [&](int l, long long tile) {
      if (by) {
        tc::mbar_arrive_expect_tx(bar_rec + l, 2 * TILE);
        tc::bulk_load(REC + l * 2 * TILE, a.saved + tile * (long long)RECORD + P::REC(l) * 2 * TILE, 2 * TILE, bar_rec + l);
      }
      pending |= 1u << l;
    };
    if (blockIdx.x < tiles)
      for (int l = 0; l < NL; ++l) load_slot(l, blockIdx.x);
    for (long long tile = blockIdx.x; tile < tiles && ok; tile += gridDim.x) {
      const long long next = tile + gridDim.x;
#pragma unroll 1
      for (int l = NL - 1; l >= 0; --l) {
        const uint8_t* D = smem + lay.d + db * (3 * DTILE);
        named_sync(BAR_DELTA, CHAIN_ALL);  // this delta is in place; the previous propagation was waited for
        tc::fence_after_sync();
        mma_prop(by, tmem, D, Bb + P::POFF(l), P::KPROP(l));
        tc::mma_commit_by(by, bar);
        // that propagation's commit covered the gradient MMAs of two steps ago: their slot takes
        // its next input (layers 0 and 1: this tile's)
        const int f = (l + 2) % NL;
        if (f >= 2 ? next < tiles : !first) load_slot(f, f >= 2 ? next : tile);
        const bool arrived = tc::mbar_wait_bounded(bar_rec + l, (phase_rec >> l) & 1u);
        if (arrived) {
          phase_rec ^= 1u << l;
          pending &= ~(1u << l);
          const uint8_t* act = REC + l * 2 * TILE;  // this layer's input, two terms TILE apart
          mma_dw(by, tmem + P::DWCOL(l), D, act, !first);
          if (l == PEL)
            mma_dw(by, tmem + P::DWCOL(PEL) + 64, D, PE, !first);  // with its bias gradient (the ones column)
          else
            mma_db(by, tmem + P::DBCOL(l), D, ONES, !first);
        }
        ok &= arrived;
        db ^= 1u;
      }
      first = false;
      ok = named_and(BAR_CHAIN, CHAIN_ALL, ok);
    }
    // what is still in flight ends before the CTA frees its shared memory and
    // TMEM: the last MMAs, and after a failure record loads (bounded waits)
    if (!first) {
      tc::mma_commit_by(by, bar_end);
      for (int l = 0; l < NL; ++l)
        if ((pending >> l) & 1u) tc::mbar_wait_bounded(bar_rec + l, (phase_rec >> l) & 1u);
      ok &= tc::mbar_wait_bounded(bar_end, 0);
      ok = named_and(BAR_CHAIN, CHAIN_ALL, ok);
      if (!ok && by && a.err) atomicExch(a.err, 1);
    }
  } else if (warp > CHAIN / 32) {
    // ---- scatter group
    const int i = t - CHAIN_ALL, q = i % (C / 4), ls = (i / (C / 4)) * HRUN;
    float* ahead = reinterpret_cast<float*>(smem + lay.seg) + 6 * i;  // this thread's own segment of the next tile
    auto fetch = [&](long long tile) {
      if (P::AHEAD && i < 128 && tile < tiles && tile * 128 + i < S)
#pragma unroll
        for (int j = 0; j < 6; ++j) cp_async4(ahead + j, a.seg + (tile * 128 + i) * 6 + j);
    };
    fetch(blockIdx.x);
    int p = 0;  // the staging tile
    for (long long tile = blockIdx.x; tile < tiles; tile += gridDim.x, p = (p + 1) % P::NST) {
      const long long s0 = tile * 128;
      if (P::AHEAD) cp_async_wait();
      if (i < 128 && s0 + i < S) put_coefs(a, coefs + i * COEF, P::AHEAD ? ahead : a.seg + (s0 + i) * 6);
      fetch(tile + gridDim.x);
      named_sync(BAR_SCATTER, SCATTER);
      named_sync(BAR_STAGED + p, CHAIN + SCATTER);
      if (*stop) break;
      const long long left = S - (s0 + ls);
      scatter_run(a, coefs + ls * COEF, left >= HRUN ? HRUN : (left > 0 ? (int)left : 0),
                  stage + p * STAGE + ls * (C + 4) + 4 * q, q, BAR_TAKEN + p);
      named_sync(BAR_SCATTER, SCATTER);  // the next tile's corners overwrite these
    }
    if (P::AHEAD) cp_async_wait();  // none left in flight after a break
  } else {
    // ---- chain
    const uint32_t lane = (uint32_t)((warp & 3) * 32) << 16;
    const uint32_t trow = tmem + lane;
    const int r = 32 * (warp & 3) + (t & 31), h = warp > 4 ? 1 : 0;
    uint32_t phase = 0, phase_rec = 0, db = 0;
    uint32_t done = 0;  // tiles staged
    float v[32];
    // the CTA's first tile: PE tile, first delta
    long long tile = blockIdx.x;
    if (tile < tiles) {
      const long long s = tile * 128 + r;
      const bool valid = s < S;
      load_pe(a, valid ? __ldg(a.seg_ray + s) : 0, h, v);
      put2(PE, r, 16 * h, v, 16);
      if (h == 0)
        write_delta4(smem + lay.d, r, valid ? a.d4[s] : make_float4(0.f, 0.f, 0.f, 0.f),
                     valid ? a.out4[s] : make_float4(0.f, 0.f, 0.f, 0.f));
      delta_ready();
    }
    for (; tile < tiles && ok; tile += gridDim.x) {
      const long long s = tile * 128 + r;
      const bool valid = s < S;
      const long long next = tile + gridDim.x;
      const long long sn = next * 128 + r;
      const bool valid_next = next < tiles && sn < S;
      const float gx = valid ? a.d4[s].x : 0.f;  // dL/dsigma of this row (layer 2's delta)
      const int ray_next = valid_next ? __ldg(a.seg_ray + sn) : 0;
      float4 gn = make_float4(0.f, 0.f, 0.f, 0.f), on = gn;  // the next tile's first delta
      float pe[16];                                          // the next tile's PE row
      // layers last to first
#pragma unroll 1
      for (int l = NL - 1; l >= 0; --l) {
        const uint8_t* act = REC + l * 2 * TILE;  // this layer's input, two terms TILE apart
        uint8_t* Dn = smem + lay.d + (db ^ 1u) * (3 * DTILE);
        if (l == PEL - 1 && next < tiles) load_pe(a, ray_next, h, pe);
        if (l == 1 && valid_next && h == 0) {
          gn = a.d4[sn];
          on = a.out4[sn];
        }
        // this layer's input for the ReLU masks, and its propagation
        ok &= tc::mbar_wait_bounded(bar_rec + l, (phase_rec >> l) & 1u);
        phase_rec ^= 1u << l;
        ok &= tc::mbar_wait_bounded(bar, phase);
        phase ^= 1u;
        tc::fence_after_sync();
        if (l == 3) {
          // delta of layer 2: (dL/dsigma, that of its other 32 outputs) in columns 0..32, zeros to
          // 47; half 0 writes columns 0..23, half 1 columns 24..47
          prop_row32(trow, v);
          if (FOLD) relu_mask(act, r, 0, v, 32);
          float w[24];
          if (h == 0) {
            w[0] = gx;
#pragma unroll
            for (int i = 1; i < 24; ++i) w[i] = v[i - 1];
          } else {
#pragma unroll
            for (int i = 0; i < 24; ++i) w[i] = (i + 23 < W) ? v[i + 23] : 0.f;
          }
          put3(Dn, r, 24 * h, w, 24);
        } else if (l > 0) {
          prop_row16(trow + 16 * h, v);
          relu_mask(act, r, 16 * h, v, 16);  // this layer's input is relu of the previous layer's output
          put3(Dn, r, 16 * h, v, 16);
          // layer PEL's gradient MMAs are done with this tile's PE: the next tile's goes in
          if (l == PEL - 1 && next < tiles) put2(PE, r, 16 * h, pe, 16);
        } else {
          // the next tile's first delta; then dL/dfeature (FP32) to the staging rows, once the
          // scatter group has taken the rows before them
          prop_row16(trow + 16 * h, v);
          if (next < tiles) {
            if (h == 0) write_delta4(Dn, r, gn, on);
            delta_ready();
          }
          if (done >= P::NST) named_sync(BAR_TAKEN + done % P::NST, CHAIN + SCATTER);
          float* st = stage + (done % P::NST) * STAGE + r * (C + 4) + 16 * h;
#pragma unroll
          for (int i = 0; i < 16; i += 4)
            *reinterpret_cast<float4*>(st + i) =
                valid ? make_float4(v[i], v[i + 1], v[i + 2], v[i + 3]) : make_float4(0.f, 0.f, 0.f, 0.f);
        }
        if (l > 0) delta_ready();
        db ^= 1u;
      }
      first = false;
      ok = named_and(BAR_CHAIN, CHAIN_ALL, ok);
      if (!ok && t == 32) *stop = 1;
      if (!ok) named_sync(BAR_STOP, CHAIN);
      named_arrive(BAR_STAGED + done % P::NST, CHAIN + SCATTER);
      ++done;
    }
    if (ok)  // the last tiles'
      for (uint32_t u = done > P::NST ? done - P::NST : 0; u < done; ++u) named_sync(BAR_TAKEN + u % P::NST, CHAIN + SCATTER);
    if (!first) {
      tc::fence_before_sync();
      ok = named_and(BAR_CHAIN, CHAIN_ALL, ok);  // the issuer has seen the last MMAs end
      tc::fence_after_sync();
    }
    // ---- flush: accumulator row m holds delta term 0 (m < 48) or 1 (48 <= m < 96) of
    // output o = m % 48; per input block, columns c and 32 + c hold activation terms 0
    // and 1 of input c.  Rows of both delta terms add into the same gradient entries.
    if (ok && !first) {
      const int o = r < FD ? r : r - FD;
      const bool row = r < 2 * FD;
      // folded: GF (row o: output o, sigma first), W2 and WH in shared memory (the records' part)
      constexpr int LD = W + 1;
      float* G = reinterpret_cast<float*>(REC);  // [W + 1][LD]
      float* W2 = G + LD * LD;                   // [h][j]
      float* WH = W2 + W * LD;                   // [i][h]
      float* DB = WH + W * LD;                   // sum of delta [W]
      const int ct = t - 32;                     // this thread's number in the chain
      if (FOLD) {
        for (int i = ct; i < (W + 1) * LD; i += CHAIN) G[i] = 0.f;
        for (int i = ct; i < W; i += CHAIN) DB[i] = 0.f;
        for (int i = ct; i < W * W; i += CHAIN) {
          const int x = i / W, y = i % W;
          W2[x * LD + y] = __ldg(a.params + a.w_off[3] + i);
          WH[x * LD + y] = __ldg(a.params + a.w_off[2] + x * (W + 4) + 1 + y);
        }
        named_sync(BAR_CHAIN, CHAIN);
      }
#pragma unroll
      for (int l = 0; l < NL; ++l) {
        const int ol = FOLD && l == 3 ? 4 : l;  // the decoder's own layer (the folded one: see below)
#pragma unroll
        for (int b = 0; b < P::NBLK(l); ++b) {
          float u[16];
          tc::ld_32x32b_x16(tmem + lane + P::DWCOL(l) + 64 * b + 16 * h, v);
          tc::ld_32x32b_x16(tmem + lane + P::DWCOL(l) + 64 * b + 32 + 16 * h, u);
          tc::ld_wait();
          if (row && o < P::OUT(l)) {
#pragma unroll
            for (int i = 0; i < 16; ++i) {
              const int c = 32 * b + 16 * h + i;
              if (c >= P::IN(l)) continue;
              if (!FOLD || l != 2) {
                atomicAdd(a.grad_params + a.w_off[ol] + c * pad4(P::OUT(l)) + o, v[i] + u[i]);
              } else if (b == 0) {
                atomicAdd(G + o * LD + c, v[i] + u[i]);
              } else if (o > 0) {  // PE rows of mlp2's first layer
                atomicAdd(a.grad_params + a.w_off[3] + c * W + o - 1, v[i] + u[i]);
              }
            }
            // the PE block's column of ones
            if (l == PEL && b == 1 && h == 1) {
              const float sum = v[PE_ONES - 16] + u[PE_ONES - 16];
              if (!FOLD) {
                atomicAdd(a.grad_params + a.b_off[l] + o, sum);
              } else if (o == 0) {
                atomicAdd(a.grad_params + a.b_off[2], sum);
              } else {
                atomicAdd(a.grad_params + a.b_off[3] + o - 1, sum);
                atomicAdd(DB + o - 1, sum);
              }
            }
          }
        }
        if (l != PEL && h == 0) {
          tc::ld_32x32b_x16(tmem + lane + P::DBCOL(l), v);
          tc::ld_wait();
          if (row && o < P::OUT(l)) atomicAdd(a.grad_params + a.b_off[ol] + o, v[0]);
        }
      }
      if (FOLD) {
        named_sync(BAR_CHAIN, CHAIN);
        for (int e = ct; e < W * W; e += CHAIN) {
          const int x = e / W, y = e % W;
          // dL/dWH[i = x][h = y] and dL/dW2[h = x][j = y]
          float wh = 0.f, w2 = __ldg(a.params + a.b_off[2] + 1 + x) * DB[y];
#pragma unroll 4
          for (int k = 0; k < W; ++k) {
            wh = fmaf(G[(1 + k) * LD + x], W2[y * LD + k], wh);
            w2 = fmaf(WH[k * LD + x], G[(1 + y) * LD + k], w2);
          }
          atomicAdd(a.grad_params + a.w_off[2] + x * (W + 4) + 1 + y, wh);
          atomicAdd(a.grad_params + a.w_off[3] + e, w2);
        }
        if (ct < W) {
          float bh = 0.f;
          for (int j = 0; j < W; ++j) bh = fmaf(W2[ct * LD + j], DB[j], bh);
          atomicAdd(a.grad_params + a.b_off[2] + 1 + ct, bh);
          atomicAdd(a.grad_params + a.w_off[2] + ct * (W + 4), G[ct]);  // sigma's column
        }
      }
    }
  }
  tc::fence_before_sync();
  __syncthreads();
  tc::fence_after_sync();
  if (warp == 0) tc::tmem_dealloc(tmem, TMEM_COLS);
}

// folded [n + W W]: the packed parameters, then WF[i][j] = sum_h WH[i][h] W2[h][j].
__global__ void __launch_bounds__(256) fold_params_kernel(const float* __restrict__ params, int n,
                                                          float* __restrict__ folded) {
  constexpr int wh = C * W + W + W * W + W;                          // mlp1's output layer (rows of W + 4, sigma first)
  constexpr int w2 = wh + W * (W + 4) + (W + 4);                     // mlp2's first layer
  const int copies = (n + 255) / 256;
  if ((int)blockIdx.x < copies) {
    const int i = blockIdx.x * 256 + threadIdx.x;
    if (i < n) folded[i] = __ldg(params + i);
    return;
  }
  const int e = (blockIdx.x - copies) * 256 + threadIdx.x;  // four blocks
  float f = 0.f;
#pragma unroll 8
  for (int h = 0; h < W; ++h)
    f = fmaf(__ldg(params + wh + (e / W) * (W + 4) + 1 + h), __ldg(params + w2 + h * W + e % W), f);
  folded[n + e] = f;
}

}  // namespace bws
}  // namespace dv

using namespace dv;

// Checks the arguments of a split backward launch and starts it; params: folded.
template <bool FOLD>
static int bwd_split(int kind, int channels, const float* params, const void* wb, int wb_term_bytes, const int* b_layers,
                     int n_layers, int nvx, int nvy, int nvz, const float* seg, const int* seg_ray, long long n_seg,
                     const int64_t* n_seg_dev, const float* pe_feat, const float* d4, const void* saved,
                     long long saved_bytes, const float* out4, float* grad_voxels, float* grad_params,
                     unsigned char* touched, int* err, void* stream) {
  using namespace dv::bws;
  using P = Cfg<FOLD>;
  DV_CHECK(n_seg >= 0, DV_ERR_ARG);
  DV_CHECK(kind == 32 && channels == 32 && n_layers == P::NL, DV_ERR_UNSUPPORTED);
  if (n_seg == 0) return DV_OK;
  DV_CHECK(wb && b_layers && seg && seg_ray && pe_feat && d4 && saved && out4 && grad_voxels && grad_params,
           DV_ERR_ARG);
  DV_CHECK(params || !FOLD, DV_ERR_ARG);
  DV_CHECK(nvx > 0 && nvy > 0 && nvz > 0 && wb_term_bytes > 0 && wb_term_bytes % 16 == 0, DV_ERR_ARG);
  DV_CHECK(((uintptr_t)wb & 15) == 0 && ((uintptr_t)saved & 15) == 0 && ((uintptr_t)out4 & 15) == 0 &&
               ((uintptr_t)grad_voxels & 15) == 0 && ((uintptr_t)d4 & 15) == 0,
           DV_ERR_ARG);
  DV_CHECK((n_seg + 127) / 128 * (long long)RECORD <= saved_bytes, DV_ERR_ARG);
  Args a{};
  a.nvx = nvx;
  a.nvy = nvy;
  a.nvz = nvz;
  a.seg = seg;
  a.seg_ray = seg_ray;
  a.S = n_seg;
  a.S_dev = n_seg_dev;
  a.pe_feat = pe_feat;
  a.d4 = reinterpret_cast<const float4*>(d4);
  a.out4 = reinterpret_cast<const float4*>(out4);
  a.saved = reinterpret_cast<const uint8_t*>(saved);
  a.grad_grid = grad_voxels;
  a.grad_params = grad_params;
  a.touched = touched;
  a.wb = reinterpret_cast<const uint8_t*>(wb);
  a.wterm = wb_term_bytes;
  a.err = err;
  a.params = params;
  // packed torch layout offsets (same rule as dv_decoder_param_count)
  {
    int off = 0;
    const int ins[5] = {C, W, W, W + PE_DIM, W}, outs[5] = {W, W, W + 1, W, 3};
    for (int l = 0; l < 5; ++l) {
      a.w_off[l] = off;
      a.b_off[l] = off + ins[l] * pad4(outs[l]);
      off = a.b_off[l] + pad4(outs[l]);
    }
  }
  // transposed images [N = in][K = out padded to 16], inside one term
  for (int l = 0; l < P::NL; ++l) {
    const int n = l == 0 ? C : W;
    a.b_img[l] = b_layers[3 * l];
    DV_CHECK(b_layers[3 * l + 1] == P::KPROP(l) && b_layers[3 * l + 2] == n, DV_ERR_ARG);
    DV_CHECK(a.b_img[l] % 16 == 0 && a.b_img[l] >= 0, DV_ERR_ARG);
    DV_CHECK((long long)a.b_img[l] + (long long)P::KPROP(l) * n * 2 <= wb_term_bytes, DV_ERR_ARG);
  }
  const Layout<FOLD> lay = Layout<FOLD>::make();
  const size_t smem = lay.bytes();
  auto k = decode_bwd_tc_split_kernel<FOLD>;
  int dev = 0, sms = 0, smem_max = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  cudaDeviceGetAttribute(&smem_max, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
  DV_CHECK((long long)smem <= (long long)smem_max, DV_ERR_UNSUPPORTED);
  if (cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) != cudaSuccess)
    return DV_ERR_CUDA;
  const long long tiles = (n_seg + 127) / 128;
  const long long grid = std::min<long long>(tiles, (long long)sms);
  k<<<(unsigned)grid, THREADS, smem, (cudaStream_t)stream>>>(a);
  DV_TRY_LAUNCH();
  return DV_OK;
}

extern "C" {

int dv_decode_bwd_tc_split(int kind, int channels, const void* wb, int wb_term_bytes, const int* b_layers,
                           int n_layers, int nvx, int nvy, int nvz, const float* seg, const int* seg_ray,
                           long long n_seg, const int64_t* n_seg_dev, const float* pe_feat, const float* d4,
                           const void* saved, long long saved_bytes, const float* out4, float* grad_voxels,
                           float* grad_params, unsigned char* touched, int* err, void* stream) {
  return bwd_split<false>(kind, channels, nullptr, wb, wb_term_bytes, b_layers, n_layers, nvx, nvy, nvz, seg, seg_ray,
                          n_seg, n_seg_dev, pe_feat, d4, saved, saved_bytes, out4, grad_voxels, grad_params, touched, err,
                          stream);
}

int dv_decode_bwd_tc_folded(int kind, int channels, const float* params, const void* wb, int wb_term_bytes,
                            const int* b_layers, int n_layers, int nvx, int nvy, int nvz, const float* seg,
                            const int* seg_ray, long long n_seg, const int64_t* n_seg_dev, const float* pe_feat,
                            const float* d4, const void* saved, long long saved_bytes, const float* out4,
                            float* grad_voxels, float* grad_params, unsigned char* touched, int* err, void* stream) {
  return bwd_split<true>(kind, channels, params, wb, wb_term_bytes, b_layers, n_layers, nvx, nvy, nvz, seg, seg_ray,
                         n_seg, n_seg_dev, pe_feat, d4, saved, saved_bytes, out4, grad_voxels, grad_params, touched, err,
                         stream);
}

int dv_fold_params(int kind, int channels, const float* params, float* folded, void* stream) {
  DV_CHECK(kind == 32 && channels == 32, DV_ERR_UNSUPPORTED);
  DV_CHECK(params && folded, DV_ERR_ARG);
  const int n = dv_decoder_param_count(kind, channels);
  bws::fold_params_kernel<<<(n + 255) / 256 + 4, 256, 0, (cudaStream_t)stream>>>(params, n, folded);
  DV_TRY_LAUNCH();
  return DV_OK;
}

}  // extern "C"
