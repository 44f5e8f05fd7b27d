// Voxel traversal kernels: dense and masked 3D-DDA (training/offline path),
// the octree first-hit search and the 8-hit ray march (real-time path), and
// the prefix sum that turns per-ray counts into CSR segment offsets.
//
// One thread steps one ray (the masked walk's occupancy and output are other
// warps' work); the walk itself is inherently sequential (each crossing is
// computed from the previous, rounded point), so bit-exactness with the
// reference fixes the per-ray order of operations.  What changes
// against the reference is around the walk: outputs are either counted only,
// written to caller-sized padded rows, or written compacted (CSR) so that the
// segment-parallel decoder never touches padding; max(count) is reduced per
// warp before one atomic; launches are stream-ordered with no device sync.
#include "common.cuh"
#include "scan.cuh"

namespace dv {

// WALK_SLOTS: one walk both counts and writes, each ray into its own fixed
// range of `slot` rows (b * slot ...), compacted into CSR lists afterwards.
enum WalkMode { WALK_COUNT = 0, WALK_PADDED = 1, WALK_SEGMENTS = 2, WALK_SLOTS = 3 };

struct WalkArgs {
  int batch;
  int max_n;
  float xyzmin;
  float n;
  float3 o3;        // per-axis grid origin (world)
  float3 n3;        // per-axis extent in voxels
  int mx, my;       // occupancy cells along x and y (masked walk)
  float voxel_size;
  float mask_scale;
  int m;            // occupancy cells per side
  long long cells;  // m^3
  bool fast;        // grid small enough for the reciprocal-based division (< 2^22 voxels per side)
  const float* o;
  const float* v;
  const uint8_t* mask;
  float* inter;
  int* num;
  float* tns;
  int* max_count;
  int* last_step;          // count: per ray, the walk step (1-based) of its last occupied voxel, 0 if none
  const int* stop_step;    // segments: per ray, the step after which the walk may stop (last_step of the count)
  long long slot;          // slots: rows per ray
  const int64_t* offsets;
  float* seg;
  float* seg_t;
  int* seg_ray;
};

__device__ __forceinline__ void warp_max_atomic(int* dst, int value, bool active) {
  const unsigned full = __activemask();
  const int mx = __reduce_max_sync(full, active ? value : 0);
  if (dst != nullptr && (threadIdx.x & 31) == (__ffs(full) - 1)) atomicMax(dst, mx);
}

__device__ __forceinline__ float3 ray_origin_voxel(const float* o, int b, float xyzmin, float vs) {
  return make_float3(__fdiv_rn(__fsub_rn(__ldg(o + 3 * b + 0), xyzmin), vs),
                     __fdiv_rn(__fsub_rn(__ldg(o + 3 * b + 1), xyzmin), vs),
                     __fdiv_rn(__fsub_rn(__ldg(o + 3 * b + 2), xyzmin), vs));
}

__device__ __forceinline__ float3 ray_origin_voxel3(const float* o, int b, float3 o3, float vs) {
  return make_float3(__fdiv_rn(__fsub_rn(__ldg(o + 3 * b + 0), o3.x), vs),
                     __fdiv_rn(__fsub_rn(__ldg(o + 3 * b + 1), o3.y), vs),
                     __fdiv_rn(__fsub_rn(__ldg(o + 3 * b + 2), o3.z), vs));
}

__device__ __forceinline__ float3 load3(const float* p, int b) {
  return make_float3(__ldg(p + 3 * b + 0), __ldg(p + 3 * b + 1), __ldg(p + 3 * b + 2));
}

__device__ __forceinline__ float3 signs(float3 d) {
  return make_float3(step_sign(d.x), step_sign(d.y), step_sign(d.z));
}

// Dense walk: entry point, then every plane crossing while the point stays
// in [0,n]^3.  Reference ray_voxel_intersect.cu:39-150.
template <int MODE, bool FAST>
__device__ __forceinline__ int dense_walk(const WalkArgs& a, int b, float3 p, const float3 d, float t, float* row,
                                          float* trow, int64_t base, int64_t cap) {
  const float3 s = signs(d);
  const float3 r = FAST ? recip3(d) : d;
  int count = 1;
  float3 q;
  float dt;
  const int step_cap = walk_cap(a.n, a.n, a.n);
  int k = 0;
  for (; k < step_cap; ++k) {
    grid_step<FAST>(p, d, r, s, q, dt);
    const float tq = __fadd_rn(t, dt);
    if (outside_closed(q, a.n)) break;
    if (MODE == WALK_PADDED && count < a.max_n) {
      row[3 * count + 0] = q.x;
      row[3 * count + 1] = q.y;
      row[3 * count + 2] = q.z;
      trow[count] = __fmul_rn(tq, a.voxel_size);
    }
    if (MODE == WALK_SEGMENTS && count - 1 < cap) {
      float2* sg = reinterpret_cast<float2*>(a.seg + (base + count - 1) * 6);
      sg[0] = make_float2(p.x, p.y);
      sg[1] = make_float2(p.z, q.x);
      sg[2] = make_float2(q.y, q.z);
      if (a.seg_t) a.seg_t[base + count - 1] = __fmul_rn(t, a.voxel_size);
      if (a.seg_ray) a.seg_ray[base + count - 1] = b;
    }
    ++count;
    p = q;
    t = tq;
  }
  if (k == step_cap) note_cap_hit();
  return count;
}

template <int MODE>
__global__ void __launch_bounds__(256) dense_walk_kernel(const WalkArgs a) {
  const int b = blockIdx.x * blockDim.x + threadIdx.x;
  const bool live = b < a.batch;
  int count = 0;
  if (live) {
    const float3 d = load3(a.v, b);
    float3 p = ray_origin_voxel(a.o, b, a.xyzmin, a.voxel_size);
    float t;
    const bool hit = dir_ok(d) && box_entry(p, d, a.n, t);
    float* row = nullptr;
    float* trow = nullptr;
    int64_t base = 0, cap = 0;
    if (MODE == WALK_PADDED) {
      row = a.inter + (long long)b * a.max_n * 3;
      trow = a.tns + (long long)b * a.max_n;
      if (a.max_n > 0) {
        row[0] = p.x;
        row[1] = p.y;
        row[2] = p.z;
      }
    }
    if (MODE == WALK_SEGMENTS) {
      base = a.offsets[b];
      cap = a.offsets[b + 1] - base;
    }
    if (hit) {
      if (MODE == WALK_PADDED && a.max_n > 0) trow[0] = __fmul_rn(t, a.voxel_size);
      count = (a.fast && recip_ok(d)) ? dense_walk<MODE, true>(a, b, p, d, t, row, trow, base, cap)
                          : dense_walk<MODE, false>(a, b, p, d, t, row, trow, base, cap);
    }
    if (MODE != WALK_SEGMENTS) a.num[b] = count;
  }
  if (MODE != WALK_SEGMENTS) warp_max_atomic(a.max_count, count, live);
}

// Masked walk: (entry, exit) of every voxel whose occupancy byte is set.
// Reference ray_voxel_intersect.cu:203-318.
//
// A ray's crossing points are a dependent chain of some hundred steps; what
// each point means (its voxel, the occupancy byte, the output record) is not.
// So the two are different warps' work.  Warp 0 walks 32 rays, a lane each,
// and does nothing else: it writes chunks of 32 points per ray into a
// double-buffered ring in shared memory.  The other warps take the rays one
// by one, a lane per step of the chunk: the 32 occupancy bytes of a ray's
// chunk are one load per lane, a ballot gives the count and every segment's
// place, and a ray's run goes out as contiguous stores.
//
// What bounds it: a small batch, the walker's step (68 clocks of dependent
// chain measured alone, against 93 with the planes recomputed each step); a
// large one, the hand-over's latency and instruction issue.
template <int NC>
struct WalkRing {
  static constexpr int STEPS = 32, ROW = STEPS + 1;  // points per ray and chunk: the chunk's start and its steps' ends
  float4 pt[2][32 * ROW];                            // (x, y, z, t); rows of 33 keep both access patterns conflict-free
  int steps[2][32];                                  // steps of the chunk that count, if they stay inside the box
  int more[2];                                       // another chunk follows
  float2 out[NC][STEPS * 3];                         // a ray's segments of one chunk on their way out
};

// Ring barriers of slot 0 / 1: FULL (the walker arrives, the consumers wait) and
// EMPTY (the consumers arrive, the walker waits), n threads in all.
template <int ID>
__device__ __forceinline__ void ring_sync(int slot, int n) {
  if (slot)
    asm volatile("bar.sync %0, %1;" ::"n"(ID + 1), "r"(n) : "memory");
  else
    asm volatile("bar.sync %0, %1;" ::"n"(ID), "r"(n) : "memory");
}
template <int ID>
__device__ __forceinline__ void ring_arrive(int slot, int n) {
  if (slot)
    asm volatile("bar.arrive %0, %1;" ::"n"(ID + 1), "r"(n) : "memory");
  else
    asm volatile("bar.arrive %0, %1;" ::"n"(ID), "r"(n) : "memory");
}

// A ray's walk state: the point, the next plane of each axis, the distance.
struct Walk {
  float3 a, B;
  float t;
};

__device__ __forceinline__ float3 next_planes(const float3 a, const float3 s) {
  return make_float3(floorf(__fmaf_rn(a.x, s.x, 1.f)), floorf(__fmaf_rn(a.y, s.y, 1.f)),
                     floorf(__fmaf_rn(a.z, s.z, 1.f)));
}

// grid_step<true>, bit for bit, without recomputing the next plane of an
// axis, floor(a s + 1) s, from the point each time (FRND runs at a quarter of
// the rate and sits on the step's dependent chain).  B = floor(a s + 1) is
// kept instead: an axis that was hit sits on its plane, so its B grows by
// exactly 1; on another axis the coordinate moved towards its plane and B
// stands, unless rounding took a s + 1 up to B + 1, which needs a point within
// a few ulp of the plane.  `gap` takes the smallest distance to a next plane
// met so far: when it ends up below near_plane() the caller redoes its steps
// with EXACT, which recomputes the planes every time.
template <bool EXACT>
__device__ __forceinline__ void walk_step(Walk& w, const float3 d, const float3 r, const float3 s, float& gap) {
  if (EXACT) w.B = next_planes(w.a, s);
  const float gx = __fmaf_rn(w.B.x, s.x, -w.a.x), gy = __fmaf_rn(w.B.y, s.y, -w.a.y), gz = __fmaf_rn(w.B.z, s.z, -w.a.z);
  if (!EXACT) gap = fminf(gap, fminf(fminf(fabsf(gx), fabsf(gy)), fabsf(gz)));
  const float tx = div_by_recip(gx, d.x, r.x), ty = div_by_recip(gy, d.y, r.y), tz = div_by_recip(gz, d.z, r.z);
  const float dt = fminf(tx, fminf(ty, tz));
  const bool hx = dt == tx, hy = !hx && dt == ty, hz = !hx && !hy;
  w.a = make_float3(hx ? __fmul_rn(w.B.x, s.x) : __fmaf_rn(d.x, dt, w.a.x),
                    hy ? __fmul_rn(w.B.y, s.y) : __fmaf_rn(d.y, dt, w.a.y),
                    hz ? __fmul_rn(w.B.z, s.z) : __fmaf_rn(d.z, dt, w.a.z));
  w.B.x = __fadd_rn(w.B.x, hx ? 1.f : 0.f);
  w.B.y = __fadd_rn(w.B.y, hy ? 1.f : 0.f);
  w.B.z = __fadd_rn(w.B.z, hz ? 1.f : 0.f);
  w.t = __fadd_rn(w.t, dt);
}

// 2^-22 of the extent, 2 ulp of any coordinate or more: a point that rounding
// carried to or past its plane is nearer (within half an ulp before it, or past
// it by the rounding of dt and of the point, at most one ulp).
__device__ __forceinline__ float near_plane(const float3 n) {
  return (fmaxf(n.x, fmaxf(n.y, n.z)) + 2.f) * 2.38418579e-7f;
}

// 32 steps of a lane's ray, written to row[1..32] (row[0]: where they start).
// The coordinates only move outwards, so a ray that left the box is outside
// at the chunk's end too: the walker looks there, the consumers find the step.
// Every lane of the warp takes part (planes are checked once per 8 steps and
// warp).
__device__ __forceinline__ void walk_chunk_fast(Walk& w, const float3 d, const float3 r, const float3 s, float near,
                                                float4* row) {
  row[0] = make_float4(w.a.x, w.a.y, w.a.z, w.t);
#pragma unroll 1
  for (int k0 = 1; k0 <= 32; k0 += 8) {
    const Walk w0 = w;
    float gap = near;
#pragma unroll
    for (int k = 0; k < 8; ++k) {
      walk_step<false>(w, d, r, s, gap);
      row[k0 + k] = make_float4(w.a.x, w.a.y, w.a.z, w.t);
    }
    if (__any_sync(0xffffffffu, gap < near)) {
      w = w0;
#pragma unroll 1
      for (int k = 0; k < 8; ++k) {
        walk_step<true>(w, d, r, s, gap);
        row[k0 + k] = make_float4(w.a.x, w.a.y, w.a.z, w.t);
      }
    }
  }
}

// The same for warps with a ray whose direction has a zero or extreme
// component (recip_ok): the plain step, until the first point outside.  The
// rest of the row repeats that point.
__device__ __forceinline__ void walk_chunk_any(Walk& w, const float3 d, const float3 r, const float3 s, bool fast,
                                               const float3 n, bool alive, float4* row) {
  row[0] = make_float4(w.a.x, w.a.y, w.a.z, w.t);
#pragma unroll 1
  for (int k = 1; k <= 32; ++k) {
    if (alive) {
      float3 q;
      float dt;
      if (fast)
        grid_step<true>(w.a, d, r, s, q, dt);
      else
        grid_step<false>(w.a, d, r, s, q, dt);
      w.t = __fadd_rn(w.t, dt);
      alive = !outside_closed3(q, n);
      w.a = q;
    }
    row[k] = make_float4(w.a.x, w.a.y, w.a.z, w.t);
  }
}

// Threads of a block: the walker, an idle warp 4 (warps 0, 4, 8, ... share a
// scheduler, and the walker's should be the least loaded) and NC consumers.
__host__ __device__ constexpr int walk_threads(int nc) { return 32 * (2 + nc); }

// MODE: WALK_COUNT counts (num, max_count, last_step); WALK_PADDED fills rows
// of max_n; WALK_SEGMENTS fills CSR ranges up to stop_step; WALK_SLOTS counts
// and fills fixed ranges.  NC consumer warps, each owning 32 / NC of the rays.
template <int MODE, int NC>
__global__ void __launch_bounds__(walk_threads(NC)) masked_walk_kernel(const WalkArgs a) {
  using R = WalkRing<NC>;
  constexpr int FULL = 1, EMPTY = 3, ALL = 32 * (1 + NC), OWN = 32 / NC;
  extern __shared__ __align__(16) uint8_t walk_smem[];
  R& ring = *reinterpret_cast<R*>(walk_smem);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int b = blockIdx.x * 32 + lane;
  if (warp == 0) {
    bool alive = false, fast = true;
    // a lane without a ray walks a harmless one
    float3 d = make_float3(1.f, 1.f, 1.f), p = make_float3(0.5f, 0.25f, 0.125f);
    float t = 0.f;
    if (b < a.batch) {
      const float3 v = load3(a.v, b);
      float3 o = ray_origin_voxel3(a.o, b, a.o3, a.voxel_size);
      float te;
      if (dir_ok(v) && box_entry3(o, v, a.n3, te)) {
        alive = true;
        fast = a.fast && recip_ok(v);
        d = v;
        p = o;
        t = te;
      }
    }
    const float3 s = signs(d);
    const float3 r = fast ? recip3(d) : d;
    Walk w{p, next_planes(p, s), t};
    const float near = near_plane(a.n3);
    const int step_cap = walk_cap(a.n3.x, a.n3.y, a.n3.z);
    const int limit =
        alive && MODE == WALK_SEGMENTS && a.stop_step ? min(a.stop_step[b], step_cap) : step_cap;
    alive = alive && limit > 0;
    const bool all_fast = __all_sync(0xffffffffu, fast);
    int steps = 0, c = 0;
    for (;; ++c) {
      const int slot = c & 1;
      if (c >= 2) ring_sync<EMPTY>(slot, ALL);
      float4* row = ring.pt[slot] + lane * R::ROW;
      const int allowed = alive ? min(32, limit - steps) : 0;  // steps that the consumers may look at
      if (all_fast)
        walk_chunk_fast(w, d, r, s, near, row);
      else
        walk_chunk_any(w, d, r, s, fast, a.n3, alive, row);
      steps += 32;
      alive = alive && !outside_closed3(w.a, a.n3);
      if (alive && steps >= limit) {
        if (limit == step_cap) note_cap_hit();
        alive = false;
      }
      ring.steps[slot][lane] = allowed;
      const bool more = __any_sync(0xffffffffu, alive);
      if (lane == 0) ring.more[slot] = more;
      __threadfence_block();
      ring_arrive<FULL>(slot, ALL);
      if (!more) break;
    }
    // the consumers' last releases
    if (c >= 1) ring_sync<EMPTY>((c - 1) & 1, ALL);
    ring_sync<EMPTY>(c & 1, ALL);
    return;
  }
  if (warp == 4) return;
  const int consumer = warp > 4 ? warp - 2 : warp - 1;
  const int first = consumer * OWN;  // this warp's rays: first .. first + OWN - 1, state in the lane of that number
  const bool own = lane >= first && lane < first + OWN && b < a.batch;
  int count = 0, last = 0;
  long long base = 0, cap = 0x7fffffff;
  if (own) {
    if (MODE == WALK_SEGMENTS) {
      base = a.offsets[b];
      cap = a.offsets[b + 1] - base;
    } else if (MODE == WALK_SLOTS) {
      base = (long long)b * a.slot;
      cap = a.slot;
    } else if (MODE == WALK_PADDED) {
      base = (long long)b * a.max_n;
      cap = a.max_n;
    }
  }
  const int room = (int)(cap < 0x7fffffff ? cap : 0x7fffffff);
  float2* out = ring.out[consumer];
  float* seg = MODE == WALK_PADDED ? a.inter : a.seg;
  float* seg_t = MODE == WALK_PADDED ? a.tns : a.seg_t;
  int* seg_ray = MODE == WALK_SEGMENTS ? a.seg_ray : nullptr;
  for (int c = 0;; ++c) {
    const int slot = c & 1;
    ring_sync<FULL>(slot, ALL);
    const int steps = ring.steps[slot][lane];
    const bool more = ring.more[slot] != 0;
    constexpr int U = OWN < 8 ? OWN : 8;  // rays whose occupancy loads are in flight together
#pragma unroll 1
    for (int i = first; i < first + OWN; i += U) {
      uint8_t occ[U];
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const int n = __shfl_sync(0xffffffffu, steps, i + u);
        occ[u] = 0;
        if (n == 0) continue;
        const float4* row = ring.pt[slot] + (i + u) * R::ROW + lane;
        const float4 p = row[0], q = row[1];
        const unsigned out = __ballot_sync(0xffffffffu, outside_closed3(make_float3(q.x, q.y, q.z), a.n3));
        if (lane < n && (out & (0xffffffffu >> (31 - lane))) == 0u) {  // no step up to this one left the box
          const long long idx =
              cell_index3(make_float3(p.x, p.y, p.z), make_float3(q.x, q.y, q.z), a.mask_scale, a.mx, a.my);
          if (idx >= 0 && idx < a.cells) occ[u] = __ldg(a.mask + idx);
        }
      }
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const unsigned m = __ballot_sync(0xffffffffu, occ[u] != 0);
        if (m == 0u) continue;
        const int got = __popc(m);
        if (MODE != WALK_COUNT) {
          const int have = __shfl_sync(0xffffffffu, count, i + u);
          const long long g = __shfl_sync(0xffffffffu, base, i + u) + have;
          const int n = min(got, __shfl_sync(0xffffffffu, room, i + u) - have);  // segments that fit
          const int rank = __popc(m & ((1u << lane) - 1u));
          __syncwarp();  // the previous ray's run has left `out`
          if (occ[u] != 0 && rank < n) {
            const float4* row = ring.pt[slot] + (i + u) * R::ROW + lane;
            const float4 p = row[0], q = row[1];
            out[3 * rank] = make_float2(p.x, p.y);
            out[3 * rank + 1] = make_float2(p.z, q.x);
            out[3 * rank + 2] = make_float2(q.y, q.z);
            if (seg_t) seg_t[g + rank] = __fmul_rn(q.w, a.voxel_size);
            if (seg_ray) seg_ray[g + rank] = blockIdx.x * 32 + i + u;
          }
          __syncwarp();
          if (MODE == WALK_PADDED) {
            for (int w = lane; w < 6 * n; w += 32) seg[6 * g + w] = reinterpret_cast<const float*>(out)[w];
          } else {
            for (int w = lane; w < 3 * n; w += 32) reinterpret_cast<float2*>(seg)[3 * g + w] = out[w];
          }
        }
        if (lane == i + u) {
          count += got;
          last = 32 * c + 32 - __clz(m);
        }
      }
    }
    __threadfence_block();
    ring_arrive<EMPTY>(slot, ALL);
    if (!more) break;
  }
  if (MODE != WALK_SEGMENTS) {
    if (own) a.num[b] = count;
    if (MODE == WALK_COUNT && own && a.last_step) a.last_step[b] = last;
    const int mx = __reduce_max_sync(0xffffffffu, own ? count : 0);
    if (a.max_count && lane == 0) atomicMax(a.max_count, mx);
  }
}

// Counts for large batches: a thread per ray, 8 steps at a time, their 8
// occupancy loads issued back to back.  With enough rays to fill the
// schedulers, total instructions set the time and the ring's hand-over only
// adds to them.
__global__ void __launch_bounds__(256) masked_count_kernel(const WalkArgs a) {
  constexpr int K = 8;
  const int b = blockIdx.x * blockDim.x + threadIdx.x;
  int count = 0, last = 0;
  if (b < a.batch) {
    const float3 d = load3(a.v, b);
    float3 p = ray_origin_voxel3(a.o, b, a.o3, a.voxel_size);
    float t;
    if (dir_ok(d) && box_entry3(p, d, a.n3, t)) {
      const bool fast = a.fast && recip_ok(d);
      const float3 s = signs(d), r = fast ? recip3(d) : d;
      const float near = near_plane(a.n3);
      const int step_cap = walk_cap(a.n3.x, a.n3.y, a.n3.z);
      Walk w{p, next_planes(p, s), t};
      for (int steps = 0;; steps += K) {
        float3 P[K + 1];
        unsigned out = 0;
        P[0] = w.a;
        const Walk w0 = w;
        float gap = near;
        if (fast) {
#pragma unroll
          for (int k = 0; k < K; ++k) {
            walk_step<false>(w, d, r, s, gap);
            P[k + 1] = w.a;
            out |= outside_closed3(w.a, a.n3) ? 1u << k : 0u;
          }
        }
        if (!fast || gap < near) {
          w = w0;
          out = 0;
#pragma unroll
          for (int k = 0; k < K; ++k) {
            if (out != 0) continue;
            float3 q;
            float dt;
            if (fast)
              grid_step<true>(w.a, d, r, s, q, dt);
            else
              grid_step<false>(w.a, d, r, s, q, dt);
            w.a = P[k + 1] = q;
            out |= outside_closed3(q, a.n3) ? 1u << k : 0u;
          }
          w.B = next_planes(w.a, s);
        }
        const int inside = min(out ? __ffs(out) - 1 : K, step_cap - steps);
        uint8_t occ[K];
        unsigned in_mask = 0;
#pragma unroll
        for (int k = 0; k < K; ++k) {
          const long long idx = cell_index3(P[k], P[k + 1], a.mask_scale, a.mx, a.my);
          const bool ok = k < inside && idx >= 0 && idx < a.cells;
          occ[k] = __ldg(a.mask + (ok ? idx : 0));
          in_mask |= ok ? 1u << k : 0u;
        }
        unsigned m = 0;
#pragma unroll
        for (int k = 0; k < K; ++k) m |= occ[k] != 0 ? 1u << k : 0u;
        m &= in_mask;
        count += __popc(m);
        if (m) last = steps + 32 - __clz(m);
        if (out) break;
        if (steps + K >= step_cap) {
          note_cap_hit();
          break;
        }
      }
    }
    a.num[b] = count;
    if (a.last_step) a.last_step[b] = last;
  }
  warp_max_atomic(a.max_count, count, b < a.batch);
}

// Slots -> CSR: row k of ray b moves from b * slot + k to offsets[b] + k.
__global__ void __launch_bounds__(256) compact_slots_kernel(int batch, long long slot, const int64_t* __restrict__ offsets,
                                                            const float* __restrict__ sseg,
                                                            const float* __restrict__ st, float* __restrict__ seg,
                                                            float* __restrict__ t, int* __restrict__ ray) {
  const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  const long long b = i / slot, k = i - b * slot;
  if (b >= batch) return;
  const long long beg = offsets[b];
  if (k >= offsets[b + 1] - beg) return;
  const long long src = i, dst = beg + k;
  const float2* s2 = reinterpret_cast<const float2*>(sseg + src * 6);
  float2* d2 = reinterpret_cast<float2*>(seg + dst * 6);
  d2[0] = s2[0];
  d2[1] = s2[1];
  d2[2] = s2[2];
  if (t) t[dst] = st[src];
  if (ray) ray[dst] = (int)b;
}

// Octree first hit.  Reference ray_march.cu:33-148, generalised from the
// N in {128, 256} templates to any N that is a multiple of 64.
template <bool FAST>
__device__ __forceinline__ void octree_descend(float* slot, uint8_t* finish, int b, float3 p, const float3 d,
                                               const uint8_t* __restrict__ oct, int N, long long oct_cells) {
  const float3 s = signs(d);
  const float3 r = FAST ? recip3(d) : d;
  int m = N / 64;
  long long off = 0;
  float3 last = p;
  // the levels walk fewer than 3 (N/64 + N/16 + N/4) + 9 <= N + 9 steps in all
  const int cap = walk_cap((float)N, 0.f, 0.f) + 6;
  int steps = 0;
  while (m < N) {
    if (steps++ == cap) {
      note_cap_hit();
      slot[0] = -1.f;
      finish[b] = 1;
      return;
    }
    last = p;
    float3 q;
    float dt;
    grid_step<FAST>(last, d, r, s, q, dt);
    if (outside_closed(q, (float)m)) {
      slot[0] = -1.f;
      finish[b] = 1;
      return;
    }
    const long long idx = off + cell_index1(last, q, m);
    if (occupied(oct, idx, oct_cells)) {
      off += (long long)m * m * m;
      last = make_float3(__fmul_rn(last.x, 4.f), __fmul_rn(last.y, 4.f), __fmul_rn(last.z, 4.f));
      p = last;
      m *= 4;
    } else {
      p = q;
    }
  }
  slot[0] = last.x;
  slot[1] = last.y;
  slot[2] = last.z;
}

__global__ void __launch_bounds__(256) aabb_kernel(int batch, float* __restrict__ coords,
                                                   const float* __restrict__ v,
                                                   const float* __restrict__ center,
                                                   uint8_t* __restrict__ finish,
                                                   float* __restrict__ rgba,
                                                   const uint8_t* __restrict__ oct, int N,
                                                   long long oct_cells) {
  const int b = blockIdx.x * blockDim.x + threadIdx.x;
  if (b >= batch) return;
  float* slot = coords + (long long)batch * 6 * 7 + (long long)b * 6 + 3;
  reinterpret_cast<float4*>(rgba)[b] = make_float4(0.f, 0.f, 0.f, 1.f);
  finish[b] = 0;
  const float3 d = load3(v, b);
  float3 p = make_float3(__ldg(center + 0), __ldg(center + 1), __ldg(center + 2));
  float t;
  if (!dir_ok(d) || !box_entry(p, d, (float)N, t)) {
    slot[0] = -1.f;
    finish[b] = 1;
    return;
  }
  p = make_float3(__fmul_rn(p.x, 0.015625f), __fmul_rn(p.y, 0.015625f), __fmul_rn(p.z, 0.015625f));
  if (N < (1 << 22) && recip_ok(d))
    octree_descend<true>(slot, finish, b, p, d, oct, N, oct_cells);
  else
    octree_descend<false>(slot, finish, b, p, d, oct, N, oct_cells);
}

// Next 8 occupied voxels of a ray, put(k, entry, exit) for each in order and
// put_end(k) where the ray leaves the grid before its k-th.  Reference
// ray_march.cu:159-229.  8 steps at a time: their occupancy loads are issued
// back to back (one at a time the walk waits for every byte), and the planes
// are kept from step to step (walk_step).
template <class Put, class End>
__device__ __forceinline__ void march8(const float3 last, const float3 d, bool fast, const uint8_t* __restrict__ mask,
                                       int N, Put put, End put_end) {
  constexpr int K = 8;
  const float3 s = signs(d);
  const float3 r = fast ? recip3(d) : d;
  const float n = (float)N;
  const long long cells = (long long)N * N * N;
  const int cap = walk_cap(n, n, n);
  const float near = near_plane(make_float3(n, n, n));
  int hits = 0;
  Walk w{last, next_planes(last, s), 0.f};
  for (int steps = 0;; steps += K) {
    float3 P[K + 1];
    unsigned out = 0;
    P[0] = w.a;
    const Walk w0 = w;
    float gap = near;
    if (fast) {
#pragma unroll
      for (int k = 0; k < K; ++k) {
        walk_step<false>(w, d, r, s, gap);
        P[k + 1] = w.a;
        out |= outside_open(w.a, n) ? 1u << k : 0u;
      }
    }
    if (!fast || gap < near) {
      w = w0;
      out = 0;
#pragma unroll
      for (int k = 0; k < K; ++k) {
        if (out != 0) continue;
        float3 q;
        float dt;
        if (fast)
          grid_step<true>(w.a, d, r, s, q, dt);
        else
          grid_step<false>(w.a, d, r, s, q, dt);
        w.a = P[k + 1] = q;
        out |= outside_open(q, n) ? 1u << k : 0u;
      }
      w.B = next_planes(w.a, s);
    }
    const int inside = min(out ? __ffs(out) - 1 : K, cap - steps);
    uint8_t occ[K];
    unsigned in_mask = 0;
#pragma unroll
    for (int k = 0; k < K; ++k) {
      const long long idx = cell_index1(P[k], P[k + 1], N);
      const bool ok = k < inside && idx >= 0 && idx < cells;
      occ[k] = __ldg(mask + (ok ? idx : 0));
      in_mask |= ok ? 1u << k : 0u;
    }
#pragma unroll
    for (int k = 0; k < K; ++k) {
      if (((in_mask >> k) & 1u) && occ[k] != 0 && hits < 8) {
        put(hits, P[k], P[k + 1]);
        ++hits;
      }
    }
    if (hits == 8) return;
    if (out != 0 || steps + K >= cap) {
      if (out == 0) note_cap_hit();
      put_end(hits);
      return;
    }
  }
}

// The reference leaves its grid-stride loop when an unfinished ray has no
// resume point (x < 0), a state that aabb_intersect + mlp_eval never produce;
// here such a ray is skipped on its own so the result does not depend on the
// launch shape.
__global__ void __launch_bounds__(256) march_kernel(int batch, float* __restrict__ coords,
                                                    const float* __restrict__ v,
                                                    const uint8_t* __restrict__ mask,
                                                    const uint8_t* __restrict__ finish, int N) {
  const int b = blockIdx.x * blockDim.x + threadIdx.x;
  if (b >= batch || finish[b]) return;
  const long long stride = (long long)batch * 6;
  const float* rs = coords + 7 * stride + (long long)b * 6 + 3;
  const float3 last = make_float3(rs[0], rs[1], rs[2]);
  coords[(long long)b * 6] = -1.f;
  if (last.x < 0.f) return;
  const float3 d = load3(v, b);
  if (!dir_ok(d)) return;  // a miss (aabb_intersect finished such a ray already)
  const float lim = (float)N;  // a resume point from outside the grid takes the __fdiv_rn form
  const bool fast = N < (1 << 22) && recip_ok(d) && fabsf(last.x) <= lim && fabsf(last.y) <= lim && fabsf(last.z) <= lim;
  march8(
      last, d, fast, mask, N,
      [&](int k, const float3 p, const float3 q) {
        float2* rr = reinterpret_cast<float2*>(coords + k * stride + (long long)b * 6);
        rr[0] = make_float2(p.x, p.y);
        rr[1] = make_float2(p.z, q.x);
        rr[2] = make_float2(q.y, q.z);
      },
      [&](int k) { coords[k * stride + (long long)b * 6] = -1.f; });
}

// ---- the same over the live pixels of a frame --------------------------------
//
// Most pixels of a frame finish in its first rounds, the last ones after
// dozens.  Each round works on a list of the pixels still alive, so that its
// tiles of pixels are full: begin makes the first list, the decoder
// (mlp_eval_tc_kernel) the next one.  Hits are stored by list position,
// resume points by pixel; what happens to a pixel does not depend on its
// position.

// Appends `pixel` of the lanes with `alive` to list (one atomic per warp; every lane takes part).
__device__ __forceinline__ void append_live(bool alive, int pixel, int* __restrict__ list, int* __restrict__ count) {
  const unsigned m = __ballot_sync(0xffffffffu, alive);
  if (m == 0u) return;
  const int lane = threadIdx.x & 31, leader = __ffs(m) - 1;
  int at = 0;
  if (lane == leader) at = atomicAdd(count, __popc(m));
  at = __shfl_sync(0xffffffffu, at, leader);
  if (alive) list[at + __popc(m & ((1u << lane) - 1u))] = pixel;
}

__global__ void __launch_bounds__(256) begin_kernel(int batch, const float* __restrict__ v,
                                                    const float* __restrict__ center, const uint8_t* __restrict__ oct,
                                                    int N, long long oct_cells, float* __restrict__ resume,
                                                    float* __restrict__ rgba, int* __restrict__ list,
                                                    int* __restrict__ count) {
  const int b = blockIdx.x * blockDim.x + threadIdx.x;
  uint8_t done = 1;
  if (b < batch) {
    done = 0;
    reinterpret_cast<float4*>(rgba)[b] = make_float4(0.f, 0.f, 0.f, 1.f);
    const float3 d = load3(v, b);
    float3 p = make_float3(__ldg(center + 0), __ldg(center + 1), __ldg(center + 2));
    float t;
    if (!dir_ok(d) || !box_entry(p, d, (float)N, t)) {
      done = 1;
    } else {
      p = make_float3(__fmul_rn(p.x, 0.015625f), __fmul_rn(p.y, 0.015625f), __fmul_rn(p.z, 0.015625f));
      float slot[3];
      if (N < (1 << 22) && recip_ok(d))
        octree_descend<true>(slot, &done, 0, p, d, oct, N, oct_cells);
      else
        octree_descend<false>(slot, &done, 0, p, d, oct, N, oct_cells);
      if (!done) {
        resume[3LL * b] = slot[0];
        resume[3LL * b + 1] = slot[1];
        resume[3LL * b + 2] = slot[2];
      }
    }
  }
  append_live(!done, b, list, count);
}

__global__ void __launch_bounds__(256) march_live_kernel(int capacity, const int* __restrict__ list,
                                                         const int* __restrict__ count, float* __restrict__ hits,
                                                         float* __restrict__ resume, const float* __restrict__ v,
                                                         const uint8_t* __restrict__ mask, int N) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= min(*count, capacity)) return;
  const int b = list[i];
  const long long stride = (long long)capacity * 6;
  const float3 last = make_float3(resume[3LL * b], resume[3LL * b + 1], resume[3LL * b + 2]);
  const float3 d = load3(v, b);
  const float lim = (float)N;
  const bool fast = N < (1 << 22) && recip_ok(d) && fabsf(last.x) <= lim && fabsf(last.y) <= lim && fabsf(last.z) <= lim;
  march8(
      last, d, fast, mask, N,
      [&](int k, const float3 p, const float3 q) {
        float2* rr = reinterpret_cast<float2*>(hits + k * stride + (long long)i * 6);
        rr[0] = make_float2(p.x, p.y);
        rr[1] = make_float2(p.z, q.x);
        rr[2] = make_float2(q.y, q.z);
        if (k == 7) {
          resume[3LL * b] = q.x;
          resume[3LL * b + 1] = q.y;
          resume[3LL * b + 2] = q.z;
        }
      },
      [&](int k) { hits[k * stride + (long long)i * 6] = -1.f; });
}

// Pinhole camera rays (utils/dataset/ray_utils.py:5-55): pixel (i, j) looks
// along ((i + 0.5 - W/2) / focal, -(j + 0.5 - H/2) / focal, -1), rotated by
// the camera-to-world matrix and normalised; the origin is its translation.
struct Camera {
  float r[9];  // rotation, row-major (world = R * camera)
  float t[3];
  float focal;
  int H, W;
  long long first, count;  // pixel range [first, first + count) of the H x W image
};

__global__ void __launch_bounds__(256) camera_rays_kernel(const Camera c, float* __restrict__ o, float* __restrict__ d) {
  const long long p = (long long)blockIdx.x * blockDim.x + threadIdx.x;  // output row
  if (p >= c.count) return;
  const long long px = c.first + p;
  const int j = (int)(px / c.W), i = (int)(px - (long long)j * c.W);
  const float x = __fdiv_rn(__fsub_rn((float)i + 0.5f, 0.5f * (float)c.W), c.focal);
  const float y = -__fdiv_rn(__fsub_rn((float)j + 0.5f, 0.5f * (float)c.H), c.focal);
  float w[3];
#pragma unroll
  for (int k = 0; k < 3; ++k) w[k] = fmaf(c.r[3 * k], x, fmaf(c.r[3 * k + 1], y, -c.r[3 * k + 2]));
  const float n = sqrtf(fmaf(w[0], w[0], fmaf(w[1], w[1], w[2] * w[2])));
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    d[3 * p + k] = __fdiv_rn(w[k], n);
    o[3 * p + k] = c.t[k];
  }
}

__global__ void pair_counts_kernel(int batch, const int* __restrict__ num, int* __restrict__ out) {
  const int b = blockIdx.x * blockDim.x + threadIdx.x;
  if (b < batch) out[b] = max(num[b] - 1, 0);
}

// ---- exclusive scan: int32 counts -> int64 offsets --------------------------

__device__ __forceinline__ long long block_exclusive_scan(long long x, long long* smem, long long* total) {
  // warp inclusive scan, then scan of warp totals
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  long long incl = x;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const long long y = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane >= o) incl += y;
  }
  if (lane == 31) smem[warp] = incl;
  __syncthreads();
  if (warp == 0) {
    long long w = lane < (SCAN_THREADS / 32) ? smem[lane] : 0;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const long long y = __shfl_up_sync(0xffffffffu, w, o);
      if (lane >= o) w += y;
    }
    if (lane < SCAN_THREADS / 32) smem[lane] = w;  // inclusive warp-total prefix
  }
  __syncthreads();
  const long long warp_prefix = warp > 0 ? smem[warp - 1] : 0;
  *total = smem[SCAN_THREADS / 32 - 1];
  __syncthreads();
  return warp_prefix + incl - x;
}

__global__ void __launch_bounds__(SCAN_THREADS) scan_tile_sums(const int* __restrict__ in, long long n,
                                                               long long* __restrict__ tile_sum) {
  __shared__ long long smem[32];
  const long long base = (long long)blockIdx.x * SCAN_TILE + threadIdx.x * SCAN_ITEMS;
  long long s = 0;
#pragma unroll
  for (int i = 0; i < SCAN_ITEMS; ++i)
    if (base + i < n) s += in[base + i];
  long long total;
  block_exclusive_scan(s, smem, &total);
  if (threadIdx.x == 0) tile_sum[blockIdx.x] = total;
}

// Single block: exclusive scan of the tile sums in place.
__global__ void __launch_bounds__(SCAN_THREADS) scan_tile_prefix(long long* __restrict__ tile_sum, long long tiles) {
  __shared__ long long smem[32];
  long long carry = 0;
  for (long long start = 0; start < tiles; start += SCAN_THREADS) {
    const long long i = start + threadIdx.x;
    const long long x = i < tiles ? tile_sum[i] : 0;
    long long total;
    const long long ex = block_exclusive_scan(x, smem, &total);
    if (i < tiles) tile_sum[i] = carry + ex;
    carry += total;
  }
}

__global__ void __launch_bounds__(SCAN_THREADS) scan_tiles(const int* __restrict__ in, long long n,
                                                           const long long* __restrict__ tile_prefix,
                                                           int64_t* __restrict__ out) {
  __shared__ long long smem[32];
  const long long base = (long long)blockIdx.x * SCAN_TILE + threadIdx.x * SCAN_ITEMS;
  int vals[SCAN_ITEMS];
  long long s = 0;
#pragma unroll
  for (int i = 0; i < SCAN_ITEMS; ++i) {
    vals[i] = base + i < n ? in[base + i] : 0;
    s += vals[i];
  }
  long long total;
  long long run = tile_prefix[blockIdx.x] + block_exclusive_scan(s, smem, &total);
#pragma unroll
  for (int i = 0; i < SCAN_ITEMS; ++i) {
    if (base + i < n) out[base + i] = run;
    run += vals[i];
  }
  if (base < n && base + SCAN_ITEMS >= n) out[n] = run;  // thread owning the last element
}

// ---- offsets, total and largest count in one go -----------------------------

__device__ __forceinline__ long long warp_max64(long long v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v = max(v, __shfl_xor_sync(0xffffffffu, v, o));
  return v;
}

// Up to SMALL_SCAN counts in one block: SMALL_SCAN / 1024 consecutive ones per
// thread.  totals = (sum, largest count).
constexpr int SMALL_SCAN = 16384;

__global__ void __launch_bounds__(1024) small_offsets_kernel(const int* __restrict__ in, int n, int64_t* __restrict__ out,
                                                             long long* __restrict__ totals) {
  __shared__ long long sums[32], maxs[32];
  constexpr int PER = SMALL_SCAN / 1024;
  const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
  const int per = (n + 1023) / 1024;  // <= PER, spread over all threads
  int v[PER];
  long long s = 0, m = 0;
#pragma unroll
  for (int i = 0; i < PER; ++i) {
    v[i] = i < per && t * per + i < n ? in[t * per + i] : 0;
    s += v[i];
    m = max(m, (long long)v[i]);
  }
  long long incl = s;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const long long y = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane >= o) incl += y;
  }
  m = warp_max64(m);
  if (lane == 31) {
    sums[warp] = incl;
    maxs[warp] = m;
  }
  __syncthreads();
  if (warp == 0) {
    long long w = sums[lane];
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const long long y = __shfl_up_sync(0xffffffffu, w, o);
      if (lane >= o) w += y;
    }
    sums[lane] = w;
    const long long mm = warp_max64(maxs[lane]);
    if (lane == 31) {
      totals[0] = w;
      totals[1] = mm;
      out[n] = w;
    }
  }
  __syncthreads();
  long long run = (warp ? sums[warp - 1] : 0) + incl - s;
#pragma unroll
  for (int i = 0; i < PER; ++i)
    if (i < per && t * per + i < n) {
      out[t * per + i] = run;
      run += v[i];
    }
}

// Larger n: the tiles' sums as in scan_tile_sums, and their largest counts.
__global__ void __launch_bounds__(SCAN_THREADS) tile_max_kernel(const int* __restrict__ in, long long n,
                                                                long long* __restrict__ tile_max) {
  __shared__ long long maxs[SCAN_THREADS / 32];
  const long long base = (long long)blockIdx.x * SCAN_TILE + threadIdx.x;
  long long m = 0;
#pragma unroll
  for (int i = 0; i < SCAN_ITEMS; ++i)
    if (base + i * SCAN_THREADS < n) m = max(m, (long long)in[base + i * SCAN_THREADS]);
  m = warp_max64(m);
  if ((threadIdx.x & 31) == 0) maxs[threadIdx.x >> 5] = m;
  __syncthreads();
  if (threadIdx.x == 0) {
#pragma unroll
    for (int w = 1; w < SCAN_THREADS / 32; ++w) m = max(m, maxs[w]);
    tile_max[blockIdx.x] = m;
  }
}

__global__ void __launch_bounds__(1024) totals_kernel(const long long* __restrict__ tile_max, long long tiles,
                                                      const int64_t* __restrict__ end, long long* __restrict__ totals) {
  __shared__ long long maxs[32];
  long long m = 0;
  for (long long i = threadIdx.x; i < tiles; i += 1024) m = max(m, tile_max[i]);
  m = warp_max64(m);
  if ((threadIdx.x & 31) == 0) maxs[threadIdx.x >> 5] = m;
  __syncthreads();
  if (threadIdx.x < 32) {
    m = warp_max64(maxs[threadIdx.x]);
    if (threadIdx.x == 0) {
      totals[0] = *end;
      totals[1] = m;
    }
  }
}

}  // namespace dv

using namespace dv;

long long realtime_walk_cap_hits(int reset);  // realtime.cu

// int(voxel_num * mask_scale) with the product rounded to float first, as the
// reference computes it on the device (ray_voxel_intersect.cu:268).
static int cells_per_side(float n, float scale) {
  volatile float prod = n * scale;
  return (int)prod;
}

static int sm_count() {
  static int sms = 0;
  if (sms == 0) {
    int dev = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    if (sms <= 0) sms = 1;
  }
  return sms;
}

// Launches a masked walk.  Up to two blocks per SM, 16 consumer warps (2 rays
// each): the hand-over is latency, and only the walker should set the time;
// beyond that 8, as blocks share the SM.  Measured, 16 / 8 consumers: a
// 4096-ray batch into slots 54 / 85 us (4 consumers 165, a thread per ray
// 251), 65,792 rays' segments 78 / 75 us (4: 99, 2: 150), 640,000 rays'
// 1442 / 1224 us (a thread per ray with staged stores 2075).  A count has
// less to hand over: from 768 rays per SM on, a thread per ray is faster
// (65,792 rays: 91 us here, 105 there; 640,000 rays: 997 and 697 us).
template <int MODE>
static int masked_walk_launch(const WalkArgs& a, void* stream) {
  const long long blocks = ceil_div(a.batch, 32);
  const cudaStream_t st = (cudaStream_t)stream;
  const int sms = sm_count();
  if (MODE == WALK_COUNT && a.batch >= 768LL * sms)
    masked_count_kernel<<<ceil_div(a.batch, 256), 256, 0, st>>>(a);
  else if (blocks <= 2LL * sms)
    masked_walk_kernel<MODE, 16><<<(unsigned)blocks, walk_threads(16), sizeof(WalkRing<16>), st>>>(a);
  else
    masked_walk_kernel<MODE, 8><<<(unsigned)blocks, walk_threads(8), sizeof(WalkRing<8>), st>>>(a);
  DV_TRY_LAUNCH();
  return DV_OK;
}

// Threads per block of a dense walk launch.  One thread walks one ray and the
// walk is a long dependent chain, so a small batch runs faster spread thinly:
// with fewer rays than 8 warps per SM, blocks of one warp put each warp on its
// own SM instead of several warps sharing a scheduler.
static int walk_block(int batch) { return batch < sm_count() * 256 ? 32 : 256; }

#define DV_WALK_LAUNCH(kernel, batch, stream, args)                              \
  do {                                                                             \
    const int bs__ = walk_block(batch);                                            \
    kernel<<<ceil_div((batch), bs__), bs__, 0, (cudaStream_t)(stream)>>>(args);   \
  } while (0)

static bool aligned_to(const void* p, uintptr_t n) { return ((uintptr_t)p % n) == 0; }

// What the segment lists' entry points take.  The walks need 8 bytes for seg
// (8-byte stores) and 4 for the others; the entry points have asked for more
// (masked lists: seg on 16 bytes; seg_t and seg_ray on 8) since their earlier
// writers' vector stores, and go on refusing what they refused.
static bool segment_buffers_aligned(const float* seg, const float* seg_t, const int* seg_ray, uintptr_t seg_align) {
  return aligned_to(seg, seg_align) && aligned_to(seg_t, 8) && aligned_to(seg_ray, 8);
}

static WalkArgs walk_args(int batch, float xyzmin, float n, float vs, float mask_scale,
                          const float* o, const float* v, const uint8_t* mask) {
  WalkArgs a{};
  a.batch = batch;
  a.xyzmin = xyzmin;
  a.n = n;
  a.o3 = make_float3(xyzmin, xyzmin, xyzmin);
  a.n3 = make_float3(n, n, n);
  a.voxel_size = vs;
  a.mask_scale = mask_scale;
  a.m = cells_per_side(n, mask_scale);
  a.mx = a.my = a.m;
  a.cells = (long long)a.m * a.m * a.m;
  a.fast = n < 4194304.f;
  a.o = o;
  a.v = v;
  a.mask = mask;
  return a;
}

extern "C" {

int dv_ray_voxel_intersect(int batch_size, int max_n, float xyzmin, float xyzmax, float voxel_num,
                           float voxel_size, const float* o, const float* v, float* intersection,
                           int* intersect_num, float* tns, int* max_count, void* stream) {
  (void)xyzmax;  // unused by the reference kernel as well
  DV_CHECK(batch_size >= 0 && max_n >= 0, DV_ERR_ARG);
  if (batch_size == 0) return DV_OK;
  DV_CHECK(o && v && intersect_num && (max_n == 0 || (intersection && tns)), DV_ERR_ARG);
  WalkArgs a = walk_args(batch_size, xyzmin, voxel_num, voxel_size, 1.f, o, v, nullptr);
  a.max_n = max_n;
  a.inter = intersection;
  a.num = intersect_num;
  a.tns = tns;
  a.max_count = max_count;
  DV_WALK_LAUNCH(dense_walk_kernel<WALK_PADDED>, batch_size, stream, a);
  DV_TRY_LAUNCH();
  return DV_OK;
}

int dv_ray_voxel_count(int batch_size, float xyzmin, float voxel_num, float voxel_size,
                       const float* o, const float* v, int* intersect_num, int* max_count,
                       void* stream) {
  DV_CHECK(batch_size >= 0, DV_ERR_ARG);
  if (batch_size == 0) return DV_OK;
  DV_CHECK(o && v && intersect_num, DV_ERR_ARG);
  WalkArgs a = walk_args(batch_size, xyzmin, voxel_num, voxel_size, 1.f, o, v, nullptr);
  a.num = intersect_num;
  a.max_count = max_count;
  DV_WALK_LAUNCH(dense_walk_kernel<WALK_COUNT>, batch_size, stream, a);
  DV_TRY_LAUNCH();
  return DV_OK;
}

int dv_masked_intersect(int batch_size, int max_n, float xyzmin, float xyzmax, float voxel_num,
                        float voxel_size, float mask_scale, const float* o, const float* v,
                        const uint8_t* mask, float* intersection, int* intersect_num, float* tns,
                        int* max_count, void* stream) {
  (void)xyzmax;
  DV_CHECK(batch_size >= 0 && max_n >= 0, DV_ERR_ARG);
  if (batch_size == 0) return DV_OK;
  DV_CHECK(o && v && mask && intersect_num && (max_n == 0 || (intersection && tns)), DV_ERR_ARG);
  WalkArgs a = walk_args(batch_size, xyzmin, voxel_num, voxel_size, mask_scale, o, v, mask);
  a.max_n = max_n;
  a.inter = intersection;
  a.num = intersect_num;
  a.tns = tns;
  a.max_count = max_count;
  return masked_walk_launch<WALK_PADDED>(a, stream);
}

int dv_masked_count(int batch_size, float xyzmin, float voxel_num, float voxel_size,
                    float mask_scale, const float* o, const float* v, const uint8_t* mask,
                    int* intersect_num, int* max_count, int* last_step, void* stream) {
  DV_CHECK(batch_size >= 0, DV_ERR_ARG);
  if (batch_size == 0) return DV_OK;
  DV_CHECK(o && v && mask && intersect_num, DV_ERR_ARG);
  WalkArgs a = walk_args(batch_size, xyzmin, voxel_num, voxel_size, mask_scale, o, v, mask);
  a.num = intersect_num;
  a.max_count = max_count;
  a.last_step = last_step;
  return masked_walk_launch<WALK_COUNT>(a, stream);
}

int dv_masked_segments(int batch_size, float xyzmin, float voxel_num, float voxel_size,
                       float mask_scale, const float* o, const float* v, const uint8_t* mask,
                       const int64_t* offsets, float* seg, float* seg_t, int* seg_ray,
                       const int* stop_step, void* stream) {
  DV_CHECK(batch_size >= 0, DV_ERR_ARG);
  if (batch_size == 0) return DV_OK;
  DV_CHECK(o && v && mask && offsets && seg, DV_ERR_ARG);
  DV_CHECK(segment_buffers_aligned(seg, seg_t, seg_ray, 16), DV_ERR_ARG);
  WalkArgs a = walk_args(batch_size, xyzmin, voxel_num, voxel_size, mask_scale, o, v, mask);
  a.offsets = offsets;
  a.seg = seg;
  a.seg_t = seg_t;
  a.seg_ray = seg_ray;
  a.stop_step = stop_step;
  return masked_walk_launch<WALK_SEGMENTS>(a, stream);
}

int dv_masked_segments_slots(int batch_size, float xyzmin, float voxel_num, float voxel_size, float mask_scale,
                             const float* o, const float* v, const uint8_t* mask, long long slot, float* seg_slots,
                             float* t_slots, int* intersect_num, int* max_count, void* stream) {
  DV_CHECK(batch_size >= 0, DV_ERR_ARG);
  if (batch_size == 0) return DV_OK;
  DV_CHECK(o && v && mask && seg_slots && t_slots && intersect_num, DV_ERR_ARG);
  DV_CHECK(slot >= (long long)(3.0f * voxel_num) + 3, DV_ERR_ARG);  // no ray crosses more planes
  DV_CHECK(segment_buffers_aligned(seg_slots, t_slots, nullptr, 16), DV_ERR_ARG);
  WalkArgs a = walk_args(batch_size, xyzmin, voxel_num, voxel_size, mask_scale, o, v, mask);
  a.slot = slot;
  a.seg = seg_slots;
  a.seg_t = t_slots;
  a.num = intersect_num;
  a.max_count = max_count;
  return masked_walk_launch<WALK_SLOTS>(a, stream);
}

int dv_compact_slots(int batch_size, long long slot, const int64_t* offsets, const float* seg_slots,
                     const float* t_slots, float* seg, float* seg_t, int* seg_ray, void* stream) {
  DV_CHECK(batch_size >= 0 && slot > 0, DV_ERR_ARG);
  if (batch_size == 0) return DV_OK;
  DV_CHECK(offsets && seg_slots && t_slots && seg, DV_ERR_ARG);
  DV_CHECK(aligned_to(seg_slots, 8) && aligned_to(seg, 8), DV_ERR_ARG);
  compact_slots_kernel<<<ceil_div((long long)batch_size * slot, 256), 256, 0, (cudaStream_t)stream>>>(
      batch_size, slot, offsets, seg_slots, t_slots, seg, seg_t, seg_ray);
  DV_TRY_LAUNCH();
  return DV_OK;
}

int dv_dense_segments(int batch_size, float xyzmin, float voxel_num, float voxel_size,
                      const float* o, const float* v, const int64_t* offsets, float* seg,
                      float* seg_t, int* seg_ray, void* stream) {
  DV_CHECK(batch_size >= 0, DV_ERR_ARG);
  if (batch_size == 0) return DV_OK;
  DV_CHECK(o && v && offsets && seg, DV_ERR_ARG);
  DV_CHECK(segment_buffers_aligned(seg, seg_t, seg_ray, 8), DV_ERR_ARG);
  WalkArgs a = walk_args(batch_size, xyzmin, voxel_num, voxel_size, 1.f, o, v, nullptr);
  a.offsets = offsets;
  a.seg = seg;
  a.seg_t = seg_t;
  a.seg_ray = seg_ray;
  DV_WALK_LAUNCH(dense_walk_kernel<WALK_SEGMENTS>, batch_size, stream, a);
  DV_TRY_LAUNCH();
  return DV_OK;
}

int dv_dense_pair_counts(int batch_size, const int* intersect_num, int* seg_count, void* stream) {
  DV_CHECK(batch_size >= 0, DV_ERR_ARG);
  if (batch_size == 0) return DV_OK;
  DV_CHECK(intersect_num && seg_count, DV_ERR_ARG);
  pair_counts_kernel<<<ceil_div(batch_size, 256), 256, 0, (cudaStream_t)stream>>>(batch_size, intersect_num, seg_count);
  DV_TRY_LAUNCH();
  return DV_OK;
}

// Per-axis grids: origin xyzmin[3] (world), extents dims[3] = (nx, ny, nz)
// voxels, occupancy [nz][ny][nx] bytes (mask scale 1).
static WalkArgs walk_args_grid(int batch, const float* xyzmin, const int* dims, float vs, const float* o,
                               const float* v, const uint8_t* mask) {
  WalkArgs a{};
  a.batch = batch;
  a.o3 = make_float3(xyzmin[0], xyzmin[1], xyzmin[2]);
  a.n3 = make_float3((float)dims[0], (float)dims[1], (float)dims[2]);
  a.voxel_size = vs;
  a.mask_scale = 1.f;
  a.mx = dims[0];
  a.my = dims[1];
  a.cells = (long long)dims[0] * dims[1] * dims[2];
  a.fast = dims[0] < (1 << 22) && dims[1] < (1 << 22) && dims[2] < (1 << 22);
  a.o = o;
  a.v = v;
  a.mask = mask;
  return a;
}

int dv_camera_rays(int H, int W, float focal, const float* c2w, long long first_pixel, long long n_pixels,
                   float* rays_o, float* rays_d, void* stream) {
  DV_CHECK(H >= 0 && W >= 0 && c2w && first_pixel >= 0 && n_pixels >= 0, DV_ERR_ARG);
  DV_CHECK(first_pixel + n_pixels <= (long long)H * W, DV_ERR_ARG);
  if (n_pixels == 0) return DV_OK;
  DV_CHECK(rays_o && rays_d, DV_ERR_ARG);
  Camera c{};
  for (int k = 0; k < 3; ++k) {
    for (int l = 0; l < 3; ++l) c.r[3 * k + l] = c2w[4 * k + l];
    c.t[k] = c2w[4 * k + 3];
  }
  c.focal = focal;
  c.H = H;
  c.W = W;
  c.first = first_pixel;
  c.count = n_pixels;
  camera_rays_kernel<<<ceil_div(n_pixels, 256), 256, 0, (cudaStream_t)stream>>>(c, rays_o, rays_d);
  DV_TRY_LAUNCH();
  return DV_OK;
}

int dv_masked_count_grid(int batch_size, const float* xyzmin, const int* dims, float voxel_size, const float* o,
                         const float* v, const uint8_t* mask, int* intersect_num, int* max_count, int* last_step,
                         void* stream) {
  DV_CHECK(batch_size >= 0 && xyzmin && dims && dims[0] > 0 && dims[1] > 0 && dims[2] > 0, DV_ERR_ARG);
  if (batch_size == 0) return DV_OK;
  DV_CHECK(o && v && mask && intersect_num, DV_ERR_ARG);
  WalkArgs a = walk_args_grid(batch_size, xyzmin, dims, voxel_size, o, v, mask);
  a.num = intersect_num;
  a.max_count = max_count;
  a.last_step = last_step;
  return masked_walk_launch<WALK_COUNT>(a, stream);
}

int dv_masked_segments_grid(int batch_size, const float* xyzmin, const int* dims, float voxel_size, const float* o,
                            const float* v, const uint8_t* mask, const int64_t* offsets, float* seg, float* seg_t,
                            int* seg_ray, const int* stop_step, void* stream) {
  DV_CHECK(batch_size >= 0 && xyzmin && dims && dims[0] > 0 && dims[1] > 0 && dims[2] > 0, DV_ERR_ARG);
  if (batch_size == 0) return DV_OK;
  DV_CHECK(o && v && mask && offsets && seg, DV_ERR_ARG);
  DV_CHECK(segment_buffers_aligned(seg, seg_t, seg_ray, 16), DV_ERR_ARG);
  WalkArgs a = walk_args_grid(batch_size, xyzmin, dims, voxel_size, o, v, mask);
  a.offsets = offsets;
  a.seg = seg;
  a.seg_t = seg_t;
  a.seg_ray = seg_ray;
  a.stop_step = stop_step;
  return masked_walk_launch<WALK_SEGMENTS>(a, stream);
}

long long dv_walk_cap_hits(int reset) {
  unsigned long long v = 0, w = 0;
  if (cudaMemcpyFromSymbol(&v, g_walk_cap_hits, sizeof(v)) != cudaSuccess) return -1;
  const long long rt = realtime_walk_cap_hits(reset);
  if (rt < 0) return -1;
  if (reset && cudaMemcpyToSymbol(g_walk_cap_hits, &w, sizeof(w)) != cudaSuccess) return -1;
  return (long long)v + rt;
}

long long dv_scan_scratch_bytes(long long n) {
  const long long tiles = n > 0 ? (n + SCAN_TILE - 1) / SCAN_TILE : 1;
  return tiles * (long long)sizeof(long long);
}

int dv_exclusive_scan(const int* counts, long long n, int64_t* offsets, void* scratch, void* stream) {
  DV_CHECK(n >= 0 && offsets, DV_ERR_ARG);
  cudaStream_t st = (cudaStream_t)stream;
  if (n == 0) {
    if (cudaMemsetAsync(offsets, 0, sizeof(int64_t), st) != cudaSuccess) return DV_ERR_CUDA;
    return DV_OK;
  }
  DV_CHECK(counts && scratch, DV_ERR_ARG);
  const long long tiles = (n + SCAN_TILE - 1) / SCAN_TILE;
  DV_CHECK(tiles < (1LL << 31), DV_ERR_ARG);
  long long* tile_sum = (long long*)scratch;
  scan_tile_sums<<<(unsigned)tiles, SCAN_THREADS, 0, st>>>(counts, n, tile_sum);
  scan_tile_prefix<<<1, SCAN_THREADS, 0, st>>>(tile_sum, tiles);
  scan_tiles<<<(unsigned)tiles, SCAN_THREADS, 0, st>>>(counts, n, tile_sum, offsets);
  DV_TRY_LAUNCH();
  return DV_OK;
}

long long dv_segment_offsets_scratch_bytes(long long n) {
  return n <= SMALL_SCAN ? 0 : 2 * dv_scan_scratch_bytes(n);
}

int dv_segment_offsets(const int* counts, long long n, int64_t* offsets, int64_t* totals, void* scratch, void* stream) {
  DV_CHECK(n >= 0 && offsets && totals, DV_ERR_ARG);
  cudaStream_t st = (cudaStream_t)stream;
  if (n == 0) {
    if (cudaMemsetAsync(offsets, 0, sizeof(int64_t), st) != cudaSuccess) return DV_ERR_CUDA;
    if (cudaMemsetAsync(totals, 0, 2 * sizeof(int64_t), st) != cudaSuccess) return DV_ERR_CUDA;
    return DV_OK;
  }
  DV_CHECK(counts && (scratch || n <= SMALL_SCAN), DV_ERR_ARG);
  long long* tot = reinterpret_cast<long long*>(totals);
  if (n <= SMALL_SCAN) {
    small_offsets_kernel<<<1, 1024, 0, st>>>(counts, (int)n, offsets, tot);
    DV_TRY_LAUNCH();
    return DV_OK;
  }
  const int rc = dv_exclusive_scan(counts, n, offsets, scratch, stream);
  if (rc != DV_OK) return rc;
  const long long tiles = (n + SCAN_TILE - 1) / SCAN_TILE;
  long long* tile_max = (long long*)scratch + tiles;
  tile_max_kernel<<<(unsigned)tiles, SCAN_THREADS, 0, st>>>(counts, n, tile_max);
  totals_kernel<<<1, 1024, 0, st>>>(tile_max, tiles, offsets + n, tot);
  DV_TRY_LAUNCH();
  return DV_OK;
}

int dv_aabb_intersect(int batch_size, float* coords, const float* v, const float* center,
                      uint8_t* finish, float* rgba, const uint8_t* octrees, int voxel_num,
                      void* stream) {
  DV_CHECK(batch_size >= 0 && voxel_num >= 64 && voxel_num % 64 == 0, DV_ERR_ARG);
  if (batch_size == 0) return DV_OK;
  DV_CHECK(coords && v && center && finish && rgba && octrees, DV_ERR_ARG);
  DV_CHECK(((uintptr_t)rgba & 15) == 0, DV_ERR_ARG);
  const long long a = voxel_num / 64, b = voxel_num / 16, c = voxel_num / 4;
  const long long cells = a * a * a + b * b * b + c * c * c;
  aabb_kernel<<<ceil_div(batch_size, 256), 256, 0, (cudaStream_t)stream>>>(
      batch_size, coords, v, center, finish, rgba, octrees, voxel_num, cells);
  DV_TRY_LAUNCH();
  return DV_OK;
}

int dv_realtime_begin(int batch_size, const float* v, const float* center, const uint8_t* octrees, int voxel_num,
                      float* resume, float* rgba, int* list, int* count, void* stream) {
  DV_CHECK(batch_size >= 0 && voxel_num >= 64 && voxel_num % 64 == 0, DV_ERR_ARG);
  if (batch_size == 0) return DV_OK;
  DV_CHECK(v && center && octrees && resume && rgba && list && count && ((uintptr_t)rgba & 15) == 0, DV_ERR_ARG);
  const long long a = voxel_num / 64, b = voxel_num / 16, c = voxel_num / 4;
  begin_kernel<<<ceil_div(batch_size, 256), 256, 0, (cudaStream_t)stream>>>(
      batch_size, v, center, octrees, voxel_num, a * a * a + b * b * b + c * c * c, resume, rgba, list, count);
  DV_TRY_LAUNCH();
  return DV_OK;
}

int dv_march_live(int capacity, const int* list, const int* count, float* hits, float* resume, const float* v,
                  const uint8_t* mask, int voxel_num, void* stream) {
  DV_CHECK(capacity >= 0 && voxel_num > 0, DV_ERR_ARG);
  if (capacity == 0) return DV_OK;
  DV_CHECK(list && count && hits && resume && v && mask && aligned_to(hits, 8), DV_ERR_ARG);
  march_live_kernel<<<ceil_div(capacity, 256), 256, 0, (cudaStream_t)stream>>>(capacity, list, count, hits, resume, v,
                                                                              mask, voxel_num);
  DV_TRY_LAUNCH();
  return DV_OK;
}

int dv_ray_march(int batch_size, float* coords, const float* v, const uint8_t* mask,
                 const uint8_t* finish, int voxel_num, void* stream) {
  DV_CHECK(batch_size >= 0 && voxel_num > 0, DV_ERR_ARG);
  if (batch_size == 0) return DV_OK;
  DV_CHECK(coords && v && mask && finish, DV_ERR_ARG);
  DV_CHECK(aligned_to(coords, 8), DV_ERR_ARG);
  march_kernel<<<ceil_div(batch_size, 256), 256, 0, (cudaStream_t)stream>>>(batch_size, coords, v, mask,
                                                                           finish, voxel_num);
  DV_TRY_LAUNCH();
  return DV_OK;
}

}  // extern "C"
