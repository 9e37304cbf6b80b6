// Time loops on chip.
//
// One cooperative launch runs all steps of a time loop (or a long chunk of
// them) with the wavefield held on chip: a group of G CTAs owns one shot, CTA
// b the grid columns [b C, b C + C) over all rows.  A compute warp owns 128 rows
// of some of them (the CTA's columns are split over column groups of warps), a
// lane four adjacent rows: px, pz and kappa are in tensor memory, used as a
// scratchpad that a warp reads and writes by column, vx and vz in shared memory.
// What one step moves is then the history stream and three halo columns per CTA
// and half step, not the state.
//
// Halo columns go from lane to lane of neighbouring CTAs through L2: the
// writer stores (value, step tag) as one 64-bit word, so the reader's poll of
// the data is also the wait and no fence or flag follows it.  Writer and reader use
// relaxed accesses of gpu scope, whose 64-bit words are whole, and nothing else reads
// the words.  A lane needs its
// neighbour CTA's values of its own rows only, and only for the first two and
// the last column; those columns are computed last in a half step, so the
// words travel while the columns between are computed.  Buffers alternate by
// step parity: a CTA writes parity s only after it has read its neighbours'
// words of step s - 1, which they store after their last read of step s - 2.
// Rows couple neighbouring warps (vz through shared memory, p through warp
// shuffles and an edge array), ordered by the CTA barrier after each half step.
//
// Stage A stores its FP16 histories with one scale per step and field, taken
// from the maximum over the whole grid.  An extra warp per CTA exchanges the
// CTAs' maxima through tagged words during the half step after a field is
// complete, and the history of step s is stored from the tensor and shared
// memory in step s + 1, just before the values are updated (the last step's
// after the loop).
//
// Rows 0, 1 and the last rows and columns are never updated and the caller
// keeps sources away from them, so they stay zero: their update coefficients
// are set to zero instead of branching.  The same holds for px and pz above the
// free surface, where the pressure is zeroed.  (Once a value is not finite, zero times
// it is not zero, and these points hold NaN.  The wavefield output has zeros there all
// the same and the gathers leave them out; points that are updated get the same values
// as with zeros there.)
//
// Arithmetic: the reference's separately rounded FP32 operations, two rows at
// a time in packed (f32x2) instructions; bit-identical to the other kernels.
//
// Every wait is bounded: after its limit it raises kErrTimeout, and the other
// waits of the grid see the flag and stop waiting too.
//
// What bounds it: for wide CTAs instruction issue and the latency between
// dependent instructions (16 warps an SM is what 128 registers allow; about 150
// instructions per lane quad and half step, 46 of them arithmetic), for narrow
// ones the exchange latency (about 0.5 us per half step).  Tried and slower: the fields in
// registers with all columns unrolled (30 us a step against 14: instruction
// cache), lanes of two rows (13.2-14.0 us against 9.2-12.5 then: the same number of
// instructions per lane), a separate copy of the column code for the edges, the
// neighbours' words waited for inside the edge column after what does not need
// them (stage A 3.9 us against 3.7 at 151 x 461: registers spill).
// Measured per shot step against the split kernels (B200, FP16 histories):
// 751 x 2301 (17 columns a CTA) forward 7.1 us against 20.1, stage A 10.8
// against 20.7-23.0, stage B 8.4 against 19.7-24.7; 151 x 461 (4 columns)
// 2.1-3.8 us against 12-15.
#include <algorithm>

#include "resident.cuh"
#include "tma.cuh"

namespace daw {
namespace {

typedef unsigned long long u64;

__device__ __forceinline__ u64 pk(float x, float y) {
  u64 r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(x), "f"(y));
  return r;
}
__device__ __forceinline__ float2 up(u64 v) {
  float2 r;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(v));
  return r;
}
__device__ __forceinline__ u64 add2(u64 a, u64 b) {
  u64 r;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ u64 sub2(u64 a, u64 b) {
  u64 r;
  asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
// A packed product rounded by itself: the assembler contracts mul.rn.f32x2
// with a following add or sub into one rounding (whatever the contraction
// options say), so the product is an fma with -0, a value it cannot know
// (`nz`, a kernel parameter).  a * b + (-0) rounds to a * b, signs included.
__device__ __forceinline__ u64 fma2(u64 a, u64 b, u64 c) {
  u64 r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
  return r;
}
constexpr u64 kNegZero2 = 0x8000000080000000ull;

// Four rows of a lane.
struct Q4 {
  u64 a, b;  // rows 0-1, 2-3
};
__device__ __forceinline__ Q4 add4(Q4 x, Q4 y) { return {add2(x.a, y.a), add2(x.b, y.b)}; }
__device__ __forceinline__ Q4 sub4(Q4 x, Q4 y) { return {sub2(x.a, y.a), sub2(x.b, y.b)}; }
__device__ __forceinline__ Q4 lds4(const Q4* p) {
  const ulonglong2 v = *reinterpret_cast<const ulonglong2*>(p);
  return {v.x, v.y};
}
__device__ __forceinline__ void sts4(Q4* p, Q4 v) {
  *reinterpret_cast<ulonglong2*>(p) = make_ulonglong2(v.a, v.b);
}
__device__ __forceinline__ Q4 pk4(float x, float y, float z, float w) { return {pk(x, y), pk(z, w)}; }
__device__ __forceinline__ float4 up4(Q4 v) {
  const float2 a = up(v.a), b = up(v.b);
  return make_float4(a.x, a.y, b.x, b.y);
}
constexpr Q4 kZero4{0ull, 0ull};

// (value, tag) words: a lane's four rows are four of them, in two 16-byte halves.
__device__ __forceinline__ void ll_store(ulonglong2* p, Q4 v, unsigned tag) {
  const float4 f = up4(v);
  const u64 t = (u64)tag << 32;
  asm volatile("st.relaxed.gpu.global.v2.b64 [%0], {%1, %2};" ::"l"(p),
               "l"(t | __float_as_uint(f.x)), "l"(t | __float_as_uint(f.y))
               : "memory");
  asm volatile("st.relaxed.gpu.global.v2.b64 [%0], {%1, %2};" ::"l"(p + 1),
               "l"(t | __float_as_uint(f.z)), "l"(t | __float_as_uint(f.w))
               : "memory");
}
__device__ __forceinline__ ulonglong2 ll_load(const ulonglong2* p) {
  ulonglong2 v;
  asm volatile("ld.relaxed.gpu.global.v2.b64 {%0, %1}, [%2];" : "=l"(v.x), "=l"(v.y) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ void word_store(u64* p, u64 v) {
  asm volatile("st.relaxed.gpu.global.b64 [%0], %1;" ::"l"(p), "l"(v) : "memory");
}
__device__ __forceinline__ u64 word_load(const u64* p) {
  u64 v;
  asm volatile("ld.relaxed.gpu.global.b64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
  return v;
}

// A warp's bounded polling: `give_up` is called every failed round; true once
// the limit is reached or another wait of the grid has run out.
struct Poll {
  unsigned* err;
  const int& limit;
  bool dead;
  __device__ __forceinline__ bool give_up(int n) {
    if (n < limit && (n & 255) != 255) return false;
    unsigned e;
    asm volatile("ld.relaxed.gpu.global.u32 %0, [%1];" : "=r"(e) : "l"(err) : "memory");
    // one decision for the warp: its lanes may see the flag at different times
    dead = __any_sync(kAll, (e & kErrTimeout) != 0 || n >= limit);
    if (dead && (threadIdx.x & 31) == 0) atomicOr(err, kErrTimeout);
    return dead;
  }
};

// N halo columns at p, p + stride, ...: polled until all words carry the tag; other
// loads may go out with the first round (`meanwhile`).
template <int N, typename F>
__device__ __forceinline__ void halo_get(const ulonglong2* p, size_t stride, unsigned tag, Poll& w,
                                         Q4 (&v)[N], F&& meanwhile) {
  ulonglong2 x[2 * N];
#pragma unroll
  for (int k = 0; k < 2 * N; ++k) x[k] = ll_load(p + (k / 2) * stride + (k & 1));
  meanwhile();  // other loads
  for (int n = 0;; ++n) {
    bool ok = true;
#pragma unroll
    for (int k = 0; k < 2 * N; ++k)
      ok = ok && (unsigned)(x[k].x >> 32) == tag && (unsigned)(x[k].y >> 32) == tag;
    if (w.dead || __all_sync(kAll, ok) || w.give_up(n)) break;
#pragma unroll
    for (int k = 0; k < 2 * N; ++k) x[k] = ll_load(p + (k / 2) * stride + (k & 1));
  }
#pragma unroll
  for (int k = 0; k < N; ++k)
    v[k] = {(x[2 * k].y << 32) | (unsigned)x[2 * k].x, (x[2 * k + 1].y << 32) | (unsigned)x[2 * k + 1].x};
}

// Maximum of the group's tagged words at `s` (G of them), by one warp.
__device__ __forceinline__ unsigned group_max(const u64* s, int G, unsigned tag, Poll& w) {
  unsigned m = 0;
  for (int i0 = 0; i0 < G; i0 += 128) {
    u64 v[4];
    for (int n = 0;; ++n) {
      bool ok = true;
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        const int i = i0 + 32 * k + (int)(threadIdx.x & 31);
        v[k] = i < G ? word_load(s + i) : (u64)tag << 32;
        ok = ok && (unsigned)(v[k] >> 32) == tag;
      }
      if (w.dead || __all_sync(kAll, ok) || w.give_up(n)) break;
    }
#pragma unroll
    for (int k = 0; k < 4; ++k) m = max(m, (unsigned)v[k]);
  }
  return __reduce_max_sync(kAll, m);
}

// Two maxima over the group's CTAs, by the extra warps: every CTA has stored
// its tagged words at s and s + stride; the leader collects them and stores the
// results to each CTA's own line at r.  (All CTAs polling all words made the lines
// they share the bottleneck: 3 us an exchange with 126 CTAs.  Each CTA storing its
// words to an array of every other, 20000 scattered stores, cost 1.4 us more a step
// at 151 x 461.  Exchanges with a whole step of time, the histories stored a step
// later from a copy: no gain, 3.6 against 3.7 us there and 4.6 against 4.2 at
// 301 x 703.)
constexpr int kLine = 16;  // words of a 128-byte line
__device__ __forceinline__ uint2 exchange_max(const u64* s, size_t stride, int fields, u64* r, int b,
                                              int G, int leader, unsigned tag, Poll& w) {
  const int lane = threadIdx.x & 31;
  uint2 m = make_uint2(0u, 0u);
  if (b == leader) {
    m.x = group_max(s, G, tag, w);
    if (fields > 1) m.y = group_max(s + stride, G, tag, w);
    for (int i = lane; i < G; i += 32) {
      word_store(r + (size_t)i * kLine, (u64)tag << 32 | m.x);
      word_store(r + (size_t)i * kLine + 1, (u64)tag << 32 | m.y);
    }
    return m;
  }
  const u64* own = r + (size_t)b * kLine + (lane & 1);
  u64 v;
  for (int n = 0;; ++n) {
    v = word_load(own);
    if (w.dead || __all_sync(kAll, (unsigned)(v >> 32) == tag) || w.give_up(n)) break;
  }
  m.x = __shfl_sync(kAll, (unsigned)v, 0);
  m.y = __shfl_sync(kAll, (unsigned)v, 1);
  return m;
}

// The history of a lane's four rows: FP16 in 64 bits, FP32 in 128.  Loads and
// stores are predicated (a load that is off gives 0), so that they cost no branch.
template <bool FP16>
struct HQuad;
template <>
struct HQuad<true> {
  typedef uint2 T;
  static __device__ __forceinline__ T load(const char* p, unsigned on) {
    T v;
    asm volatile(
        "{\n .reg .pred p;\n setp.ne.u32 p, %3, 0;\n mov.b32 %0, 0;\n mov.b32 %1, 0;\n"
        " @p ld.global.nc.L1::no_allocate.v2.b32 {%0, %1}, [%2];\n}"
        : "=&r"(v.x), "=&r"(v.y)
        : "l"(p), "r"(on));
    return v;
  }
  static __device__ __forceinline__ Q4 get(T v) {
    const float2 a = __half22float2(*reinterpret_cast<const __half2*>(&v.x));
    const float2 b = __half22float2(*reinterpret_cast<const __half2*>(&v.y));
    return {pk(a.x, a.y), pk(b.x, b.y)};
  }
  static __device__ __forceinline__ void put(char* p, Q4 v, uint64_t pol, unsigned on) {
    const float4 f = up4(v);
    const __half2 a = __floats2half2_rn(f.x, f.y), b = __floats2half2_rn(f.z, f.w);
    asm volatile(
        "{\n .reg .pred p;\n setp.ne.u32 p, %4, 0;\n"
        " @p st.global.L2::cache_hint.v2.b32 [%0], {%1, %2}, %3;\n}" ::"l"(p),
        "r"(*reinterpret_cast<const uint32_t*>(&a)), "r"(*reinterpret_cast<const uint32_t*>(&b)),
        "l"(pol), "r"(on)
        : "memory");
  }
};
template <>
struct HQuad<false> {
  typedef ulonglong2 T;
  static __device__ __forceinline__ T load(const char* p, unsigned on) {
    T v;
    asm volatile(
        "{\n .reg .pred p;\n setp.ne.u32 p, %3, 0;\n mov.b64 %0, 0;\n mov.b64 %1, 0;\n"
        " @p ld.global.nc.L1::no_allocate.v2.b64 {%0, %1}, [%2];\n}"
        : "=&l"(v.x), "=&l"(v.y)
        : "l"(p), "r"(on));
    return v;
  }
  static __device__ __forceinline__ Q4 get(T v) { return {v.x, v.y}; }
  static __device__ __forceinline__ void put(char* p, Q4 v, uint64_t pol, unsigned on) {
    asm volatile(
        "{\n .reg .pred p;\n setp.ne.u32 p, %4, 0;\n"
        " @p st.global.L2::cache_hint.v2.b64 [%0], {%1, %2}, %3;\n}" ::"l"(p),
        "l"(v.a), "l"(v.b), "l"(pol), "r"(on)
        : "memory");
  }
};

// Predicated shared-memory accesses.
__device__ __forceinline__ void sts_if(u64* p, u64 v, unsigned on) {
  asm volatile("{\n .reg .pred p;\n setp.ne.u32 p, %2, 0;\n @p st.shared.b64 [%0], %1;\n}" ::"r"(
                   smem_u32(p)),
               "l"(v), "r"(on)
               : "memory");
}
__device__ __forceinline__ void sts_if(Q4* p, Q4 v, unsigned on) {
  asm volatile("{\n .reg .pred p;\n setp.ne.u32 p, %3, 0;\n @p st.shared.v2.b64 [%0], {%1, %2};\n}" ::"r"(
                   smem_u32(p)),
               "l"(v.a), "l"(v.b), "r"(on)
               : "memory");
}
__device__ __forceinline__ void lds_if(float& v, const float* p, unsigned on) {
  asm volatile("{\n .reg .pred p;\n setp.ne.u32 p, %2, 0;\n @p ld.shared.f32 %0, [%1];\n}"
               : "+f"(v)
               : "r"(smem_u32(p)), "r"(on));
}
__device__ __forceinline__ void lds_if(float& x, float& y, const float* p, unsigned on) {
  asm volatile("{\n .reg .pred p;\n setp.ne.u32 p, %3, 0;\n @p ld.shared.v2.f32 {%0, %1}, [%2];\n}"
               : "+f"(x), "+f"(y)
               : "r"(smem_u32(p)), "r"(on));
}
// Four rows `ld` floats apart, each where its bit is set.
__device__ __forceinline__ void stg_rows(float* p, int ld, float4 v, unsigned rows) {
  asm volatile(
      "{\n .reg .pred p, q, r, s;\n .reg .b64 a, d;\n .reg .b32 t;\n"
      " and.b32 t, %6, 1;\n setp.ne.u32 p, t, 0;\n and.b32 t, %6, 2;\n setp.ne.u32 q, t, 0;\n"
      " and.b32 t, %6, 4;\n setp.ne.u32 r, t, 0;\n and.b32 t, %6, 8;\n setp.ne.u32 s, t, 0;\n"
      " mul.wide.s32 d, %1, 4;\n"
      " @p st.global.f32 [%0], %2;\n add.s64 a, %0, d;\n @q st.global.f32 [a], %3;\n"
      " add.s64 a, a, d;\n @r st.global.f32 [a], %4;\n add.s64 a, a, d;\n"
      " @s st.global.f32 [a], %5;\n}" ::"l"(p),
      "r"(ld), "f"(v.x), "f"(v.y), "f"(v.z), "f"(v.w), "r"(rows)
      : "memory");
}

__device__ __forceinline__ void l2_prefetch(const void* p, unsigned bytes) {
  asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(p), "r"(bytes) : "memory");
}

// Tensor memory as a scratchpad: 32-bit columns of 32 lanes per warp quadrant.
// A warp reaches the lanes of its quadrant (warp % 4) only.  A record is a
// lane's px and pz (8 words) and kappa (4 words) of one grid column.
__device__ __forceinline__ void tm_ld(unsigned a, Q4& x, Q4& z) {
  asm volatile(
      "{\n .reg .b32 r0, r1, r2, r3, r4, r5, r6, r7;\n"
      " tcgen05.ld.sync.aligned.32x32b.x8.b32 {r0, r1, r2, r3, r4, r5, r6, r7}, [%4];\n"
      " tcgen05.wait::ld.sync.aligned;\n"
      " mov.b64 %0, {r0, r1};\n mov.b64 %1, {r2, r3};\n mov.b64 %2, {r4, r5};\n mov.b64 %3, {r6, r7};\n}"
      : "=l"(x.a), "=l"(x.b), "=l"(z.a), "=l"(z.b)
      : "r"(a));
}
// the same with kappa's record at k
__device__ __forceinline__ void tm_ld(unsigned a, unsigned k, Q4& x, Q4& z, Q4& q) {
  asm volatile(
      "{\n .reg .b32 r0, r1, r2, r3, r4, r5, r6, r7, q0, q1, q2, q3;\n"
      " tcgen05.ld.sync.aligned.32x32b.x8.b32 {r0, r1, r2, r3, r4, r5, r6, r7}, [%6];\n"
      " tcgen05.ld.sync.aligned.32x32b.x4.b32 {q0, q1, q2, q3}, [%7];\n"
      " tcgen05.wait::ld.sync.aligned;\n"
      " mov.b64 %0, {r0, r1};\n mov.b64 %1, {r2, r3};\n mov.b64 %2, {r4, r5};\n mov.b64 %3, {r6, r7};\n"
      " mov.b64 %4, {q0, q1};\n mov.b64 %5, {q2, q3};\n}"
      : "=l"(x.a), "=l"(x.b), "=l"(z.a), "=l"(z.b), "=l"(q.a), "=l"(q.b)
      : "r"(a), "r"(k));
}
__device__ __forceinline__ void tm_st(unsigned a, Q4 x, Q4 z) {
  asm volatile(
      "{\n .reg .b32 r0, r1, r2, r3, r4, r5, r6, r7;\n"
      " mov.b64 {r0, r1}, %1;\n mov.b64 {r2, r3}, %2;\n mov.b64 {r4, r5}, %3;\n mov.b64 {r6, r7}, %4;\n"
      " tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {r0, r1, r2, r3, r4, r5, r6, r7};\n}" ::"r"(a),
      "l"(x.a), "l"(x.b), "l"(z.a), "l"(z.b)
      : "memory");
}
__device__ __forceinline__ void tm_st(unsigned a, Q4 x) {
  asm volatile(
      "{\n .reg .b32 r0, r1, r2, r3;\n mov.b64 {r0, r1}, %1;\n mov.b64 {r2, r3}, %2;\n"
      " tcgen05.st.sync.aligned.32x32b.x4.b32 [%0], {r0, r1, r2, r3};\n}" ::"r"(a),
      "l"(x.a), "l"(x.b)
      : "memory");
}
__device__ __forceinline__ void tm_wait_st() {
  asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
}
// The CTA barrier, which also orders tensor-memory accesses of different warps.
__device__ __forceinline__ void sync_cta() {
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
}

// Shared-memory layout (offsets in bytes, 16-byte aligned sections).
struct Lay {
  int fld, edge, col, row, tcd, term, tsta, tkap, amp, stage, p, misc, total;
};
__host__ __device__ inline Lay layout(int C, int RB, int pts, int m, int nsta, int quads, bool ps) {
  Lay l;
  int o = 0;
  auto take = [&](int bytes) {
    const int at = o;
    o += (bytes + 15) / 16 * 16;
    return at;
  };
  // [row block][column -2 .. C][vx, vz][lane] quads; columns -2, -1 and C hold
  // the neighbours' vx
  l.fld = take(RB * (C + 3) * 1024);
  l.edge = take((RB + 2) * C * 16);  // [row block + 1][column][first, last pair of p]
  l.col = take(C * 32);              // [column][d2a, d2a, d2a1, d2a1, d2b, d2b, bw2, bw2]
  l.row = take(4 * RB * 512);        // d1a, d1a1, d1b, bw1
  l.tcd = take(pts * m * 4);
  l.term = take(pts * m * 4);
  l.tsta = take(pts * m * 2);
  l.tkap = take(pts * 4);
  l.amp = take(2 * (nsta + 1) * 4);  // amplitudes of one step and the next
  l.stage = take(quads * C * 16);    // pressure of the gather rectangles [quad][column]
  l.p = take(ps ? RB * (C + 3) * 512 : 0);  // [row block][column -1 .. C + 1][lane] quads of p
  l.misc = take(64 * 4 + 16);
  l.total = o;
  return l;
}
// Where p is, and with it which warps may share a row block.  Warp w reaches the
// quadrant w % 4 of the tensor memory only, and at the borders of its columns it
// reads p of the other column groups' warps.
// - In tensor memory: a row block's warps share a quadrant, so the column groups
//   are a multiple of 4 warps apart and the extra warp is in a gap or at the end.
//   Five to seven row blocks load the four SM quadrants unevenly, one to three
//   leave some idle.
// - In shared memory too (PS, where it has room: 512 bytes per column and row
//   block): tensor memory is private to a warp and the warps fill the quadrants
//   in turn.
__host__ __device__ inline int group_warps(int RB, bool ps) { return ps ? RB : (RB + 3) / 4 * 4; }
__host__ __device__ inline int cta_warps(int RB, int CG, bool ps) {
  return !ps && RB % 4 ? CG * group_warps(RB, ps) : CG * group_warps(RB, ps) + 1;
}
__host__ __device__ inline int aux_warp(int RB, int CG, bool ps) {
  return !ps && RB % 4 ? RB : CG * group_warps(RB, ps);
}
// Tensor-memory columns.  p in tensor memory: per row block of a quadrant px, pz
// of the grid columns -1 .. C + 1 (those outside 0 .. C - 1 hold the neighbours'
// p), kappa of 0 .. C - 1; else per warp of a quadrant px, pz and kappa of its CW
// columns.
__host__ __device__ inline int tm_words(int C, int RB, int CG, int CW, bool ps) {
  return ps ? (RB * CG + 3) / 4 * (CW * 12) : (RB + 3) / 4 * ((C + 3) * 8 + C * 4);
}
__host__ __device__ inline int tm_alloc(int C, int RB, int CG, int CW, bool ps) {
  int n = 32;
  while (n < tm_words(C, RB, CG, CW, ps)) n *= 2;
  return n;
}

// The injection terms ((c dt) amp) kappa of one step, by thread t of nt.
__device__ __forceinline__ void inj_terms(unsigned char* sm, const Lay& l, int pts, int m, const float* amp,
                                          int t, int nt) {
  const float2* cd = reinterpret_cast<const float2*>(sm + l.tcd);
  float2* term = reinterpret_cast<float2*>(sm + l.term);
  const ushort2* sta = reinterpret_cast<const ushort2*>(sm + l.tsta);
  const float* kap = reinterpret_cast<const float*>(sm + l.tkap);
  const int mh = m / 2;
  for (int p = t; p < pts; p += nt) {
    const float kv = kap[p];
    for (int k = 0; k < mh; ++k) {
      const float2 c = cd[p * mh + k];
      const ushort2 s = sta[p * mh + k];
      term[p * mh + k] = make_float2(fmul(fmul(c.x, amp[s.x]), kv), fmul(fmul(c.y, amp[s.y]), kv));
    }
  }
}

template <int MODE, bool FP16, bool RHO, bool PS>
__global__ void __launch_bounds__(32 * kResWarps, 1)
    k_resident(const __grid_constant__ Grid g, const __grid_constant__ ModelDev md,
               const __grid_constant__ ResidentLaunch L) {
  constexpr bool kA = MODE == FM_STAGE_A, kB = MODE == FM_STAGE_B, kF = MODE == FM_FWD;
  constexpr int FS = 64;  // quads between a lane's columns
  constexpr int HR = 2;   // history columns read ahead
  // The wait for the right neighbour's words stands between two parts of a warp's columns,
  // or in the column code, four times over.  us per step with parts and without:
  //              751 x 2301   600 x 600    301 x 703    151 x 461
  //   forward     6.93  7.12   3.43  3.15   2.59  2.52   2.20  2.11
  //   A, FP16    10.9  10.8    4.99  4.71   4.12  3.96   3.7   3.8
  //   A, FP32    10.5  10.9    3.71  3.97   3.66  4.05   2.81  2.98
  //   B           8.41  9.19   4.15  4.10   3.45  3.86   2.63  2.78
  // Tried in place of the wait, stage B at 751 x 2301:
  // - the words copied to shared memory a few columns ahead by cp.async, which is a weak
  //   access and races with the neighbour's store in the memory model: 8.78;
  // - loaded a few columns ahead and put into shared memory by the lane, at once: 9.62; at
  //   the end of the column: 11.5 (registers spill);
  // - copied by the extra warp: 12.1.
  constexpr bool kParts = kB || (kA && !FP16);
  using HQ = HQuad<FP16>;
  using HT = typename HQ::T;
  extern __shared__ __align__(16) unsigned char sm[];
  const int C = L.C, G = L.G, RB = L.RB;
  const Lay l = layout(C, RB, L.inj_pts, L.inj_m, L.inj_sta, L.quads, PS);
  const int grp = blockIdx.x / G, b = blockIdx.x - grp * G;
  const ResidentShot& S = L.shot[grp];
  // the warp index from a shuffle: the compiler then knows that it, and all
  // control that follows from it, is uniform over the warp
  const int tid = threadIdx.x, lane = tid & 31, warp = __shfl_sync(kAll, tid >> 5, 0);
  const int rb = warp % group_warps(RB, PS), cg = warp / group_warps(RB, PS);  // row block, column group
  const bool aux = warp == aux_warp(RB, L.CG, PS);
  const bool comp = !aux && rb < RB && cg < L.CG;  // else an idle warp: barriers only
  const int c0 = b * C, i1 = 128 * rb + 4 * lane;
  const int npml = g.npml, ld = g.ld;
  const int first = S.first, last = S.last;
  if (first > last) return;             // uniform over the group
  // the warp's columns; the first group, whose edge costs more, has those left over
  const int over = L.CG * L.CW - C;
  const int clo = max(cg * L.CW - over, 0), chi = min(C, cg * L.CW + L.CW - over);
  // the lane's vx, vz of column j: F[FS j], F[FS j + 32]; the vz pair above and the row below it at FU, FD (lanes 0 and 31: in the
  // neighbouring row blocks; the grid's first and last rows, which are never
  // updated, stand for the zeros beyond them)
  const int BS = (C + 3) * FS;  // quads between row blocks
  Q4* const F = reinterpret_cast<Q4*>(sm + l.fld) + (comp ? rb : 0) * BS + 2 * FS + lane;
  const u64* const FU = lane > 0 ? &(F + 31)->b : rb > 0 ? &(F + 63 - BS)->b : &(F + 32)->a;
  const float* const FD = reinterpret_cast<const float*>(
      lane < 31 ? F + 33 : rb < RB - 1 ? F + 1 + BS : F + 32) + (lane == 31 && rb >= RB - 1 ? 3 : 0);
  Q4* const PP = reinterpret_cast<Q4*>(sm + l.p) + (comp ? rb : 0) * (C + 3) * 32 + 32 + lane;  // PS: p of column j at 32 j
  u64* const ED = reinterpret_cast<u64*>(sm + l.edge) + (rb + 1) * C * 2;
  ulonglong2* const CF = reinterpret_cast<ulonglong2*>(sm + l.col);
  Q4* const ROW = reinterpret_cast<Q4*>(sm + l.row) + rb * 32 + lane;
  const int NP = RB * 32;
  float* const TERM = reinterpret_cast<float*>(sm + l.term);
  auto amp = [&](int it) { return reinterpret_cast<float*>(sm + l.amp) + (it & 1) * (L.inj_sta + 1); };
  unsigned* const WM = reinterpret_cast<unsigned*>(sm + l.misc);     // [3] maxima: p, vx, vz
  float* const SC = reinterpret_cast<float*>(sm + l.misc + 16 * 4);  // scales
  unsigned* const TB = reinterpret_cast<unsigned*>(sm + l.misc + 64 * 4);
  const unsigned top = lane == 0, bottom = lane == 31;
  Poll poll{L.err, L.poll_limit, false};
  const int4 ih = S.inj.pts > 0 ? S.inj.head[b] : make_int4(0, 0, 0, 0);
  const int ipts = ih.y > 0 ? C * ih.y : 0;
  const int im = L.inj_m;

  // ---- set-up
  const unsigned tcols = (unsigned)tm_alloc(C, RB, L.CG, L.CW, PS);
  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                     smem_u32(TB)),
                 "r"(tcols)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  sync_cta();
  // px, pz of column j: TP + 8 j (lane 32 (warp % 4) of the allocation)
  const unsigned TQ = __shfl_sync(kAll, *TB, 0) + ((unsigned)(warp & 3) << 21);
  const unsigned TW = TQ + (warp >> 2) * L.CW * 12;  // PS: the warp's records
  const unsigned TP = PS ? TW - 8 * clo : TQ + (rb >> 2) * (C + 3) * 8 + 8;
  // kappa: TK + 4 j
  const unsigned TK = PS ? TW + 8 * L.CW - 4 * clo
                         : TQ + group_warps(RB, PS) / 4 * (C + 3) * 8 + (rb >> 2) * C * 4;
  {
    const int off = kF ? 2 : 3;
    const int hi1 = g.n1e - off, hi2 = g.n2e - off;
    const int fsrows = g.ofs == 1 ? npml + 1 : 0;
    for (int j = tid; j < C; j += blockDim.x) {
      const int c = c0 + j;
      const bool in = c < g.n2e, u = c >= 2 && c < hi2;
      const float4 q = in ? md.pcol[c] : make_float4(0.f, 0.f, 0.f, 0.f);
      CF[2 * j] = make_ulonglong2(pk(q.x, q.x), pk(q.y, q.y));
      const float w = RHO ? 1.f : q.w;
      CF[2 * j + 1] = make_ulonglong2(pk(q.z, q.z), u ? pk(w, w) : 0ull);
    }
    if (comp) {
      bool u[4];
      if (cg == 0) {
        float f[4][4];
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          const int r = i1 + k;
          const float4 q = r < g.n1e ? md.prow[r] : make_float4(0.f, 0.f, 0.f, 0.f);
          f[0][k] = q.x;
          f[1][k] = q.y;
          f[2][k] = q.z;
          f[3][k] = r >= 2 && r < hi1 ? (RHO ? 1.f : q.w) : 0.f;
        }
#pragma unroll
        for (int k = 0; k < 4; ++k) sts4(ROW + k * NP, pk4(f[k][0], f[k][1], f[k][2], f[k][3]));
      }
#pragma unroll
      for (int k = 0; k < 4; ++k) u[k] = i1 + k >= max(2, fsrows) && i1 + k < hi1;
      for (int j = clo; j < chi; ++j) {
        const int c = c0 + j;
        Q4 x = kZero4, z = kZero4, k4 = kZero4, px = kZero4, pz = kZero4;
        if (c < g.n2e && i1 < ld) {
          const size_t o = (size_t)c * ld + i1;
          if (c >= 2 && c < hi2) {
            // kappa (dtdx kappa where only that is used), zero where the
            // pressure is not updated or is zeroed at the free surface: px and
            // pz then stay zero there
            const float4 q = *reinterpret_cast<const float4*>(md.kap + o);
            const float s = kB ? 1.f : g.dtdx;
            k4 = pk4(u[0] ? fmul(s, q.x) : 0.f, u[1] ? fmul(s, q.y) : 0.f,
                     u[2] ? fmul(s, q.z) : 0.f, u[3] ? fmul(s, q.w) : 0.f);
          }
          if (L.load) {
            x = lds4(reinterpret_cast<const Q4*>(S.vx + o));
            z = lds4(reinterpret_cast<const Q4*>(S.vz + o));
            px = lds4(reinterpret_cast<const Q4*>(S.px + o));
            pz = lds4(reinterpret_cast<const Q4*>(S.pz + o));
          }
        }
        sts4(F + FS * j, x);
        sts4(F + FS * j + 32, z);
        __syncwarp();
        tm_st(TP + 8 * j, px, pz);
        tm_st(TK + 4 * j, k4);
      }
      // the neighbours' columns: zero where there is no neighbour, their vx of
      // the state where the first step needs it
      if (cg == 0)
        for (int j = -2; j <= C; j = j == -1 ? C : j + 1) {
          const int c = c0 + j;
          Q4 x = kZero4;
          if (L.load && c >= 0 && c < g.n2e && i1 < ld)
            x = lds4(reinterpret_cast<const Q4*>(S.vx + (size_t)c * ld + i1));
          sts4(F + FS * j, x);
          sts4(F + FS * j + 32, kZero4);
        }
      __syncwarp();
      if (PS && cg == 0) {
        sts4(PP - 32, kZero4);
        sts4(PP + 32 * C, kZero4);
        sts4(PP + 32 * C + 32, kZero4);
      }
      if (!PS && cg == 0) {
        tm_st(TP - 8, kZero4, kZero4);
        tm_st(TP + 8 * C, kZero4, kZero4);
        tm_st(TP + 8 * C + 8, kZero4, kZero4);
      }
      tm_wait_st();
    }
    for (int k = tid; k < C * 2 * (RB + 2); k += blockDim.x)
      reinterpret_cast<u64*>(sm + l.edge)[k] = 0ull;
    if (tid < 3) WM[tid] = 0u;
    if (tid < 8) SC[tid] = 1.f;
    if (ipts > 0) {
      const size_t o = (size_t)b * S.inj.pts;
      float* tcd = reinterpret_cast<float*>(sm + l.tcd);
      unsigned short* tst = reinterpret_cast<unsigned short*>(sm + l.tsta);
      float* tk = reinterpret_cast<float*>(sm + l.tkap);
      for (int k = tid; k < ipts * im; k += blockDim.x) {
        // the shot's own table has S.inj.m entries per point
        const int p = k / im, e = k - p * im;
        const bool in = e < S.inj.m;
        tcd[k] = in ? S.inj.cd[(o + p) * S.inj.m + e] : 0.f;
        const int s = in ? S.inj.sta[(o + p) * S.inj.m + e] : 0xffff;
        tst[k] = (unsigned short)(s < ih.w ? s : ih.w);
      }
      for (int k = tid; k < ipts; k += blockDim.x)  // rows above the surface: px stays zero
        tk[k] = ih.x + k % ih.y < fsrows ? 0.f : S.inj.kap[o + k];
      for (int k = tid; k <= ih.w; k += blockDim.x)
        amp(first - 1)[k] = k < ih.w ? S.amp[(size_t)(first - 1) * S.nsta + ih.z + k] : 0.f;
      if (tid == 0) amp(first)[ih.w] = 0.f;
    }
  }
  __syncthreads();
  // Amplitudes of step it + 1 to amp(it), by the extra warp: a step ahead and
  // without waiting, since they come from memory and the warp's exchange follows
  // (stage A at 151 x 461: 3.7 us a step against 3.9 with the loads waited for).
  auto fetch_amp = [&](int it) {
    if (!kB && ipts > 0 && it < last)
      for (int k = lane; k < ih.w; k += 32)
        asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(smem_u32(amp(it) + k)),
                     "l"(S.amp + (size_t)it * S.nsta + ih.z + k)
                     : "memory");
  };
  if (aux) fetch_amp(first);
  // the warps but the extra one
  const int it0 = tid - (warp > aux_warp(RB, L.CG, PS) ? 32 : 0), itn = blockDim.x - 32;
  if (ipts > 0 && !aux) inj_terms(sm, l, ipts, im, amp(first - 1), it0, itn);

  const u64 nz = L.nz;
  auto mul2 = [&](u64 x, u64 y) { return fma2(x, y, nz); };
  auto mul4 = [&](Q4 x, Q4 y) -> Q4 { return {mul2(x.a, y.a), mul2(x.b, y.b)}; };
  auto mul41 = [&](Q4 x, u64 y) -> Q4 { return {mul2(x.a, y), mul2(x.b, y)}; };
  // ---- per-lane constants
  unsigned rows = 0;  // bit k: row i1 + k is physical
#pragma unroll
  for (int k = 0; k < 4; ++k) rows |= (i1 + k >= npml && i1 + k < npml + g.n1 ? 1u : 0u) << k;
  if (!comp) rows = 0;
  // a warp with quads only part of which is physical masks its values
  const bool part = __any_sync(kAll, rows != 0 && rows != 15u);
  auto keep = [&](Q4 v, unsigned bits) -> Q4 {
    const float4 f = up4(v);
    return pk4(bits & 1 ? f.x : 0.f, bits & 2 ? f.y : 0.f, bits & 4 ? f.z : 0.f, bits & 8 ? f.w : 0.f);
  };
  // running max |x|, NaN if any value is
  auto amax = [&](float m, Q4 v) {
    if (part) v = keep(v, rows);
    const float4 f = up4(v);
    float d;
    asm("max.NaN.abs.f32 %0, %1, %2, %3;" : "=f"(d) : "f"(m), "f"(f.x), "f"(f.y));
    asm("max.NaN.abs.f32 %0, %1, %2, %3;" : "=f"(m) : "f"(d), "f"(f.z), "f"(f.w));
    return m;
  };
  auto splat = [](float v) { return pk(v, v); };
  const int jlo = max(0, npml - c0), jhi = min(C, npml + g.n2 - c0);  // physical columns [jlo, jhi)
  const unsigned phys = jhi > jlo ? (1u << jhi) - (1u << jlo) : 0u;
  const unsigned lphys = rows ? phys : 0u;  // of lanes with a physical row
  const int n1h = L.n1h;
  const size_t nih = (size_t)n1h * g.n2;
  const int hoff = i1 - g.hist_base() + n1h * (c0 - npml);  // history offset of column 0
  constexpr int kEs = FP16 ? 2 : 4;
  auto hist_at = [&](int slot, int f) {
    return static_cast<char*>(S.hist) + ((size_t)slot * 3 + f) * nih * kEs;
  };
  const int hstep = n1h * kEs;  // bytes from one column to the next
  const u64 A0 = pk(kA0, kA0), A1 = pk(kA1, kA1), DTDX = pk(g.dtdx, g.dtdx);
  const float mdt = fmul(-1.0f, g.dt);
  const u64 MDT = pk(mdt, mdt);
  const uint64_t pol = l2_evict_first();
  // halo words: [phase][parity][cta][3][NP][2]
  const size_t hcol = (size_t)2 * NP, hcta = 3 * hcol, hpar = hcta * gridDim.x;
  ulonglong2* const hmine = L.halo + (size_t)blockIdx.x * hcta + 2 * (32 * rb + lane);
  const bool hasl = b > 0, hasr = b + 1 < G;
  const bool inj_on = ipts > 0 && comp && i1 + 3 >= ih.x && i1 < ih.x + ih.y;
  const bool inj_warp = !kB && ipts > 0 && comp && 128 * rb + 127 >= ih.x && 128 * rb < ih.x + ih.y;
  // Rectangles kept for the gathers.  With room in shared memory (L.quads) the
  // lanes put their quads there and the extra warp writes them to memory during
  // the velocity half step, a row's columns together; else the lanes write their
  // rows: the lane's rows and the address of its first row and the CTA's first
  // column at the current step.
  unsigned rcol[2] = {}, rrow[2] = {};  // written by the lanes: the CTA's columns, the lane's rows
  float* rptr[2] = {};
  Q4* const stage = reinterpret_cast<Q4*>(sm + l.stage);
  const bool staged = !kA && L.quads > 0;
  Q4* sptr[2] = {stage, stage};
  unsigned son[2] = {};  // staged: the lane's quad is one of the rectangle's
  if (!kA && comp)
#pragma unroll
    for (int q = 0; q < 2; ++q) {
      const ResidentRect& R = S.rect[q];
      if (!R.buf || 128 * rb + 127 < R.r0 || 128 * rb >= R.r1) continue;
      unsigned rows4 = 0;
#pragma unroll
      for (int k = 0; k < 4; ++k) rows4 |= (i1 + k >= R.r0 && i1 + k < R.r1 ? 1u : 0u) << k;
      if (staged) {
        son[q] = rows4;
        if (rows4) sptr[q] = stage + (R.quad0 + (i1 - (R.r0 & ~3)) / 4) * C;
      } else {
        const int a = max(R.c0 - c0, 0), e = min(R.c1 - c0, C);
        rcol[q] = e > a ? (1u << e) - (1u << a) : 0u;
        rrow[q] = rows4;
        rptr[q] = R.buf + (ptrdiff_t)(i1 - R.r0) * R.ld + (c0 - R.c0);
      }
    }
  // warps with more to do per column than the update (warp-uniform)
  const bool extra = !kA && comp && ((rcol[0] | rcol[1]) != 0 || S.wf != nullptr);
  // free-surface copy vz(npml - 1) = vz(npml)
  const bool fs_warp = g.ofs == 1 && (npml - 1) / 128 == rb;
  const int fsk = npml - 1 - i1;  // 0 .. 3 in the lane that owns row npml - 1
  const int slo = L.slo;
  const int sjlo = max(0, npml + slo - c0), sjhi = min(C, npml + g.n2 - slo - c0);
  const unsigned srcs = sjhi > sjlo ? (1u << sjhi) - (1u << sjlo) : 0u;  // source columns
  const unsigned lsrc = rows ? srcs : 0u;
  unsigned srows = 0;  // rows of the pressure source
#pragma unroll
  for (int k = 0; k < 4; ++k)
    srows |= (i1 + k >= npml + slo && i1 + k < npml + g.n1 - slo ? 1u : 0u) << k;
  const bool spart = kB && __any_sync(kAll, (srows & rows) != rows);
  HT hq[HR] = {}, hx[HR] = {}, hz[HR] = {};  // stage B: history quads read ahead
  auto slot_b = [&](int it) { return S.nt - it - L.hist_step0; };  // the time-reversed step's
  auto ldh = [&](const char* base, int j, unsigned mask) -> HT {
    return HQ::load(base + (ptrdiff_t)(hoff + j * n1h) * kEs, mask >> j & 1u);
  };
  // stage B: scales of one step (extra warp), and the L2 prefetch of its history
  auto scales_b = [&](int it) {
    if (FP16) {
      const unsigned* a = S.amax + (size_t)slot_b(it) * 3 * kAmaxSlots;
      float sc[3];
#pragma unroll
      for (int f = 0; f < 3; ++f)
        sc[f] = pow2f(amax_exponent(__reduce_max_sync(kAll, a[f * kAmaxSlots + lane])) - 15);
      if (lane < 3) SC[(it & 1) * 3 + lane] = lane == 0 ? sc[0] : lane == 1 ? sc[1] : sc[2];
    }
  };
  auto prefetch_b = [&](int it) {
    if (lane < 3 && it <= last && jhi > jlo)
      l2_prefetch(static_cast<const char*>(S.hist) +
                      (((size_t)slot_b(it) * 3 + lane) * nih + (size_t)(c0 + jlo - npml) * n1h) * kEs,
                  (unsigned)((jhi - jlo) * n1h * kEs));
  };
  const bool ledge = comp && clo == 0, redge = comp && chi == C;
  // the warp's first columns of the pressure and velocity half steps
  const int pj0 = chi > 2 ? max(clo, 2) : clo, vj0 = ledge && chi > 1 ? 1 : clo;
  if (kB) {
    if (aux) {
      scales_b(first);
      prefetch_b(first + 1);
    } else if (comp) {
#pragma unroll
      for (int u = 0; u < HR; ++u) hq[u] = ldh(hist_at(slot_b(first), 0), pj0 + u, lsrc);
    }
  }
  // stage A: the lines of the exchanged maxima, [phase][parity][cta], and the
  // CTA that collects the velocities' (the pressure's: CTA 0)
  const int vleader = G / 2;
  auto results = [&](int phase, int s) {
    return L.slots + (size_t)8 * gridDim.x +
           ((size_t)(phase * 2 + (s & 1)) * gridDim.x + grp * G) * kLine;
  };
  auto words = [&](int phase, int s) {
    return L.slots + (size_t)(phase * 4 + (s & 1) * 2) * gridDim.x + grp * G;
  };
  // of step s: maxima to memory, scales to SC
  auto exchange_p = [&](int s) {
    const uint2 m = exchange_max(words(0, s), 0, 1, results(0, s), b, G, 0, L.tag0 + (unsigned)s, poll);
    if (lane == 0) {
      SC[0] = pow2f(15 - amax_exponent(m.x));
      if (b == 0) S.amax[(size_t)(s - 1) * 3 * kAmaxSlots] = m.x;
    }
  };
  auto exchange_v = [&](int s) {
    const uint2 m = exchange_max(words(1, s), gridDim.x, 2, results(1, s), b, G, vleader,
                                 L.tag0 + (unsigned)s, poll);
    if (lane == 0) {
      SC[1] = pow2f(15 - amax_exponent(m.x));
      SC[2] = pow2f(15 - amax_exponent(m.y));
      if (b == 0) {
        unsigned* am = S.amax + (size_t)(s - 1) * 3 * kAmaxSlots;
        am[kAmaxSlots] = m.x;
        am[2 * kAmaxSlots] = m.y;
      }
    }
  };
  sync_cta();

  for (int it = first; it <= last; ++it) {
    const unsigned tag = L.tag0 + (unsigned)it;
    // =============== pressure half step ===============
    if (comp) {
      const Q4 d1a = lds4(ROW), d1a1 = lds4(ROW + NP);
      const u64 INV = splat(kA && FP16 ? SC[0] : 1.f), SCP = splat(kB ? SC[(it & 1) * 3] : 1.f);
      const unsigned put = kA && it > first && rows ? 1u : 0u;
      char* const hp = hist_at(kA ? max(it - 2, 0) : slot_b(it), 0);
      float lmax = 0.f;
      ulonglong2* const hout = hmine + (size_t)(it & 1) * hpar;  // phase 0: p words
      const ulonglong2* const hin = hmine + (size_t)(2 + ((it - 1) & 1)) * hpar;  // vx words
      // The warp's columns in order, those of the left edge (0 and 1) last: the
      // neighbours' words are put into columns C, -2 and -1 when they are needed.
      const bool rhalo = hasr && redge && it > first, lhalo = hasl && clo < 2 && it > first;
      const unsigned outs = (hasr ? 1u << (C - 1) : 0u) | (hasl ? 3u : 0u);
      auto put_left = [&]() {
        auto histories = [&]() {  // of the warp's columns below 2
          if (!kB) return;
          hq[0] = ldh(hp, clo, lsrc);
          hq[1] = ldh(hp, clo + 1, lsrc);
        };
        if (!lhalo) {
          histories();
          return;
        }
        Q4 h[2];
        halo_get(hin - hcta, hcol, tag - 1, poll, h, histories);
        sts4(F - 2 * FS, h[0]);
        sts4(F - FS, h[1]);
      };
      auto put_right = [&]() {
        Q4 r[1];
        halo_get(hin + hcta + 2 * hcol, hcol, tag - 1, poll, r, [] {});
        sts4(F + FS * C, r[0]);
      };
      const unsigned wait = !kParts && rhalo ? 1u << (C - 1) : 0u;
      // Columns [j, je): four to an iteration, so that the window's registers
      // rotate without copies.  Arrays at column j, masks shifted by j.
      auto columns = [&](int j, int je) {
        Q4* f = F + FS * j;
        const u64* fu = FU + 2 * FS * j;
        const float* fd = FD + 4 * FS * j;
        Q4* pp = PP + 32 * j;
        const ulonglong2* cf = CF + 2 * j;
        u64* ed = ED + 2 * j;
        unsigned tp = TP + 8 * j, tk = TK + 4 * j, ho = (unsigned)((hoff + j * n1h) * kEs);
        unsigned ev = wait >> j, ot = outs >> j, ph = phys >> j, src = lsrc >> j;
        int n = je - j;
        Q4 *sp0 = sptr[0] + j, *sp1 = sptr[1] + j;
        Q4 w0 = lds4(f - 2 * FS), w1 = lds4(f - FS), w2 = lds4(f), w3;
        auto column = [&](const int k, const Q4& w0, const Q4& w1, const Q4& w2, Q4& w3) {
          if (!kParts && (ev & (1u << k))) put_right();
          w3 = lds4(f + FS * (k + 1));
          const float4 z = up4(lds4(f + FS * k + 32));
          const float2 zm = up(fu[2 * FS * k]);
          const float zp = fd[4 * FS * k];
          const ulonglong2 c2 = cf[2 * k];
          Q4 px, pz, kap;
          tm_ld(tp + 8 * k, tk + 4 * k, px, pz, kap);
          const Q4 der2 = add4(mul41(sub4(w2, w1), A0), mul41(sub4(w3, w0), A1));
          const Q4 der1 = add4(mul41(pk4(fsub(z.x, zm.y), fsub(z.y, z.x), fsub(z.z, z.y), fsub(z.w, z.z)), A0),
                               mul41(pk4(fsub(z.y, zm.x), fsub(z.z, zm.y), fsub(z.w, z.x), fsub(zp, z.y)), A1));
          if (kA && (ph & (1u << k))) {  // history of the previous step's pressure
            Q4 v = mul41(add4(px, pz), INV);
            if (part) v = keep(v, rows);
            HQ::put(hp + (ho + k * hstep), v, pol, put);
          }
          const Q4 kd = kB ? mul41(kap, DTDX) : kap;
          const Q4 bx = mul4(mul41(kd, c2.y), der2), bz = mul4(mul4(kd, d1a1), der1);
          const Q4 ax = mul41(px, c2.x), az = mul4(d1a, pz);
          px = kA ? sub4(ax, bx) : add4(ax, bx);
          pz = kA ? sub4(az, bz) : add4(az, bz);
          if (inj_warp) {
            if (inj_on) {  // the lane's four rows are rows of the table
              float4 v = up4(px);
              const float* t0 = TERM + ((j + k) * ih.y + (i1 - ih.x)) * im;
              const float2* t = reinterpret_cast<const float2*>(t0);
              // a forward run's map has one station: one term a point
              const int mh = kF ? 0 : im >> 1;
              if (kF) {
                v.x = fadd(v.x, t0[0]);
                v.y = fadd(v.y, t0[im]);
                v.z = fadd(v.z, t0[2 * im]);
                v.w = fadd(v.w, t0[3 * im]);
              }
              for (int q = 0; q < mh; ++q) {
                const float2 a = t[q], e = t[mh + q], c = t[2 * mh + q], d = t[3 * mh + q];
                v.x = fsub(fsub(v.x, a.x), a.y);
                v.y = fsub(fsub(v.y, e.x), e.y);
                v.z = fsub(fsub(v.z, c.x), c.y);
                v.w = fsub(fsub(v.w, d.x), d.y);
              }
              px = pk4(v.x, v.y, v.z, v.w);
            }
            __syncwarp();
          }
          if (kB) {  // points outside the physical range read 0
            Q4 v = mul41(HQ::get(hq[k % HR]), SCP);
            if (spart) v = keep(v, srows);
            px = add4(px, mul4(mul41(v, MDT), kap));
            hq[k % HR] = HQ::load(hp + (ho + (k + HR) * hstep), src & (1u << (k + HR)));
          }
          tm_st(tp + 8 * k, px, pz);
          const Q4 p = add4(px, pz);
          if (PS) sts4(pp + 32 * k, p);
          sts_if(ed + 2 * k, p.a, top);
          sts_if(ed + 2 * k + 1, p.b, bottom);
          if (kA && (ph & (1u << k))) lmax = amax(lmax, p);
          if (!kA) {  // no branch: its code would be cold for the few warps that take it
            sts_if(sp0 + k, p, son[0]);
            sts_if(sp1 + k, p, son[1]);
          }
          if (extra) {
            // pressure rows of the gather rectangles, and the wavefield output
            const float4 v = up4(p);
            if (rcol[0] >> (j + k) & 1u) stg_rows(rptr[0] + j + k, S.rect[0].ld, v, rrow[0]);
            if (rcol[1] >> (j + k) & 1u) stg_rows(rptr[1] + j + k, S.rect[1].ld, v, rrow[1]);
            if (S.wf && (ph & (1u << k))) {
              float* w = S.wf + (size_t)(it - 1) * g.int_elems() + (size_t)g.n1 * (c0 + j + k - npml) + (i1 - npml);
              const bool acc = S.wf_acc != 0;
              const int top_zero = g.ofs == 1 ? npml - i1 : -1;  // the lane's last row of zeros
              const float4 u = make_float4(top_zero < 0 ? v.x : 0.f, top_zero < 1 ? v.y : 0.f,
                                           top_zero < 2 ? v.z : 0.f, top_zero < 3 ? v.w : 0.f);
              if (rows & 1u) w[0] = acc ? fadd(w[0], u.x) : u.x;
              if (rows & 2u) w[1] = acc ? fadd(w[1], u.y) : u.y;
              if (rows & 4u) w[2] = acc ? fadd(w[2], u.z) : u.z;
              if (rows & 8u) w[3] = acc ? fadd(w[3], u.w) : u.w;
              __syncwarp();
            }
          }
          // to the neighbours: the last column to the right, 0 and 1 to the left
          if (ot & (1u << k)) ll_store(hout + (j + k < 2 ? 1 + j + k : 0) * hcol, p, tag);
        };
        for (;;) {
          column(0, w0, w1, w2, w3);
          if (n == 1) break;
          column(1, w1, w2, w3, w0);
          if (n == 2) break;
          column(2, w2, w3, w0, w1);
          if (n == 3) break;
          column(3, w3, w0, w1, w2);
          if (n == 4) break;
          n -= 4;
          j += 4;
          f += 4 * FS;
          fu += 8 * FS;
          sp0 += 4;
          sp1 += 4;
          fd += 16 * FS;
          pp += 4 * 32;
          cf += 8;
          ed += 8;
          tp += 32;
          tk += 16;
          ho += 4 * hstep;
          if (!kParts) ev >>= 4;
          ot >>= 4;
          ph >>= 4;
          src >>= 4;
        }
      };
      if (!kParts) {
        for (int j = pj0, je = chi;;) {
          if (j < 2) put_left();
          columns(j, je);
          if (clo > 1 || je <= 2) break;
          j = clo;  // the left edge's columns
          je = 2;
        }
      } else {
#pragma unroll 1
      for (int part = chi > 2 ? 0 : 2; part < 3; ++part) {  // the columns between, C - 1, 0 and 1
        int j = pj0, je = kParts && rhalo ? C - 1 : chi;
        if (part == 1) {
          if (!kParts || !rhalo) continue;
          put_right();
          if (kB && (C - 1 - pj0) % HR) {  // the quads read ahead go on where they are
            const HT t = hq[0];
            hq[0] = hq[1];
            hq[1] = t;
          }
          j = C - 1;
          je = C;
        } else if (part == 2) {
          if (clo > 1) break;
          put_left();
          j = clo;
          je = min(chi, 2);
        }
        if (j < je) columns(j, je);
      }
      }
      tm_wait_st();
      if (kA) {
        const unsigned m = __reduce_max_sync(kAll, rows ? __float_as_uint(lmax) & 0x7fffffffu : 0u);
        if (lane == 0) atomicMax(&WM[0], m);
      }
      if (kB) {  // velocity histories of the first columns of the next half step
        const char *hbx = hist_at(slot_b(it), 1), *hbz = hist_at(slot_b(it), 2);
#pragma unroll
        for (int u = 0; u < HR; ++u) {
          hx[u] = ldh(hbx, vj0 + u, lphys);
          hz[u] = ldh(hbz, vj0 + u, lphys);
        }
      }
    } else if (aux) {
      if (kA && FP16 && it > first) exchange_v(it - 1);  // velocity maxima of the previous step
      if (!kB) {
        asm volatile("cp.async.wait_all;" ::: "memory");
        fetch_amp(it + 1);
      }
      if (kB) prefetch_b(it + 2);
    }
    if (extra) {
      rptr[0] += S.rect[0].step;
      rptr[1] += S.rect[1].step;
    }
    sync_cta();
    // =============== velocity half step ===============
    if (!kB && ipts > 0 && it < last && !aux) inj_terms(sm, l, ipts, im, amp(it), it0, itn);
    if (comp) {
      const Q4 d1b = lds4(ROW + 2 * NP), bw1 = lds4(ROW + 3 * NP);
      const u64 INVX = splat(kA && FP16 ? SC[1] : 1.f), INVZ = splat(kA && FP16 ? SC[2] : 1.f);
      const unsigned put = kA && it > first && rows ? 1u : 0u;
      char* const hpx = hist_at(kA ? max(it - 2, 0) : slot_b(it), 1);
      char* const hpz = hist_at(kA ? max(it - 2, 0) : slot_b(it), 2);
      const u64 SCX = splat(kB ? SC[(it & 1) * 3 + 1] : 1.f), SCZ = splat(kB ? SC[(it & 1) * 3 + 2] : 1.f);
      float lmx = 0.f, lmz = 0.f;
      ulonglong2* const hout = hmine + (size_t)(2 + (it & 1)) * hpar;  // phase 1: vx words
      const ulonglong2* const hin = hmine + (size_t)(it & 1) * hpar;   // p words
      auto pload = [&](int jj) {
        if (PS) return lds4(PP + 32 * jj);
        Q4 x, z;
        tm_ld(TP + 8 * jj, x, z);
        return add4(x, z);
      };
      // The warp's columns in order, column 0 last; the neighbours' words go into
      // the columns C, C + 1 and -1 of p.
      const bool rhalo = hasr && chi > C - 2, lhalo = hasl && ledge;
      const unsigned outs = (hasr ? 3u << (C - 2) : 0u) | (hasl ? 1u : 0u);
      auto put_p = [&](int c, Q4 v) {
        if (PS)
          sts4(PP + 32 * c, v);
        else
          tm_st(TP + 8 * c, v, kZero4);
      };
      auto put_right = [&]() {
        Q4 r[2];
        halo_get(hin + hcta + hcol, hcol, tag, poll, r, [] {});
        put_p(C, r[0]);
        put_p(C + 1, r[1]);
        if (!PS) tm_wait_st();
      };
      const unsigned wait = !kParts && rhalo && clo <= C - 2 ? 1u << (C - 2) : 0u;
      auto put_left = [&]() {
        auto histories = [&]() {  // of column 0
          if (!kB) return;
          hx[0] = ldh(hpx, 0, lphys);
          hz[0] = ldh(hpz, 0, lphys);
        };
        if (!lhalo) {
          histories();
          return;
        }
        Q4 h[1];
        halo_get(hin - hcta, hcol, tag, poll, h, histories);
        put_p(-1, h[0]);
        if (!PS) tm_wait_st();
      };
      // Columns [j, je), as in the pressure half step.
      auto columns = [&](int j, int je) {
        Q4* f = F + FS * j;
        const ulonglong2* cf = CF + 2 * j + 1;
        const Q4* pp = PP + 32 * (j + 2);
        const u64* ed = ED + 2 * j;
        unsigned tp = TP + 8 * (j + 2), ho = (unsigned)((hoff + j * n1h) * kEs);
        unsigned ev = wait >> j, ot = outs >> j, ph = phys >> j, src = lphys >> j;
        int n = je - j;
        Q4 w0 = pload(j - 1), w1 = pload(j), w2 = pload(j + 1), w3;
        auto column = [&](const int k, const Q4& w0, const Q4& w1, const Q4& w2, Q4& w3) {
          if (!kParts && (ev & (1u << k))) put_right();
          const float4 p = up4(w1);
          float pm1 = __shfl_up_sync(kAll, p.w, 1);
          float n0 = __shfl_down_sync(kAll, p.x, 1), n1 = __shfl_down_sync(kAll, p.y, 1);
          // the neighbouring blocks' pairs: last of the one above, first of the one below
          lds_if(pm1, reinterpret_cast<const float*>(ed + 2 * k + 1 - 2 * C) + 1, top);
          lds_if(n0, n1, reinterpret_cast<const float*>(ed + 2 * k + 2 * C), bottom);
          Q4 vx = lds4(f + FS * k), vz = lds4(f + FS * k + 32), qx, qz;
          const ulonglong2 c2 = cf[2 * k];
          if (PS) {
            w3 = lds4(pp + 32 * k);
          } else {
            tm_ld(tp + 8 * k, qx, qz);
            w3 = add4(qx, qz);
          }
          Q4 k2{c2.y, c2.y}, k1 = bw1, bu = kZero4;
          if (RHO) {
            const size_t o = (size_t)min(c0 + j + k, g.n2e - 1) * ld + min(i1, ld - 4);
            const ulonglong2 r2 = __ldg(reinterpret_cast<const ulonglong2*>(md.rbw2 + o));
            const ulonglong2 r1 = __ldg(reinterpret_cast<const ulonglong2*>(md.rbw1 + o));
            k2 = mul4(k2, Q4{r2.x, r2.y});
            k1 = mul4(k1, Q4{r1.x, r1.y});
            if (kB) {
              const ulonglong2 r = __ldg(reinterpret_cast<const ulonglong2*>(md.rbue + o));
              bu = {r.x, r.y};
            }
          }
          const Q4 der1 = add4(mul41(pk4(fsub(p.y, p.x), fsub(p.z, p.y), fsub(p.w, p.z), fsub(n0, p.w)), A0),
                               mul41(pk4(fsub(p.z, pm1), fsub(p.w, p.x), fsub(n0, p.y), fsub(n1, p.z)), A1));
          if (kA && (ph & (1u << k))) {
            Q4 x = mul41(vx, INVX), z = mul41(vz, INVZ);
            if (part) {
              x = keep(x, rows);
              z = keep(z, rows);
            }
            HQ::put(hpx + (ho + k * hstep), x, pol, put);
            HQ::put(hpz + (ho + k * hstep), z, pol, put);
          }
          const Q4 az = mul4(d1b, vz), bz = mul4(k1, der1);
          vz = kA ? sub4(az, bz) : add4(az, bz);
          const Q4 der2 = add4(mul41(sub4(w2, w1), A0), mul41(sub4(w3, w0), A1));
          const Q4 ax = mul41(vx, c2.x), bx = mul4(k2, der2);
          vx = kA ? sub4(ax, bx) : add4(ax, bx);
          if (kB) {  // outside the physical range: the term is 0 (history read as 0)
            Q4 tx = mul41(mul41(HQ::get(hx[k % HR]), SCX), MDT), tz = mul41(mul41(HQ::get(hz[k % HR]), SCZ), MDT);
            if (RHO) {
              tx = mul4(tx, bu);
              tz = mul4(tz, bu);
            }
            vx = add4(vx, tx);
            vz = add4(vz, tz);
            const unsigned on = src & (1u << (k + HR));
            hx[k % HR] = HQ::load(hpx + (ho + (k + HR) * hstep), on);
            hz[k % HR] = HQ::load(hpz + (ho + (k + HR) * hstep), on);
          }
          if (fs_warp) {
            float4 v = up4(vz);
            const float below = __shfl_down_sync(kAll, v.x, 1);
            if (fsk == 0) v.x = v.y;
            if (fsk == 1) v.y = v.z;
            if (fsk == 2) v.z = v.w;
            if (fsk == 3) v.w = below;
            vz = pk4(v.x, v.y, v.z, v.w);
          }
          sts4(f + FS * k, vx);
          sts4(f + FS * k + 32, vz);
          if (kA && (ph & (1u << k))) {
            lmx = amax(lmx, vx);
            lmz = amax(lmz, vz);
          }
          // to the neighbours: the last two columns to the right, 0 to the left
          if (ot & (1u << k)) ll_store(hout + (j + k ? j + k + 2 - C : 2) * hcol, vx, tag);
        };
        for (;;) {
          column(0, w0, w1, w2, w3);
          if (n == 1) break;
          column(1, w1, w2, w3, w0);
          if (n == 2) break;
          column(2, w2, w3, w0, w1);
          if (n == 3) break;
          column(3, w3, w0, w1, w2);
          if (n == 4) break;
          n -= 4;
          j += 4;
          f += 4 * FS;
          cf += 8;
          ed += 8;
          tp += 32;
          pp += 4 * 32;
          ho += 4 * hstep;
          if (!kParts) ev >>= 4;
          ot >>= 4;
          ph >>= 4;
          src >>= 4;
        }
      };
      if (!kParts) {
        for (int j = vj0, je = chi;;) {
          if (j == 0) put_left();
          if (j == C - 1 && rhalo) put_right();  // the warp's only column: p of column C before it starts
          columns(j, je);
          if (clo > 0 || je <= 1) break;
          j = 0;  // column 0
          je = 1;
        }
      } else {
#pragma unroll 1
      for (int part = ledge && chi == 1 ? 2 : 0; part < 3; ++part) {  // ..., C - 2 and C - 1, 0
        int j = vj0, je = kParts && rhalo ? C - 2 : chi;
        if (part == 1) {
          if (!kParts || !rhalo) continue;
          put_right();
          if (kB && vj0 < C - 2 && (C - 2 - vj0) % HR) {
            const HT tx = hx[0], tz = hz[0];
            hx[0] = hx[1];
            hz[0] = hz[1];
            hx[1] = tx;
            hz[1] = tz;
          }
          j = max(vj0, C - 2);
          je = chi;
        } else if (part == 2) {
          if (!ledge) break;
          put_left();
          j = 0;
          je = 1;
        }
        // the last column is the warp's only one: p of column C before it starts
        if (!kParts && rhalo && j == C - 1) put_right();
        if (j < je) columns(j, je);
      }
      }
      if (kA) {
        const unsigned mx = __reduce_max_sync(kAll, rows ? __float_as_uint(lmx) & 0x7fffffffu : 0u);
        const unsigned mz = __reduce_max_sync(kAll, rows ? __float_as_uint(lmz) & 0x7fffffffu : 0u);
        if (lane == 0) {
          atomicMax(&WM[1], mx);
          atomicMax(&WM[2], mz);
        }
      }
      if (kB && it < last) {
        const char* hn = hist_at(slot_b(it + 1), 0);
#pragma unroll
        for (int u = 0; u < HR; ++u) hq[u] = ldh(hn, pj0 + u, lsrc);
      }
    } else if (aux) {
      if (kA) {  // pressure maximum of this step
        const unsigned m = WM[0];
        __syncwarp();
        if (lane == 0) {
          WM[0] = 0;
          if (m >= 0x7f800000u) atomicOr(L.err, kErrNonFinite);
        }
        if (FP16) {
          if (lane == 0) word_store(words(0, it) + b, (u64)tag << 32 | m);
          exchange_p(it);
        }
      }
      if (staged) {
        const int c = c0 + lane;
        for (int q = 0; q < 2; ++q) {
          const ResidentRect& R = S.rect[q];
          if (!R.buf || lane >= C || c < R.c0 || c >= R.c1) continue;
          const float* v = reinterpret_cast<const float*>(stage + R.quad0 * C + lane);
          float* o = R.buf + (size_t)(it - first) * R.step + (c - R.c0);
#pragma unroll 4
          for (int r = R.r0; r < R.r1; ++r) {
            const int k = r - (R.r0 & ~3);
            o[(ptrdiff_t)(r - R.r0) * R.ld] = v[(k >> 2) * 4 * C + (k & 3)];
          }
        }
        __syncwarp();
      }
      if (kB && it < last) scales_b(it + 1);
    }
    sync_cta();
    if (kA && aux) {  // publish the velocity maxima of this step
      const unsigned x = WM[1], z = WM[2];
      __syncwarp();
      if (lane == 0) {
        WM[1] = WM[2] = 0;
        if (max(x, z) >= 0x7f800000u) atomicOr(L.err, kErrNonFinite);
        if (FP16) {
          word_store(words(1, it) + b, (u64)tag << 32 | x);
          word_store(words(1, it) + gridDim.x + b, (u64)tag << 32 | z);
        }
      }
      __syncwarp();
    }
  }

  // ---- the last step's histories
  if (kA) {
    if (aux && FP16) exchange_v(last);
    __syncthreads();
  }
  if (comp && (kA || L.save)) {
    const u64 ip = splat(kA && FP16 ? SC[0] : 1.f), ix = splat(kA && FP16 ? SC[1] : 1.f),
              iz = splat(kA && FP16 ? SC[2] : 1.f);
    for (int j = clo; j < chi; ++j) {
      Q4 px, pz;
      tm_ld(TP + 8 * j, px, pz);
      const Q4 vx = lds4(F + FS * j), vz = lds4(F + FS * j + 32);
      if (kA) {
        const unsigned on = lphys >> j & 1u;
        const ptrdiff_t o = (ptrdiff_t)(hoff + j * n1h) * kEs;
        HQ::put(hist_at(last - 1, 0) + o, keep(mul41(add4(px, pz), ip), rows), pol, on);
        HQ::put(hist_at(last - 1, 1) + o, keep(mul41(vx, ix), rows), pol, on);
        HQ::put(hist_at(last - 1, 2) + o, keep(mul41(vz, iz), rows), pol, on);
      }
      if (L.save && c0 + j < g.n2e && i1 < ld) {
        const size_t o = (size_t)(c0 + j) * ld + i1;
        sts4(reinterpret_cast<Q4*>(S.px + o), px);
        sts4(reinterpret_cast<Q4*>(S.pz + o), pz);
        sts4(reinterpret_cast<Q4*>(S.vx + o), vx);
        sts4(reinterpret_cast<Q4*>(S.vz + o), vz);
      }
      __syncwarp();
    }
  }
  sync_cta();
  if (warp == 0)
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(*TB), "r"(tcols));
}

// Injection tables: one CTA per grid CTA.
__global__ void k_resident_tables(const Grid g, const float* kap, const InjMapDev map, int C,
                                  const int4* head, int pts, int m, float* cd,
                                  unsigned short* sta, float* kp) {
  const int b = blockIdx.x;
  const int4 h = head[b];
  const int n = C * h.y;
  for (int p = threadIdx.x; p < n; p += blockDim.x) {
    const int j = p / h.y, r = h.x + p % h.y, c = b * C + j;
    const size_t o = (size_t)b * pts + p;
    int e0 = 0, e1 = 0;
    float kv = 0.f;
    if (c < g.n2e && r < g.n1e) {
      kv = kap[(size_t)c * g.ld + r];
      const int lo = map.col_lo[c], hi = map.col_hi[c];
      if (r >= lo && r <= hi) {
        const int q = map.col_base[c] + r - lo;
        e0 = map.rowptr[2 * q];
        e1 = map.rowptr[2 * q + 1];
      }
    }
    kp[o] = kv;
    for (int k = 0; k < m; ++k) {
      const bool in = e0 + k < e1;
      const float2 q = in ? map.ent[e0 + k] : make_float2(0.f, 0.f);
      cd[o * m + k] = in ? fmul(q.x, g.dt) : 0.f;
      sta[o * m + k] = in ? (unsigned short)(__float_as_int(q.y) - h.z) : (unsigned short)0xffff;
    }
  }
}

// Hicks sums from a rectangle buffer.  A warp takes 32 stations (lanes) and
// four steps at a time: each lane adds its station's products in the
// reference's order (i1 outer, i2 inner) in four independent chains.  The
// block's coefficients sit in shared memory, transposed.
constexpr int kGatherWarps = 8, kGatherSteps = 4;
__global__ void __launch_bounds__(32 * kGatherWarps)
    k_resident_gather(const ResidentRect r, const StationsDev st, int ra, int rb, int ca, int cb,
                      int nsteps, float* out, int nt, int row0, int reverse) {
  extern __shared__ float tl[];  // [441][33]
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int s0 = blockIdx.x * 32, s = s0 + lane;
  for (int k = threadIdx.x; k < 32 * kTile; k += blockDim.x) {
    const int q = k / kTile, t = k - q * kTile;
    tl[t * 33 + q] = s0 + q < st.n ? st.tile[(size_t)(s0 + q) * kTile + t] : 0.f;
  }
  __syncthreads();
  const bool on = s < st.n;
  // 0-based first tap of the station; support clipped to [ra, rb) x [ca, cb)
  const int a0 = on ? st.ix1[s] - 1 - kRad : 0, b0 = on ? st.ix2[s] - 1 - kRad : 0;
  const int alo = max(0, ra - a0), ahi = min(kTap, rb - a0);
  const bool allfull = __all_sync(kAll, (b0 >= ca && b0 + kTap <= cb) || !on);  // all columns
  for (int t0 = (blockIdx.y * kGatherWarps + warp) * kGatherSteps; t0 < nsteps;
       t0 += gridDim.y * kGatherWarps * kGatherSteps) {
    float acc[kGatherSteps] = {};
    const float* base[kGatherSteps];
#pragma unroll
    for (int k = 0; k < kGatherSteps; ++k)
      base[k] = r.buf + (size_t)min(t0 + k, nsteps - 1) * r.step;
    if (on) {
      if (allfull) {
        for (int a = alo; a < ahi; ++a) {
          const size_t o = (size_t)(a0 + a - r.r0) * r.ld + (b0 - r.c0);
#pragma unroll
          for (int q = 0; q < kTap; ++q) {
            const float c = tl[(a + kTap * q) * 33 + lane];
#pragma unroll
            for (int k = 0; k < kGatherSteps; ++k) acc[k] = fadd(acc[k], fmul(c, base[k][o + q]));
          }
        }
      } else {
        for (int a = alo; a < ahi; ++a)
          for (int q = max(0, ca - b0); q < kTap && b0 + q < cb; ++q) {
            const float c = tl[(a + kTap * q) * 33 + lane];
            const size_t o = (size_t)(a0 + a - r.r0) * r.ld + (b0 + q - r.c0);
#pragma unroll
            for (int k = 0; k < kGatherSteps; ++k) acc[k] = fadd(acc[k], fmul(c, base[k][o]));
          }
      }
#pragma unroll
      for (int k = 0; k < kGatherSteps; ++k)
        if (t0 + k < nsteps) {
          const int row = reverse ? row0 - (t0 + k) : row0 + t0 + k;
          out[row + (size_t)nt * s] = acc[k];
        }
    }
  }
}

template <typename F>
void with_kernel(int mode, bool fp16, bool rho, bool ps, F&& f) {
  auto pick = [&](auto m, auto h) {
    constexpr int M = decltype(m)::value;
    constexpr bool H = decltype(h)::value;
    constexpr bool P = M == FM_STAGE_B || (M == FM_STAGE_A && !H);  // the modes that have it
    if (ps && P)
      rho ? f(k_resident<M, H, true, P>) : f(k_resident<M, H, false, P>);
    else if (!ps)
      rho ? f(k_resident<M, H, true, false>) : f(k_resident<M, H, false, false>);
  };
  using std::false_type;
  using std::integral_constant;
  using std::true_type;
  if (mode == FM_FWD)
    pick(integral_constant<int, FM_FWD>{}, false_type{});
  else if (mode == FM_STAGE_A) {
    if (fp16)
      pick(integral_constant<int, FM_STAGE_A>{}, true_type{});
    else
      pick(integral_constant<int, FM_STAGE_A>{}, false_type{});
  } else {
    if (fp16)
      pick(integral_constant<int, FM_STAGE_B>{}, true_type{});
    else
      pick(integral_constant<int, FM_STAGE_B>{}, false_type{});
  }
}

constexpr size_t kMaxSmem = 227 * 1024;
constexpr int kTmCols = 512;

}  // namespace

void resident_groups(int C, int RB, bool ps, int* cg, int* cw) {
  const int w = group_warps(RB, ps);
  const int most = !ps && RB % 4 ? kResWarps / w : (kResWarps - 1) / w;
  *cg = std::max(1, std::min(most, C));
  *cw = (C + *cg - 1) / *cg;
  *cg = (C + *cw - 1) / *cw;
}

size_t resident_smem(int C, int RB, bool ps, int inj_pts, int inj_m, int inj_sta, int quads) {
  int cg, cw;
  resident_groups(C, RB, ps, &cg, &cw);
  if (tm_words(C, RB, cg, cw, ps) > kTmCols) return kMaxSmem + 1;
  // No more CTAs may be resident on an SM than its tensor memory holds: shared
  // memory is padded until it admits just as many (an allocation that does not
  // fit would block inside the kernel).
  const size_t n = kTmCols / tm_alloc(C, RB, cg, cw, ps);
  const size_t floor_bytes = kMaxSmem / (n + 1) + 128;
  return std::max((size_t)layout(C, RB, inj_pts, inj_m, inj_sta, quads, ps).total, floor_bytes);
}

int resident_occupancy(int mode, bool fp16, bool rho, bool ps, int C, int RB, size_t smem) {
  if (smem > kMaxSmem || RB > kResRowBlocks) return 0;
  int n = 0, cg, cw;  // n stays 0 for a mode without the variant
  resident_groups(C, RB, ps, &cg, &cw);
  with_kernel(mode, fp16, rho, ps, [&](auto k) {
    if (cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kMaxSmem) !=
            cudaSuccess ||
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, k, 32 * cta_warps(RB, cg, ps), smem) !=
            cudaSuccess) {
      cudaGetLastError();
      n = 0;
    }
  });
  return n;
}

cudaError_t resident_launch(const Grid& g, const ModelDev& m, const ResidentLaunch& L, int mode,
                            bool fp16, cudaStream_t st) {
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3(L.G * L.groups);
  ResidentLaunch P = L;
  P.nz = kNegZero2;
  resident_groups(L.C, L.RB, L.ps, &P.CG, &P.CW);
  cfg.blockDim = dim3(32 * cta_warps(L.RB, P.CG, L.ps));
  cfg.dynamicSmemBytes = resident_smem(L.C, L.RB, L.ps, L.inj_pts, L.inj_m, L.inj_sta, L.quads);
  cfg.stream = st;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeCooperative;  // CTAs wait on one another: all are resident
  at[0].val.cooperative = 1;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  cudaError_t e = cudaSuccess;
  with_kernel(mode, fp16, m.rbw1 != nullptr, L.ps,
              [&](auto k) { e = cudaLaunchKernelEx(&cfg, k, g, m, P); });
  return e;
}

void resident_tables(const Grid& g, const ModelDev& m, const InjMapDev& map, int C, int G,
                     const int4* head, int pts, int mm, float* cd, unsigned short* sta, float* kap,
                     cudaStream_t st) {
  k_resident_tables<<<G, 256, 0, st>>>(g, m.kap, map, C, head, pts, mm, cd, sta, kap);
}

void resident_gather(const Grid& g, const ResidentRect& r, const StationsDev& st, int off, int lo1,
                     int hi1, int lo2, int hi2, int nsteps, float* out, int nt, int row0, int reverse,
                     cudaStream_t s) {
  if (st.n <= 0 || nsteps <= 0) return;
  lo1 = std::max({lo1, 2, g.ofs == 1 ? g.npml + 1 : 0});
  lo2 = std::max(lo2, 2);
  hi1 = std::min(hi1, g.n1e - off);
  hi2 = std::min(hi2, g.n2e - off);
  constexpr size_t smem = kTile * 33 * sizeof(float);
  cudaFuncSetAttribute(k_resident_gather, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  const int per = kGatherWarps * kGatherSteps;
  const dim3 grid((st.n + 31) / 32, std::min((nsteps + per - 1) / per, 64));
  k_resident_gather<<<grid, 32 * kGatherWarps, smem, s>>>(r, st, lo1, hi1, lo2, hi2, nsteps,
                                                          out, nt, row0, reverse);
}

}  // namespace daw
