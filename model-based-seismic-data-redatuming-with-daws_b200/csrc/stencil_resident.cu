// Time loops on chip.
//
// One cooperative launch runs all steps of a time loop (or a long chunk of
// them) with the wavefield held on chip: a group of G CTAs owns one shot, CTA
// b the grid columns [b C, b C + C) over all rows.  A compute warp owns 64 rows of
// them, a lane two adjacent rows: px and pz of the lane's 2 x C points are in
// tensor memory (used as a scratchpad a warp reads and writes by column), vx, vz
// and kappa in shared memory.  What one step moves is then the history stream
// and three halo columns per CTA and half step, not the state.
//
// Halo columns go from lane to lane of neighbouring CTAs through L2: the
// writer stores (value, step tag) as one 64-bit word, so the reader's poll of
// the data is also the wait and no fence or flag follows it.  A lane needs its
// neighbour CTA's values of its own two rows only, and only for the first two
// and the last column; those columns are computed last in a half step, so the
// words travel while the columns between are computed.  Buffers alternate by
// step parity: a CTA writes parity s only after it has read its neighbours'
// words of step s - 1, which they store after their last read of step s - 2.
// Rows couple neighbouring warps (vz through shared memory, p through warp
// shuffles and an edge array), ordered by the CTA barrier after each half step.
//
// Stage A stores its FP16 histories with one scale per step and field, taken
// from the maximum over the whole grid.  An extra warp per CTA exchanges the
// CTAs' maxima through tagged words during the half step after a field is
// complete, and the history of step s is stored from the registers and shared
// memory in step s + 1, just before the values are updated (the last step's
// after the loop).
//
// Rows 0, 1 and the last rows and columns are never updated and the caller
// keeps sources away from them, so they stay zero: their update coefficients
// are set to zero instead of branching.
//
// Arithmetic: the reference's separately rounded FP32 operations, two rows at
// a time in packed (f32x2) instructions; bit-identical to the other kernels.
//
// Every wait is bounded: after its limit it raises kErrTimeout, and the other
// waits of the grid see the flag and stop waiting too.
//
// What bounds it: instruction issue (about 230 warp instructions per 64 points
// and step of stage A, 111 of them arithmetic or memory) for wide CTAs, the
// exchange latency (about 1.5 us per half step) for narrow ones.  The fields
// are not in registers because their columns must then be unrolled: that
// version ran out of the instruction cache (30 us against 14).
// Measured per shot step against the split kernels (B200, FP16 histories):
// 751 x 2301 (17 columns a CTA) forward 13.2 us against 20.1, stage A 14.0
// against 20.7-23.0, stage B 13.8 against 19.7-24.7; 151 x 461 (4 columns)
// 4.1-6.2 us against 12-15.
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

// (value, tag) words
__device__ __forceinline__ void ll_store(ulonglong2* p, u64 v, unsigned tag) {
  const float2 f = up(v);
  const u64 a = (u64)tag << 32 | __float_as_uint(f.x), b = (u64)tag << 32 | __float_as_uint(f.y);
  asm volatile("st.relaxed.gpu.global.v2.b64 [%0], {%1, %2};" ::"l"(p), "l"(a), "l"(b) : "memory");
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
  bool dead;
  __device__ __forceinline__ bool give_up(int n) {
    if ((n & 255) != 255) return false;
    unsigned e;
    asm volatile("ld.relaxed.gpu.global.u32 %0, [%1];" : "=r"(e) : "l"(err) : "memory");
    // one decision for the warp: its lanes may see the flag at different times
    dead = __any_sync(kAll, (e & kErrTimeout) != 0 || n > (1 << 22));
    if (dead && (threadIdx.x & 31) == 0) atomicOr(err, kErrTimeout);
    return dead;
  }
};

__device__ __forceinline__ u64 ll_wait1(const ulonglong2* p, unsigned tag, Poll& w) {
  ulonglong2 a = ll_load(p);
  for (int n = 0; !w.dead; ++n) {
    const bool ok = (unsigned)(a.x >> 32) == tag && (unsigned)(a.y >> 32) == tag;
    if (__all_sync(kAll, ok) || w.give_up(n)) break;
    a = ll_load(p);
  }
  return (a.y << 32) | (a.x & 0xffffffffu);
}
__device__ __forceinline__ void ll_wait2(const ulonglong2* p, const ulonglong2* q, unsigned tag,
                                         Poll& w, u64& vp, u64& vq) {
  ulonglong2 a = ll_load(p), b = ll_load(q);
  for (int n = 0; !w.dead; ++n) {
    const bool ok = (unsigned)(a.x >> 32) == tag && (unsigned)(a.y >> 32) == tag &&
                    (unsigned)(b.x >> 32) == tag && (unsigned)(b.y >> 32) == tag;
    if (__all_sync(kAll, ok) || w.give_up(n)) break;
    a = ll_load(p);
    b = ll_load(q);
  }
  vp = (a.y << 32) | (a.x & 0xffffffffu);
  vq = (b.y << 32) | (b.x & 0xffffffffu);
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

// A history row pair: FP16 in 32 bits, FP32 in 64.  Loads and stores are
// predicated (a load that is off gives 0), so that they cost no branch.
template <bool FP16>
struct HPair;
template <>
struct HPair<true> {
  typedef uint32_t T;
  static __device__ __forceinline__ T load(const char* p, unsigned on) {
    T v;
    asm volatile(
        "{\n .reg .pred p;\n setp.ne.u32 p, %2, 0;\n mov.b32 %0, 0;\n"
        " @p ld.global.nc.L1::no_allocate.b32 %0, [%1];\n}"
        : "=&r"(v)
        : "l"(p), "r"(on));
    return v;
  }
  static __device__ __forceinline__ u64 get(T v) {
    const float2 f = __half22float2(*reinterpret_cast<const __half2*>(&v));
    return pk(f.x, f.y);
  }
  static __device__ __forceinline__ void put(char* p, u64 v, uint64_t pol, unsigned on) {
    const float2 f = up(v);
    const __half2 q = __floats2half2_rn(f.x, f.y);
    asm volatile(
        "{\n .reg .pred p;\n setp.ne.u32 p, %3, 0;\n"
        " @p st.global.L2::cache_hint.b32 [%0], %1, %2;\n}" ::"l"(p),
        "r"(*reinterpret_cast<const uint32_t*>(&q)), "l"(pol), "r"(on)
        : "memory");
  }
  static __device__ __forceinline__ void put2(char* p, u64 v, char* p2, u64 v2, uint64_t pol,
                                              unsigned on) {
    const float2 f = up(v), f2 = up(v2);
    const __half2 q = __floats2half2_rn(f.x, f.y), q2 = __floats2half2_rn(f2.x, f2.y);
    asm volatile(
        "{\n .reg .pred p;\n setp.ne.u32 p, %5, 0;\n"
        " @p st.global.L2::cache_hint.b32 [%0], %1, %4;\n"
        " @p st.global.L2::cache_hint.b32 [%2], %3, %4;\n}" ::"l"(p),
        "r"(*reinterpret_cast<const uint32_t*>(&q)), "l"(p2),
        "r"(*reinterpret_cast<const uint32_t*>(&q2)), "l"(pol), "r"(on)
        : "memory");
  }
};
template <>
struct HPair<false> {
  typedef u64 T;
  static __device__ __forceinline__ T load(const char* p, unsigned on) {
    T v;
    asm volatile(
        "{\n .reg .pred p;\n setp.ne.u32 p, %2, 0;\n mov.b64 %0, 0;\n"
        " @p ld.global.nc.L1::no_allocate.b64 %0, [%1];\n}"
        : "=&l"(v)
        : "l"(p), "r"(on));
    return v;
  }
  static __device__ __forceinline__ u64 get(T v) { return v; }
  static __device__ __forceinline__ void put(char* p, u64 v, uint64_t pol, unsigned on) {
    asm volatile(
        "{\n .reg .pred p;\n setp.ne.u32 p, %3, 0;\n"
        " @p st.global.L2::cache_hint.b64 [%0], %1, %2;\n}" ::"l"(p),
        "l"(v), "l"(pol), "r"(on)
        : "memory");
  }
  static __device__ __forceinline__ void put2(char* p, u64 v, char* p2, u64 v2, uint64_t pol,
                                              unsigned on) {
    put(p, v, pol, on);
    put(p2, v2, pol, on);
  }
};

// Predicated shared-memory accesses.
__device__ __forceinline__ void sts_if(u64* p, u64 v, bool on) {
  asm volatile("{\n .reg .pred p;\n setp.ne.u32 p, %2, 0;\n @p st.shared.b64 [%0], %1;\n}" ::"r"(
                   smem_u32(p)),
               "l"(v), "r"((unsigned)on)
               : "memory");
}
__device__ __forceinline__ void lds_if(float& v, const float* p, bool on) {
  asm volatile("{\n .reg .pred p;\n setp.ne.u32 p, %2, 0;\n @p ld.shared.f32 %0, [%1];\n}"
               : "+f"(v)
               : "r"(smem_u32(p)), "r"((unsigned)on)
               : "memory");
}
__device__ __forceinline__ void lds_if(float& x, float& y, const float* p, bool on) {
  asm volatile("{\n .reg .pred p;\n setp.ne.u32 p, %3, 0;\n @p ld.shared.v2.f32 {%0, %1}, [%2];\n}"
               : "+f"(x), "+f"(y)
               : "r"(smem_u32(p)), "r"((unsigned)on)
               : "memory");
}

__device__ __forceinline__ void l2_prefetch(const void* p, unsigned bytes) {
  asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(p), "r"(bytes) : "memory");
}

// Tensor memory as a scratchpad: 32-bit columns of 32 lanes per warp quadrant.
// A warp reaches the lanes of its quadrant (warp % 4) only.
__device__ __forceinline__ void tm_ld4(unsigned a, unsigned (&r)[4]) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x4.b32 {%0, %1, %2, %3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
               : "r"(a));
}
// The loads' registers are read after this wait only (they are its operands).
__device__ __forceinline__ void tm_wait(unsigned (&r)[4]) {
  asm volatile("tcgen05.wait::ld.sync.aligned;"
               : "+r"(r[0]), "+r"(r[1]), "+r"(r[2]), "+r"(r[3])::"memory");
}
__device__ __forceinline__ void tm_st4(unsigned a, u64 x, u64 z) {
  asm volatile("tcgen05.st.sync.aligned.32x32b.x4.b32 [%0], {%1, %2, %3, %4};" ::"r"(a),
               "r"((unsigned)x), "r"((unsigned)(x >> 32)), "r"((unsigned)z), "r"((unsigned)(z >> 32))
               : "memory");
}
__device__ __forceinline__ void tm_wait_st() {
  asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ u64 pku(unsigned x, unsigned y) {
  return pk(__uint_as_float(x), __uint_as_float(y));
}

// Shared-memory layout (offsets in bytes, 16-byte aligned sections).
struct Lay {
  int fld, edge, col, row, tcd, term, tsta, tkap, amp, misc, total;
};
__host__ __device__ inline Lay layout(int C, int RB, int pts, int m, int nsta) {
  Lay l;
  int o = 0;
  auto take = [&](int bytes) {
    const int at = o;
    o += (bytes + 15) / 16 * 16;
    return at;
  };
  l.fld = take(RB * C * 768);        // [warp][column][vx, vz, kappa][lane]
  l.edge = take((RB + 2) * C * 16);  // [warp + 1][column][first, last pair of p]
  l.col = take(C * 32);              // [column][d2a, d2a, d2a1, d2a1, d2b, d2b, bw2, bw2]
  l.row = take(5 * RB * 32 * 8);
  l.tcd = take(pts * m * 4);
  l.term = take(pts * m * 4);
  l.tsta = take(pts * m * 2);
  l.tkap = take(pts * 4);
  l.amp = take((nsta + 1) * 4);
  l.misc = take(64 * 4 + 16);
  l.total = o;
  return l;
}
// Tensor-memory columns: px, pz (4 words a grid column and warp of the quadrant).
__host__ __device__ inline int tm_words(int C, int RB) { return (RB + 3) / 4 * C * 4; }
__host__ __device__ inline int tm_alloc(int C, int RB) {
  int n = 32;
  while (n < tm_words(C, RB)) n *= 2;
  return n;
}

// The injection terms ((c dt) amp) kappa of one step, by the compute warps.
__device__ __forceinline__ void inj_terms(unsigned char* sm, const Lay& l, int pts, int m,
                                          int nthreads) {
  const float2* cd = reinterpret_cast<const float2*>(sm + l.tcd);
  float2* term = reinterpret_cast<float2*>(sm + l.term);
  const ushort2* sta = reinterpret_cast<const ushort2*>(sm + l.tsta);
  const float* kap = reinterpret_cast<const float*>(sm + l.tkap);
  const float* amp = reinterpret_cast<const float*>(sm + l.amp);
  const int mh = m / 2;
  for (int p = threadIdx.x; p < pts; p += nthreads) {
    const float kv = kap[p];
    for (int k = 0; k < mh; ++k) {
      const float2 c = cd[p * mh + k];
      const ushort2 s = sta[p * mh + k];
      term[p * mh + k] = make_float2(fmul(fmul(c.x, amp[s.x]), kv), fmul(fmul(c.y, amp[s.y]), kv));
    }
  }
}

template <int MODE, bool FP16, bool RHO>
__global__ void __launch_bounds__(32 * (kResRowBlocks + 1), 1)
    k_resident(const __grid_constant__ Grid g, const __grid_constant__ ModelDev md,
               const __grid_constant__ ResidentLaunch L) {
  constexpr bool kA = MODE == FM_STAGE_A, kB = MODE == FM_STAGE_B, kF = MODE == FM_FWD;
  constexpr int U = 4;  // columns per loop iteration
  using HP = HPair<FP16>;
  using HT = typename HP::T;
  extern __shared__ __align__(16) unsigned char sm[];
  const int C = L.C, G = L.G, RB = L.RB;
  const Lay l = layout(C, RB, L.inj_pts, L.inj_m, L.inj_sta);
  const int grp = blockIdx.x / G, b = blockIdx.x - grp * G;
  const ResidentShot& S = L.shot[grp];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int ncomp = RB * 32;            // compute threads
  const bool aux = warp == RB;          // the extra warp
  const int c0 = b * C, i1 = 64 * warp + 2 * lane;
  const int npml = g.npml, ld = g.ld;
  const int first = S.first, last = S.last;
  if (first > last) return;             // uniform over the group
  // the lane's vx, vz, kappa of column j: F[96 j], F[96 j + 32], F[96 j + 64];
  // the vz pairs above and below it at FU, FD (lanes 0 and 31: in the
  // neighbouring warps' areas; the grid's first and last pair, which are never
  // updated, stand for the zeros beyond them)
  u64* const F = reinterpret_cast<u64*>(sm + l.fld) + warp * C * 96 + lane;
  const u64* const FU = F + 32 + (lane > 0 ? -1 : warp > 0 ? 31 - C * 96 : 0);
  const u64* const FD = F + 32 + (lane < 31 ? 1 : warp < RB - 1 ? C * 96 - 31 : 0);
  u64* const ED = reinterpret_cast<u64*>(sm + l.edge) + (warp + 1) * C * 2;
  u64* const EDL = ED + (lane == 31);  // where lanes 0 and 31 put their pairs
  const bool edge_lane = lane == 0 || lane == 31;
  ulonglong2* const CF = reinterpret_cast<ulonglong2*>(sm + l.col);
  u64* const ROW = reinterpret_cast<u64*>(sm + l.row);
  float* const TERM = reinterpret_cast<float*>(sm + l.term);
  float* const AMP = reinterpret_cast<float*>(sm + l.amp);
  unsigned* const WM = reinterpret_cast<unsigned*>(sm + l.misc);       // [3][16] warp maxima
  float* const SC = reinterpret_cast<float*>(sm + l.misc + 48 * 4);    // scales
  unsigned* const TB = reinterpret_cast<unsigned*>(sm + l.misc + 64 * 4);
  const int own = 32 * warp + lane;
  const int NP = RB * 32;
  Poll poll{L.err, false};
  const int4 ih = S.inj.pts > 0 ? S.inj.head[b] : make_int4(0, 0, 0, 0);
  const int ipts = ih.y > 0 ? C * ih.y : 0;
  const int im = L.inj_m;

  // ---- set-up
  const unsigned tcols = (unsigned)tm_alloc(C, RB);
  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                     smem_u32(TB)),
                 "r"(tcols)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const unsigned tbase = *TB + ((unsigned)(warp & 3) << 21);  // lane 32 (warp % 4)
  const unsigned TP = tbase + (warp >> 2) * C * 4;            // px, pz of column j: + 4 j
  {
    const int off = kF ? 2 : 3;
    const int hi1 = g.n1e - off, hi2 = g.n2e - off;
    for (int j = tid; j < C; j += blockDim.x) {
      const int c = c0 + j;
      const bool in = c < g.n2e, u = c >= 2 && c < hi2;
      const float4 q = in ? md.pcol[c] : make_float4(0.f, 0.f, 0.f, 0.f);
      CF[2 * j] = make_ulonglong2(pk(q.x, q.x), u ? pk(q.y, q.y) : 0ull);
      const float w = RHO ? 1.f : q.w;
      CF[2 * j + 1] = make_ulonglong2(pk(q.z, q.z), u ? pk(w, w) : 0ull);
    }
    if (!aux) {
      const bool u0 = i1 >= 2 && i1 < hi1, u1 = i1 + 1 >= 2 && i1 + 1 < hi1;
      const float4 z4 = make_float4(0.f, 0.f, 0.f, 0.f);
      const float4 a = i1 < g.n1e ? md.prow[i1] : z4, c = i1 + 1 < g.n1e ? md.prow[i1 + 1] : z4;
      ROW[own] = pk(a.x, c.x);
      ROW[NP + own] = pk(u0 ? a.y : 0.f, u1 ? c.y : 0.f);
      ROW[2 * NP + own] = pk(a.z, c.z);
      ROW[3 * NP + own] = pk(u0 ? (RHO ? 1.f : a.w) : 0.f, u1 ? (RHO ? 1.f : c.w) : 0.f);
      const int fsrows = g.ofs == 1 ? npml + 1 : 0;
      ROW[4 * NP + own] = pk(i1 < fsrows ? 0.f : 1.f, i1 + 1 < fsrows ? 0.f : 1.f);
      for (int j = 0; j < C; ++j) {
        const int c = c0 + j;
        u64 x = 0ull, z = 0ull, k = 0ull, px = 0ull, pz = 0ull;
        if (c < g.n2e) {
          const size_t o = (size_t)c * ld + i1;
          k = *reinterpret_cast<const u64*>(md.kap + o);
          if (L.load) {
            x = *reinterpret_cast<const u64*>(S.vx + o);
            z = *reinterpret_cast<const u64*>(S.vz + o);
            px = *reinterpret_cast<const u64*>(S.px + o);
            pz = *reinterpret_cast<const u64*>(S.pz + o);
          }
        }
        F[96 * j] = x;
        F[96 * j + 32] = z;
        F[96 * j + 64] = k;
        tm_st4(TP + 4 * j, px, pz);
      }
      tm_wait_st();
    }
    for (int k = tid; k < C * 2 * (RB + 2); k += blockDim.x)
      reinterpret_cast<u64*>(sm + l.edge)[k] = 0ull;
    if (tid < 48) WM[tid] = 0u;
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
      for (int k = tid; k < ipts; k += blockDim.x) tk[k] = S.inj.kap[o + k];
      for (int k = tid; k <= ih.w; k += blockDim.x)
        AMP[k] = k < ih.w ? S.amp[(size_t)(first - 1) * S.nsta + ih.z + k] : 0.f;
    }
  }
  __syncthreads();
  if (ipts > 0 && !aux) inj_terms(sm, l, ipts, im, ncomp);

  const u64 nz = L.nz;
  auto mul2 = [&](u64 x, u64 y) { return fma2(x, y, nz); };
  // ---- per-lane constants
  const bool r0 = i1 >= npml && i1 < npml + g.n1, r1 = i1 + 1 >= npml && i1 + 1 < npml + g.n1;
  const bool r01 = (r0 || r1) && !aux;
  const unsigned m0 = r0 ? 0x7fffffffu : 0u, m1 = r1 ? 0x7fffffffu : 0u;
  const int jlo = max(0, npml - c0), jhi = min(C, npml + g.n2 - c0);  // physical columns [jlo, jhi)
  const unsigned phys = jhi > jlo ? (1u << jhi) - (1u << jlo) : 0u;
  const unsigned lphys = r01 ? phys : 0u;  // of lanes with a physical row
  const int n1h = L.n1h;
  const size_t nih = (size_t)n1h * g.n2;
  const int hoff = i1 - g.hist_base() + n1h * (c0 - npml);  // history offset of column 0
  constexpr int kEs = FP16 ? 2 : 4;
  auto hist_at = [&](int slot, int f) {
    return static_cast<char*>(S.hist) + (((size_t)slot * 3 + f) * nih + hoff) * kEs;
  };
  const int hstep = n1h * kEs;  // bytes from one column's pair to the next
  const u64 A0 = pk(kA0, kA0), A1 = pk(kA1, kA1), DTDX = pk(g.dtdx, g.dtdx);
  const float mdt = fmul(-1.0f, g.dt);
  const u64 MDT = pk(mdt, mdt);
  const uint64_t pol = l2_evict_first();
  // halo words: [phase][parity][cta][3][NP]
  const size_t hcta = (size_t)3 * NP, hpar = hcta * gridDim.x;
  ulonglong2* const hmine = L.halo + (size_t)blockIdx.x * hcta + own;
  const bool hasl = b > 0, hasr = b + 1 < G;
  const bool inj_on = ipts > 0 && !aux && i1 + 1 >= ih.x && i1 < ih.x + ih.y;
  const bool inj_warp = ipts > 0 && !aux && 64 * warp + 63 >= ih.x && 64 * warp < ih.x + ih.y;
  // rectangles kept for the gathers
  bool rect_warp = false;
#pragma unroll
  for (int q = 0; q < 2; ++q)
    rect_warp |= !kA && S.rect[q].buf && 64 * warp + 63 >= S.rect[q].r0 && 64 * warp < S.rect[q].r1;
  const bool extra = !kA && !aux && (rect_warp || S.wf != nullptr);  // warp-uniform
  // free-surface copy vz(npml - 1) = vz(npml)
  const bool fs_warp = g.ofs == 1 && (npml - 1) / 64 == warp;
  const int slo = L.slo, shi1 = g.n1 - L.slo;
  const int sjlo = max(0, npml + slo - c0), sjhi = min(C, npml + g.n2 - slo - c0);
  const unsigned srcs = sjhi > sjlo ? (1u << sjhi) - (1u << sjlo) : 0u;  // source columns
  const unsigned lsrc = r01 ? srcs : 0u;
  const bool s0 = r0 && i1 - npml >= slo && i1 - npml < shi1;
  const bool s1 = r1 && i1 + 1 - npml >= slo && i1 + 1 - npml < shi1;
  HT hq[U] = {}, hx[U] = {}, hz[U] = {};  // stage B: history pairs read ahead
  auto slot_b = [&](int it) { return S.nt - it - L.hist_step0; };  // the time-reversed step's
  auto ldh = [&](const char* base, int j, unsigned mask) -> HT {
    return HP::load(base + (ptrdiff_t)j * hstep, mask >> j & 1u);
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
  if (kB) {
    if (aux) {
      scales_b(first);
      prefetch_b(first + 1);
    } else {
#pragma unroll
      for (int u = 0; u < U; ++u) hq[u] = ldh(hist_at(slot_b(first), 0), 2 + u, lsrc);
    }
  }
  const u64 fsm = aux ? 0ull : ROW[4 * NP + own];
  __syncthreads();

  for (int it = first; it <= last; ++it) {
    const unsigned tag = L.tag0 + (unsigned)it;
    // =============== pressure half step ===============
    if (!aux) {
      const u64 d1a = ROW[own], d1a1 = ROW[NP + own];
      const float inv = kA && FP16 ? SC[0] : 1.f;
      const u64 INV = pk(r0 ? inv : 0.f, r1 ? inv : 0.f);
      const unsigned putm = kA && it > first ? 0xffffffffu : 0u;
      char* const hp = hist_at(kA ? max(it - 2, 0) : slot_b(it), 0);
      const float scp = kB ? SC[(it & 1) * 3] : 1.f;
      const u64 SCP = pk(s0 ? scp : 0.f, s1 ? scp : 0.f);
      unsigned lmax = 0;
      ulonglong2* const hout = hmine + (size_t)(it & 1) * hpar;  // phase 0: p words
      // One column j, its arrays at f, fu, fd, cf, ed, tp, hb: qm2 .. qp1 are
      // vx of columns j-2 .. j+1, h the history pair, `on` whether this lane has
      // physical points of the column.
      auto column = [&](int j, u64* f, const u64* fu, const u64* fd, const ulonglong2* cfp, u64* ed,
                        unsigned tp, char* hb, unsigned on, u64 qm2, u64 qm1, u64 q0, u64 qp1,
                        HT h) {
        unsigned t4[4];
        tm_ld4(tp, t4);
        const float2 z = up(f[32]), zm = up(*fu);
        const float zp2 = *reinterpret_cast<const float*>(fd);
        const u64 kap = f[64];
        const ulonglong2 cf = *cfp;
        const u64 der2 = add2(mul2(A0, sub2(q0, qm1)), mul2(A1, sub2(qp1, qm2)));
        const u64 der1 = add2(mul2(A0, pk(fsub(z.x, zm.y), fsub(z.y, z.x))),
                              mul2(A1, pk(fsub(z.y, zm.x), fsub(zp2, zm.y))));
        const u64 kd = mul2(DTDX, kap);
        const u64 bx = mul2(mul2(kd, cf.y), der2), bz = mul2(mul2(kd, d1a1), der1);
        tm_wait(t4);
        u64 px = pku(t4[0], t4[1]), pz = pku(t4[2], t4[3]);
        if (kA)  // history of the previous step's pressure
          HP::put(hb, mul2(mul2(fsm, add2(px, pz)), INV), pol, on & putm);
        const u64 ax = mul2(cf.x, px), az = mul2(d1a, pz);
        px = kA ? sub2(ax, bx) : add2(ax, bx);
        pz = kA ? sub2(az, bz) : add2(az, bz);
        if (!kB && inj_warp) {
          if (inj_on) {
            const float2* t =
                reinterpret_cast<const float2*>(TERM + (size_t)(j * ih.y + (i1 - ih.x)) * im);
            float2 v = up(px);
            for (int k = 0; k < im / 2; ++k) {
              const float2 t0 = t[k], t1 = t[im / 2 + k];
              v.x = kA ? fsub(fsub(v.x, t0.x), t0.y) : fadd(fadd(v.x, t0.x), t0.y);
              v.y = kA ? fsub(fsub(v.y, t1.x), t1.y) : fadd(fadd(v.y, t1.x), t1.y);
            }
            px = pk(v.x, v.y);
          }
          __syncwarp();
        }
        // lanes outside the source range have a zero scale or read no history
        if (kB) px = add2(px, mul2(mul2(MDT, mul2(HP::get(h), SCP)), kap));
        tm_st4(tp, px, pz);
        const u64 p = mul2(fsm, add2(px, pz));
        sts_if(ed, p, edge_lane);
        if (kA) {
          const float2 pv = up(p);
          if (on) lmax = max(lmax, max(__float_as_uint(pv.x) & m0, __float_as_uint(pv.y) & m1));
        }
        return p;
      };
      auto column_at = [&](int j, u64 qm2, u64 qm1, u64 q0, u64 qp1, HT h) {
        return column(j, F + 96 * j, FU + 96 * j, FD + 96 * j, CF + 2 * j, EDL + 2 * j, TP + 4 * j,
                      hp + (ptrdiff_t)j * hstep, lphys >> j & 1u, qm2, qm1, q0, qp1, h);
      };
      // columns 2 .. C-2, U at a time, then one by one
      u64 q[U + 3];
      q[0] = F[0];
      q[1] = F[96];
      q[2] = F[192];
      {
        u64* f = F + 192;
        const u64 *fu = FU + 192, *fd = FD + 192;
        const ulonglong2* cf = CF + 4;
        u64* ed = EDL + 4;
        unsigned tp = TP + 8, on = (kB ? lsrc : lphys) >> 2;
        char* hb = hp + 2 * (ptrdiff_t)hstep;
        int j = 2;
        for (; j + U <= C - 1; j += U) {
#pragma unroll
          for (int u = 0; u < U; ++u) {
            q[u + 3] = f[96 * (u + 1)];
            column(j + u, f + 96 * u, fu + 96 * u, fd + 96 * u, cf + 2 * u, ed + 2 * u, tp + 4 * u, hb,
                   on & (1u << u), q[u], q[u + 1], q[u + 2], q[u + 3], hq[u]);
            if (kA) hb += hstep;
            // source columns beyond C - 1 have no bit
            if (kB) hq[u] = HP::load(hb + (ptrdiff_t)(u + U) * hstep, on & (1u << (u + U)));
          }
          q[0] = q[U];
          q[1] = q[U + 1];
          q[2] = q[U + 2];
          f += 96 * U;
          fu += 96 * U;
          fd += 96 * U;
          cf += 2 * U;
          ed += 2 * U;
          tp += 4 * U;
          on >>= U;
          if (kB) hb += (ptrdiff_t)U * hstep;
        }
#pragma unroll 1
        for (; j < C - 1; ++j) {
          const u64 qn = f[96];
          column(j, f, fu, fd, cf, ed, tp, hb, on & 1u, q[0], q[1], q[2], qn, hq[0]);
          q[0] = q[1];
          q[1] = q[2];
          q[2] = qn;
          hq[0] = hq[1];
          hq[1] = hq[2];
          f += 96;
          fu += 96;
          fd += 96;
          cf += 2;
          ed += 2;
          tp += 4;
          on >>= 1;
          hb += hstep;
        }
      }
      // the last column, with the right neighbour's first
      HT he[3] = {};
      if (kB) {
        he[0] = ldh(hp, C - 1, lsrc);
        he[1] = ldh(hp, 0, lsrc);
        he[2] = ldh(hp, 1, lsrc);
      }
      u64 qd = 0ull;
      if (hasr) {
        if (it == first) {
          const int c = c0 + C;
          if (L.load && c < g.n2e) qd = *reinterpret_cast<const u64*>(S.vx + (size_t)c * ld + i1);
        } else {
          qd = ll_wait1(hmine + (size_t)(2 + ((it - 1) & 1)) * hpar + hcta + 2 * NP, tag - 1, poll);
        }
      }
      const u64 pe = column_at(C - 1, q[0], q[1], q[2], qd, he[0]);
      if (hasr) ll_store(hout, pe, tag);
      // columns 0 and 1, with the left neighbour's last two
      u64 ha = 0ull, hb = 0ull;
      if (hasl) {
        if (it == first) {
          if (L.load) {
            ha = *reinterpret_cast<const u64*>(S.vx + (size_t)(c0 - 2) * ld + i1);
            hb = *reinterpret_cast<const u64*>(S.vx + (size_t)(c0 - 1) * ld + i1);
          }
        } else {
          const ulonglong2* h = hmine + (size_t)(2 + ((it - 1) & 1)) * hpar - hcta;
          ll_wait2(h, h + NP, tag - 1, poll, ha, hb);
        }
      }
      const u64 qa = F[0], qb = F[96], qc = F[192];
      const u64 p0 = column_at(0, ha, hb, qa, qb, he[1]);
      if (hasl) ll_store(hout + NP, p0, tag);
      const u64 p1 = column_at(1, hb, qa, qb, qc, he[2]);
      if (hasl) ll_store(hout + 2 * NP, p1, tag);
      tm_wait_st();
      if (kA) {
        lmax = __reduce_max_sync(kAll, lmax);
        if (lane == 0) WM[warp] = lmax;
      }
      if (kB) {  // velocity histories of the first columns of the next half step
        const char *hbx = hist_at(slot_b(it), 1), *hbz = hist_at(slot_b(it), 2);
#pragma unroll
        for (int u = 0; u < U; ++u) {
          hx[u] = ldh(hbx, 1 + u, lphys);
          hz[u] = ldh(hbz, 1 + u, lphys);
        }
      }
      if (extra) {
        // pressure rows of the gather rectangles, and the wavefield output
        for (int j = 0; j < C; ++j) {
          unsigned t4[4];
          tm_ld4(TP + 4 * j, t4);
          tm_wait(t4);
          const float2 pv = up(mul2(fsm, add2(pku(t4[0], t4[1]), pku(t4[2], t4[3]))));
          const int c = c0 + j;
#pragma unroll
          for (int q2 = 0; q2 < 2; ++q2) {
            const ResidentRect& R = S.rect[q2];
            if (R.buf && c >= R.c0 && c < R.c1) {
              float* o2 = R.buf + (size_t)(it - first) * R.step + (ptrdiff_t)(i1 - R.r0) * R.ld + (c - R.c0);
              if (i1 >= R.r0 && i1 < R.r1) o2[0] = pv.x;
              if (i1 + 1 >= R.r0 && i1 + 1 < R.r1) o2[R.ld] = pv.y;
            }
          }
          if (S.wf && (phys >> j & 1u)) {
            float* w = S.wf + (size_t)(it - 1) * g.int_elems() + (size_t)g.n1 * (c - npml) + (i1 - npml);
            if (r0) w[0] = S.wf_acc ? fadd(w[0], pv.x) : pv.x;
            if (r1) w[1] = S.wf_acc ? fadd(w[1], pv.y) : pv.y;
          }
          __syncwarp();
        }
      }
    } else {
      if (!kB && ipts > 0 && it < last)  // amplitudes of the next step
        for (int k = lane; k < ih.w; k += 32) AMP[k] = S.amp[(size_t)it * S.nsta + ih.z + k];
      if (kA && it > first) {            // velocity maxima of the previous step
        if (FP16) {
          u64* sl = L.slots + (size_t)(4 + ((it - 1) & 1) * 2) * gridDim.x + grp * G;
          const unsigned vx = group_max(sl, G, tag - 1, poll);
          const unsigned vz = group_max(sl + gridDim.x, G, tag - 1, poll);
          if (lane == 0) {
            SC[1] = pow2f(15 - amax_exponent(vx));
            SC[2] = pow2f(15 - amax_exponent(vz));
            if (b == 0) {
              unsigned* am = S.amax + (size_t)(it - 2) * 3 * kAmaxSlots;
              am[kAmaxSlots] = vx;
              am[2 * kAmaxSlots] = vz;
            }
          }
        }
      }
      if (kB) prefetch_b(it + 2);
    }
    __syncthreads();
    // =============== velocity half step ===============
    if (!aux) {
      if (!kB && ipts > 0 && it < last) inj_terms(sm, l, ipts, im, ncomp);
      const u64 d1b = ROW[2 * NP + own], bw1 = ROW[3 * NP + own];
      const float ix = kA && FP16 ? SC[1] : 1.f, iz = kA && FP16 ? SC[2] : 1.f;
      const u64 INVX = pk(r0 ? ix : 0.f, r1 ? ix : 0.f), INVZ = pk(r0 ? iz : 0.f, r1 ? iz : 0.f);
      const unsigned putm = kA && it > first ? 0xffffffffu : 0u;
      char* const hpx = hist_at(kA ? max(it - 2, 0) : slot_b(it), 1);
      char* const hpz = hist_at(kA ? max(it - 2, 0) : slot_b(it), 2);
      const float sx = kB ? SC[(it & 1) * 3 + 1] : 1.f, sz = kB ? SC[(it & 1) * 3 + 2] : 1.f;
      const u64 SCX = pk(r0 ? sx : 0.f, r1 ? sx : 0.f), SCZ = pk(r0 ? sz : 0.f, r1 ? sz : 0.f);
      unsigned lmx = 0, lmz = 0;
      ulonglong2* const hout = hmine + (size_t)(2 + (it & 1)) * hpar;  // phase 1: vx words
      auto pcol = [&](unsigned (&t4)[4]) { return mul2(fsm, add2(pku(t4[0], t4[1]), pku(t4[2], t4[3]))); };
      auto pload = [&](int j) {
        unsigned t4[4];
        tm_ld4(TP + 4 * j, t4);
        tm_wait(t4);
        return pcol(t4);
      };
      // One column j, its arrays at f, cf, ed, hbx, hbz: pm .. p2 are p of
      // columns j-1 .. j+2 (p2 read from the tensor memory here when tp != 0).
      auto column = [&](int j, u64* f, const ulonglong2* cfp, const u64* ed, unsigned tp, char* hbx,
                        char* hbz, unsigned on, u64 pm, u64 p0, u64 p1, u64& p2, HT hvx, HT hvz) {
        unsigned t4[4];
        if (tp) tm_ld4(tp, t4);
        const float2 p = up(p0);
        float pm1 = __shfl_up_sync(kAll, p.y, 1);
        float ppx = __shfl_down_sync(kAll, p.x, 1), ppy = __shfl_down_sync(kAll, p.y, 1);
        // the neighbouring warps' pairs: last of the warp above, first of the warp below
        lds_if(pm1, reinterpret_cast<const float*>(ed - 2 * C + 1) + 1, lane == 0);
        lds_if(ppx, ppy, reinterpret_cast<const float*>(ed + 2 * C), lane == 31);
        u64 vx = f[0], vz = f[32];
        const ulonglong2 cf = *cfp;
        const u64 der1 = add2(mul2(A0, pk(fsub(p.y, p.x), fsub(ppx, p.y))),
                              mul2(A1, pk(fsub(ppx, pm1), fsub(ppy, p.x))));
        if (kA) HP::put2(hbx, mul2(vx, INVX), hbz, mul2(vz, INVZ), pol, on & putm);
        u64 w2 = cf.y, w1 = bw1;
        u64 bu = 0ull;
        if (RHO) {
          const size_t k = (size_t)min(c0 + j, g.n2e - 1) * ld + i1;
          w2 = mul2(w2, __ldg(reinterpret_cast<const u64*>(md.rbw2 + k)));
          w1 = mul2(w1, __ldg(reinterpret_cast<const u64*>(md.rbw1 + k)));
          if (kB) bu = __ldg(reinterpret_cast<const u64*>(md.rbue + k));
        }
        const u64 az = mul2(d1b, vz), bz = mul2(w1, der1);
        vz = kA ? sub2(az, bz) : add2(az, bz);
        if (tp) {
          tm_wait(t4);
          p2 = pcol(t4);
        }
        const u64 der2 = add2(mul2(A0, sub2(p1, p0)), mul2(A1, sub2(p2, pm)));
        const u64 ax = mul2(cf.x, vx), bx = mul2(w2, der2);
        vx = kA ? sub2(ax, bx) : add2(ax, bx);
        if (kB) {  // outside the physical range: the term is 0 (history read as 0)
          u64 tx = mul2(MDT, mul2(HP::get(hvx), SCX)), tz = mul2(MDT, mul2(HP::get(hvz), SCZ));
          if (RHO) {
            tx = mul2(tx, bu);
            tz = mul2(tz, bu);
          }
          vx = add2(vx, tx);
          vz = add2(vz, tz);
        }
        if (fs_warp) {
          float2 v = up(vz);
          const float below = __shfl_down_sync(kAll, v.x, 1);
          if (i1 == npml - 1) v.x = v.y;
          if (i1 + 1 == npml - 1) v.y = below;
          vz = pk(v.x, v.y);
        }
        f[0] = vx;
        f[32] = vz;
        if (kA) {
          const float2 x = up(vx), z = up(vz);
          if (on) {
            lmx = max(lmx, max(__float_as_uint(x.x) & m0, __float_as_uint(x.y) & m1));
            lmz = max(lmz, max(__float_as_uint(z.x) & m0, __float_as_uint(z.y) & m1));
          }
        }
        return vx;
      };
      auto column_at = [&](int j, u64 pm, u64 p0, u64 p1, u64 p2, HT hvx, HT hvz) {
        return column(j, F + 96 * j, CF + 2 * j + 1, ED + 2 * j, 0u, hpx + (ptrdiff_t)j * hstep,
                      hpz + (ptrdiff_t)j * hstep, lphys >> j & 1u, pm, p0, p1, p2, hvx, hvz);
      };
      const u64 P0 = pload(0), P1 = pload(1), P2 = pload(2);
      // columns 1 .. C-3, U at a time, then one by one
      u64 q[U + 3];
      q[0] = P0;
      q[1] = P1;
      q[2] = P2;
      {
        u64* f = F + 96;
        const ulonglong2* cf = CF + 3;
        const u64* ed = ED + 2;
        unsigned tp = TP + 12, on = lphys >> 1;
        char *hbx = hpx + hstep, *hbz = hpz + hstep;
        int j = 1;
        for (; j + U <= C - 2; j += U) {
#pragma unroll
          for (int u = 0; u < U; ++u) {
            column(j + u, f + 96 * u, cf + 2 * u, ed + 2 * u, tp + 4 * u, hbx, hbz, on & (1u << u),
                   q[u], q[u + 1], q[u + 2], q[u + 3], hx[u], hz[u]);
            if (kA) {
              hbx += hstep;
              hbz += hstep;
            }
            if (kB) {
              hx[u] = HP::load(hbx + (ptrdiff_t)(u + U) * hstep, on & (1u << (u + U)));
              hz[u] = HP::load(hbz + (ptrdiff_t)(u + U) * hstep, on & (1u << (u + U)));
            }
          }
          q[0] = q[U];
          q[1] = q[U + 1];
          q[2] = q[U + 2];
          f += 96 * U;
          cf += 2 * U;
          ed += 2 * U;
          tp += 4 * U;
          on >>= U;
          if (kB) {
            hbx += (ptrdiff_t)U * hstep;
            hbz += (ptrdiff_t)U * hstep;
          }
        }
#pragma unroll 1
        for (; j < C - 2; ++j) {
          column(j, f, cf, ed, tp, hbx, hbz, on & 1u, q[0], q[1], q[2], q[3], hx[0], hz[0]);
          q[0] = q[1];
          q[1] = q[2];
          q[2] = q[3];
          hx[0] = hx[1];
          hx[1] = hx[2];
          hz[0] = hz[1];
          hz[1] = hz[2];
          f += 96;
          cf += 2;
          ed += 2;
          tp += 4;
          on >>= 1;
          hbx += hstep;
          hbz += hstep;
        }
      }
      HT ex[3] = {}, ez[3] = {};
      if (kB) {
        ex[0] = ldh(hpx, C - 2, lphys);
        ez[0] = ldh(hpz, C - 2, lphys);
        ex[1] = ldh(hpx, C - 1, lphys);
        ez[1] = ldh(hpz, C - 1, lphys);
        ex[2] = ldh(hpx, 0, lphys);
        ez[2] = ldh(hpz, 0, lphys);
      }
      // the last two columns, with the right neighbour's first two
      u64 ra = 0ull, rb = 0ull;
      if (hasr) {
        const ulonglong2* h = hmine + (size_t)(it & 1) * hpar + hcta;
        ll_wait2(h + NP, h + 2 * NP, tag, poll, ra, rb);
      }
      const u64 ve = column_at(C - 2, q[0], q[1], q[2], ra, ex[0], ez[0]);
      if (hasr) ll_store(hout, ve, tag);
      const u64 vf = column_at(C - 1, q[1], q[2], ra, rb, ex[1], ez[1]);
      if (hasr) ll_store(hout + NP, vf, tag);
      // column 0, with the left neighbour's last
      u64 la = 0ull;
      if (hasl) la = ll_wait1(hmine + (size_t)(it & 1) * hpar - hcta, tag, poll);
      const u64 v0 = column_at(0, la, P0, P1, P2, ex[2], ez[2]);
      if (hasl) ll_store(hout + 2 * NP, v0, tag);
      if (kA) {
        lmx = __reduce_max_sync(kAll, lmx);
        lmz = __reduce_max_sync(kAll, lmz);
        if (lane == 0) {
          WM[16 + warp] = lmx;
          WM[32 + warp] = lmz;
        }
      }
      if (kB && it < last) {
        const char* hn = hist_at(slot_b(it + 1), 0);
#pragma unroll
        for (int u = 0; u < U; ++u) hq[u] = ldh(hn, 2 + u, lsrc);
      }
    } else {
      if (kA) {  // pressure maximum of this step
        const unsigned m = __reduce_max_sync(kAll, lane < RB ? WM[lane] : 0u);
        if (lane == 0 && m >= 0x7f800000u) atomicOr(L.err, kErrNonFinite);
        if (FP16) {
          u64* sl = L.slots + (size_t)((it & 1) * 2) * gridDim.x + grp * G;
          if (lane == 0) word_store(sl + b, (u64)tag << 32 | m);
          const unsigned p = group_max(sl, G, tag, poll);
          if (lane == 0) {
            SC[0] = pow2f(15 - amax_exponent(p));
            if (b == 0) S.amax[(size_t)(it - 1) * 3 * kAmaxSlots] = p;
          }
        }
      }
      if (kB && it < last) scales_b(it + 1);
    }
    __syncthreads();
    if (kA && aux) {  // publish the velocity maxima of this step
      const unsigned x = __reduce_max_sync(kAll, lane < RB ? WM[16 + lane] : 0u);
      const unsigned z = __reduce_max_sync(kAll, lane < RB ? WM[32 + lane] : 0u);
      if (lane == 0) {
        if (max(x, z) >= 0x7f800000u) atomicOr(L.err, kErrNonFinite);
        if (FP16) {
          u64* sl = L.slots + (size_t)(4 + (it & 1) * 2) * gridDim.x + grp * G;
          word_store(sl + b, (u64)tag << 32 | x);
          word_store(sl + gridDim.x + b, (u64)tag << 32 | z);
        }
      }
    }
  }

  // ---- the last step's histories
  if (kA) {
    if (aux && FP16) {
      const unsigned tag = L.tag0 + (unsigned)last;
      u64* sl = L.slots + (size_t)(4 + (last & 1) * 2) * gridDim.x + grp * G;
      const unsigned vx = group_max(sl, G, tag, poll);
      const unsigned vz = group_max(sl + gridDim.x, G, tag, poll);
      if (lane == 0) {
        SC[1] = pow2f(15 - amax_exponent(vx));
        SC[2] = pow2f(15 - amax_exponent(vz));
        if (b == 0) {
          unsigned* am = S.amax + (size_t)(last - 1) * 3 * kAmaxSlots;
          am[kAmaxSlots] = vx;
          am[2 * kAmaxSlots] = vz;
        }
      }
    }
    __syncthreads();
  }
  if (!aux && (kA || L.save)) {
    const float ip = kA && FP16 ? SC[0] : 1.f, ix = kA && FP16 ? SC[1] : 1.f,
                iz = kA && FP16 ? SC[2] : 1.f;
    for (int j = 0; j < C; ++j) {
      unsigned t4[4];
      tm_ld4(TP + 4 * j, t4);
      tm_wait(t4);
      const u64 px = pku(t4[0], t4[1]), pz = pku(t4[2], t4[3]), vx = F[96 * j], vz = F[96 * j + 32];
      if (kA) {
        const unsigned on = lphys >> j & 1u;
        HP::put(hist_at(last - 1, 0) + j * hstep,
                mul2(mul2(fsm, add2(px, pz)), pk(r0 ? ip : 0.f, r1 ? ip : 0.f)), pol, on);
        HP::put(hist_at(last - 1, 1) + j * hstep, mul2(vx, pk(r0 ? ix : 0.f, r1 ? ix : 0.f)), pol, on);
        HP::put(hist_at(last - 1, 2) + j * hstep, mul2(vz, pk(r0 ? iz : 0.f, r1 ? iz : 0.f)), pol, on);
      }
      if (L.save && c0 + j < g.n2e) {
        const size_t o = (size_t)(c0 + j) * ld + i1;
        *reinterpret_cast<u64*>(S.px + o) = px;
        *reinterpret_cast<u64*>(S.pz + o) = pz;
        *reinterpret_cast<u64*>(S.vx + o) = vx;
        *reinterpret_cast<u64*>(S.vz + o) = vz;
      }
    }
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (warp == 0) {
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(*TB), "r"(tcols));
  }
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
  const bool full = on && a0 >= ra && a0 + kTap <= rb && b0 >= ca && b0 + kTap <= cb;
  const bool allfull = __all_sync(kAll, full || !on);
  for (int t0 = (blockIdx.y * kGatherWarps + warp) * kGatherSteps; t0 < nsteps;
       t0 += gridDim.y * kGatherWarps * kGatherSteps) {
    float acc[kGatherSteps] = {};
    const float* base[kGatherSteps];
#pragma unroll
    for (int k = 0; k < kGatherSteps; ++k)
      base[k] = r.buf + (size_t)min(t0 + k, nsteps - 1) * r.step;
    if (on) {
      if (allfull) {
        for (int a = 0; a < kTap; ++a) {
          const size_t o = (size_t)(a0 + a - r.r0) * r.ld + (b0 - r.c0);
#pragma unroll
          for (int q = 0; q < kTap; ++q) {
            const float c = tl[(a + kTap * q) * 33 + lane];
#pragma unroll
            for (int k = 0; k < kGatherSteps; ++k) acc[k] = fadd(acc[k], fmul(c, base[k][o + q]));
          }
        }
      } else {
        for (int a = max(0, ra - a0); a < kTap && a0 + a < rb; ++a)
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
void with_kernel(int mode, bool fp16, bool rho, F&& f) {
  auto pick = [&](auto m, auto h) {
    constexpr int M = decltype(m)::value;
    constexpr bool H = decltype(h)::value;
    if (rho)
      f(k_resident<M, H, true>);
    else
      f(k_resident<M, H, false>);
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

size_t resident_smem(int C, int RB, int inj_pts, int inj_m, int inj_sta) {
  const int tw = tm_words(C, RB);
  if (tw > kTmCols) return kMaxSmem + 1;
  // No more CTAs may be resident on an SM than its tensor memory holds: shared
  // memory is padded until it admits just as many (an allocation that does not
  // fit would block inside the kernel).
  const size_t n = kTmCols / tm_alloc(C, RB);
  const size_t floor_bytes = kMaxSmem / (n + 1) + 128;
  return std::max((size_t)layout(C, RB, inj_pts, inj_m, inj_sta).total, floor_bytes);
}

int resident_occupancy(int mode, bool fp16, bool rho, int RB, size_t smem) {
  if (smem > kMaxSmem || RB > kResRowBlocks) return 0;
  int n = 0;
  with_kernel(mode, fp16, rho, [&](auto k) {
    if (cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kMaxSmem) !=
            cudaSuccess ||
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, k, 32 * (RB + 1), smem) != cudaSuccess) {
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
  cfg.blockDim = dim3(32 * (L.RB + 1));
  cfg.dynamicSmemBytes = resident_smem(L.C, L.RB, L.inj_pts, L.inj_m, L.inj_sta);
  cfg.stream = st;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeCooperative;  // CTAs wait on one another: all are resident
  at[0].val.cooperative = 1;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  ResidentLaunch P = L;
  P.nz = kNegZero2;
  cudaError_t e = cudaSuccess;
  with_kernel(mode, fp16, m.rbw1 != nullptr,
              [&](auto k) { e = cudaLaunchKernelEx(&cfg, k, g, m, P); });
  return e;
}

void resident_tables(const Grid& g, const ModelDev& m, const InjMapDev& map, int C, int G,
                     const int4* head, int pts, int mm, float* cd, unsigned short* sta, float* kap,
                     cudaStream_t st) {
  k_resident_tables<<<G, 256, 0, st>>>(g, m.kap, map, C, head, pts, mm, cd, sta, kap);
}

void resident_gather(const ResidentRect& r, const StationsDev& st, int lo1, int hi1, int lo2,
                     int hi2, int nsteps, float* out, int nt, int row0, int reverse,
                     cudaStream_t s) {
  if (st.n <= 0 || nsteps <= 0) return;
  constexpr size_t smem = kTile * 33 * sizeof(float);
  cudaFuncSetAttribute(k_resident_gather, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  const int per = kGatherWarps * kGatherSteps;
  const dim3 grid((st.n + 31) / 32, std::min((nsteps + per - 1) / per, 64));
  k_resident_gather<<<grid, 32 * kGatherWarps, smem, s>>>(r, st, lo1, hi1, lo2, hi2, nsteps,
                                                          out, nt, row0, reverse);
}

}  // namespace daw
