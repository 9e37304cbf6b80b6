// Station tables on the device: the Hicks tiles of a set of stations and the
// gather-form injection map, from the acquisition table alone.
//
// On the host the map of 576 receivers (254 016 taps: tiles, a stable sort by
// grid point, row pointers) took about 9 ms of every call, more than the time
// loops of a short simulation; these two kernels take about 30 us.  The products and
// differences of the tiles are the host code's single-precision operations.
#include "kernels.cuh"

namespace daw {
namespace {

// tile[(i1 + 10) + 21 (i2 + 10)] of one station a block: the product of the two
// 1-D weights (w[tap][position]), the nodes above the free surface folded back
// with the opposite sign (hicks.cpp hicks_tile).
__global__ void k_stations(const int* __restrict__ tab, int n, const float* __restrict__ w,
                           int* __restrict__ ix1, int* __restrict__ ix2, float* __restrict__ tile) {
  const int s = blockIdx.x;
  const int a1 = tab[s + 2 * n] - 1, a2 = tab[s + 3 * n] - 1, nfs = tab[s + 4 * n];
  if (threadIdx.x == 0) {
    ix1[s] = tab[s];
    ix2[s] = tab[s + n];
  }
  for (int t = threadIdx.x; t < kTile; t += blockDim.x) {
    const int i1 = t % kTap, i2 = t / kTap;
    const float w2 = w[i2 * kNAlpha + a2];
    float v = fmul(w2, w[i1 * kNAlpha + a1]);
    const int k = i1 - nfs;  // rows below the surface node
    if (nfs > 0 && k == 0) v = 0.f;
    if (nfs > 0 && k >= 1 && k <= nfs) v = fsub(v, fmul(w2, w[(nfs - k) * kNAlpha + a1]));
    tile[(size_t)s * kTile + t] = v;
  }
}

// Entries of the points of one grid column a block, m slots a point, in station
// order: a thread per row walks the stations, 128 at a time in shared memory.
constexpr int kMapThreads = 128;
__global__ void __launch_bounds__(kMapThreads)
    k_map(const StationsDev st, const int* __restrict__ col_lo, const int* __restrict__ col_hi,
          const int* __restrict__ col_base, int m, int* __restrict__ rowptr, float2* __restrict__ ent) {
  __shared__ int s1[kMapThreads], s2[kMapThreads];
  const int c = blockIdx.x, lo = col_lo[c], hi = col_hi[c];
  if (hi < lo) return;
  for (int r0 = lo; r0 <= hi; r0 += kMapThreads) {
    const int r = r0 + (int)threadIdx.x;
    const size_t q = (size_t)col_base[c] + (r - lo);
    int k = 0;
    for (int b = 0; b < st.n; b += kMapThreads) {
      __syncthreads();
      if (b + (int)threadIdx.x < st.n) {
        s1[threadIdx.x] = st.ix1[b + threadIdx.x] - 1;
        s2[threadIdx.x] = st.ix2[b + threadIdx.x] - 1;
      }
      __syncthreads();
      if (r > hi) continue;
      const int e = min(kMapThreads, st.n - b);
      for (int i = 0; i < e; ++i) {
        const int d1 = r - s1[i], d2 = c - s2[i];
        if (d1 < -kRad || d1 > kRad || d2 < -kRad || d2 > kRad) continue;
        ent[q * m + k] = make_float2(
            st.tile[(size_t)(b + i) * kTile + (d1 + kRad) + kTap * (d2 + kRad)], __int_as_float(b + i));
        ++k;
      }
    }
    if (r <= hi) {
      rowptr[2 * q] = (int)(q * m);
      rowptr[2 * q + 1] = (int)(q * m) + k;
    }
  }
}

}  // namespace

void station_tiles(const int* tab, int n, const float* weights, const StationsDev& s, cudaStream_t st) {
  if (n > 0) k_stations<<<n, 128, 0, st>>>(tab, n, weights, s.ix1, s.ix2, s.tile);
}

void injection_map(const StationsDev& s, int n2e, int m, const InjMapDev& map, cudaStream_t st) {
  if (s.n > 0)
    k_map<<<n2e, kMapThreads, 0, st>>>(s, map.col_lo, map.col_hi, map.col_base, m, map.rowptr, map.ent);
}

}  // namespace daw
