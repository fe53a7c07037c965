// Z-marching stencils: a block owns a 32 (x) by 8 (y) tile of columns and
// marches up a chunk of levels; the planes its stencil reads, with their x and
// y halos, pass through a ring of shared-memory slots, each value fetched once
// a block by cp.async while the levels before it compute.
//
// The copies are of single elements: rows need no alignment, the periodic wrap
// in y is part of a thread's fixed offset, and any grid size can take this path
// (march_direct says which do).
// Planes below the ground or above the top repeat the nearest one, columns
// outside in x the nearest column (the stencils do not use them).
#pragma once
#include <type_traits>
#include "common.cuh"

#define MR_TX 32
#define MR_TY 8
#define MR_THREADS (MR_TX * MR_TY)
#define MR_MAXK 64

template <int BYTES>
__device__ __forceinline__ void copy_async(uint32_t dst, const void* src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], %2;" ::"r"(dst), "l"(src), "n"(BYTES)
               : "memory");
}
__device__ __forceinline__ void copy_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
// all but the newest N groups have landed
template <int N>
__device__ __forceinline__ void copy_wait() {
  asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}

// NF fields of element type T with a halo of R, SLOTS planes
template <typename T, int NF, int R, int SLOTS>
struct PlaneRing {
  static constexpr int HX = MR_TX + 2 * R, HY = MR_TY + 2 * R, PLANE = HX * HY;
  static constexpr int PER = (PLANE + MR_THREADS - 1) / MR_THREADS;
  static constexpr int BYTES = SLOTS * NF * PLANE * (int)sizeof(T);
  uint32_t dst;
  int off[PER];  // of this thread's elements in a plane
  int last;      // it has the last of them
  __device__ __forceinline__ void init(T* base, const GridDev& g) {
    const int tid = threadIdx.y * MR_TX + threadIdx.x;
    dst = (uint32_t)__cvta_generic_to_shared(base) + tid * (int)sizeof(T);
#pragma unroll
    for (int q = 0; q < PER; ++q) {
      const int e = tid + q * MR_THREADS;
      const int i = (int)blockIdx.x * MR_TX - R + e % HX;
      const int j = wrapj((int)blockIdx.y * MR_TY - R + e / HX, g.ny);
      off[q] = j * g.nx + min(max(i, 0), g.nx - 1);
    }
    last = tid + (PER - 1) * MR_THREADS < PLANE;
  }
  // plane p of every field into a slot
  __device__ __forceinline__ void load(const GridDev& g, const T* const (&f)[NF], int p, int slot) {
    const int64_t pl = (int64_t)min(max(p, 0), g.nz - 1) * ((int64_t)g.nx * g.ny);
    const uint32_t d = dst + slot * (NF * PLANE * (int)sizeof(T));
#pragma unroll
    for (int s = 0; s < NF; ++s)
#pragma unroll
      for (int q = 0; q < PER; ++q)
        if (q < PER - 1 || last)
          copy_async<(int)sizeof(T)>(d + (s * PLANE + q * MR_THREADS) * (int)sizeof(T),
                                     f[s] + pl + off[q]);
  }
  // slot s + d (0 <= s < SLOTS, |d| < SLOTS), and its first element from base
  static __device__ __forceinline__ int slot(int s, int d) {
    const int t = s + d;
    return t < 0 ? t + SLOTS : (t >= SLOTS ? t - SLOTS : t);
  }
  static __device__ __forceinline__ const T* at(const T* base, int s) {
    return base + s * (NF * PLANE) + (threadIdx.y + R) * HX + threadIdx.x + R;
  }
};

// The kernels' second form, DIRECT, for grids of few tile levels, where a ring would
// bring five planes for a level or two: a block has one level and a thread takes
// its neighbours from memory.  Offsets of a cell's neighbours in x and y there; at
// an end in x the cell itself (not used).
struct NearCells {
  int xl, xr, yl, yr, yl2, yr2;
  __device__ __forceinline__ void init(const GridDev& g, int i, int j) {
    xl = i > 0 ? -1 : 0;
    xr = i < g.nx - 1 ? 1 : 0;
    yl = (wrapj(j - 1, g.ny) - j) * g.nx;
    yr = (wrapj(j + 1, g.ny) - j) * g.nx;
    yl2 = (wrapj(j - 2, g.ny) - j) * g.nx;
    yr2 = (wrapj(j + 2, g.ny) - j) * g.nx;
  }
};
// the same in a ring's plane
template <int HX>
struct NearSlots {
  static constexpr int xl = -1, xr = 1, yl = -HX, yr = HX, yl2 = -2 * HX, yr2 = 2 * HX;
  __device__ __forceinline__ void init(const GridDev&, int, int) {}
};
template <bool DIRECT, int HX>
using Near = std::conditional_t<DIRECT, NearCells, NearSlots<HX>>;

// Whether a grid takes the DIRECT form of momentum, k-epsilon and species
// transport, by its tile levels (tiles times levels): up to six blocks an SM it was
// the faster one on all of 23 grids, beyond that the ring except on odd rows, whose
// copies touch more sectors, and a little longer in FP32.  us with the ring and
// direct, momentum, k-epsilon, species (FP32 species): 131 x 47 x 14 (420 tile levels)
// 12.8 and 6.7, 15.2 and 10.2, 12.8 and 6.8 (12.6 and 6.3); 128 x 64 x 24 (768) 12.2 and
// 11.4, 16.1 and 15.1, 12.3 and 11.4 (9.1 and 8.9); 90 x 90 x 25 (900) 12.3 and 13.4, 18.6
// and 18.1, 12.6 and 13.5 (11.1 and 9.7); 133 x 45 x 37 (1110) 18.9 and 15.3, 23.2 and
// 19.8, 19.1 and 15.6 (16.3 and 10.6); 224 x 56 x 24 (1176) 14.9 and 15.8, 17.8 and 19.9,
// 14.8 and 15.6 (9.6 and 10.8); 301 x 119 x 47 (7050) 64 and 102, 88 and 149, 68 and 107
// (43 and 60).
#define MR_DIRECT 888
#define MR_DIRECT_F32 1000
#define MR_DIRECT_ODD 1200
template <typename T>
inline bool march_direct(const GridDev& g) {
  const int tiles = ((g.nx + MR_TX - 1) / MR_TX) * ((g.ny + MR_TY - 1) / MR_TY);
  return (int64_t)tiles * g.nz <= (g.nx % 2      ? MR_DIRECT_ODD
                                   : sizeof(T) == 4 ? MR_DIRECT_F32
                                                    : MR_DIRECT);
}

// Levels a block marches.  Few tiles: one, as long as that gives no more than
// MR_FLAT blocks (an SM's blocks overlap each other's loads and barriers, a block
// alone pays two levels' worth before its first; 130 x 100 x 9: gas advection 6.3 us
// with one level, 7.3 with two, 9.1 with five).  Then the chunk count with the least
// (blocks an SM + 2) x (levels + 2).  At 400 x 120 x 60 that is 10 levels (momentum
// 99 us; 101 with 5, 105 with 15, 114 with 30).  Over 23 grids and all kernels the
// choice is 1.7 % above the best one.
#define MR_FLAT 800
inline int march_levels(const GridDev& g) {
  const int tiles = ((g.nx + MR_TX - 1) / MR_TX) * ((g.ny + MR_TY - 1) / MR_TY);
  if ((int64_t)tiles * g.nz <= MR_FLAT) return 1;
  int best = 1;
  int64_t least = INT64_MAX;
  for (int kz = 1; kz <= g.nz && kz <= MR_MAXK; ++kz) {
    const int64_t blocks = (int64_t)tiles * ((g.nz + kz - 1) / kz);
    const int64_t cost = ((blocks + 147) / 148 + 2) * (kz + 2);
    if (cost < least) {
      least = cost;
      best = kz;
    }
  }
  return best;
}
inline dim3 march_grid(const GridDev& g, int kz) {
  return dim3((g.nx + MR_TX - 1) / MR_TX, (g.ny + MR_TY - 1) / MR_TY, (g.nz + kz - 1) / kz);
}

// the shared memory a marching kernel may ask for (set on every call: the
// attribute belongs to the current device)
inline bool march_smem(const void* kernel, int bytes) {
  return cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes) ==
         cudaSuccess;
}

// The reciprocal spacings of a chunk's levels, MR_RK a level: face above, face
// below, cell, mean of the faces, and the vertical difference of the strain
// and of the buoyancy (one-sided at the ground and the top).
#define MR_RK 5
template <typename T>
__device__ __forceinline__ void march_spacings(const GridDev& g, int k0, int k1, T* rk) {
  for (int q = threadIdx.y * MR_TX + threadIdx.x; q < k1 - k0; q += MR_THREADS) {
    const int k = k0 + q;
    const double da = g.da[k], db = g.db[k];
    rk[q * MR_RK + 0] = (T)(1.0 / da);
    rk[q * MR_RK + 1] = (T)(1.0 / db);
    rk[q * MR_RK + 2] = (T)(1.0 / g.dz[k]);
    rk[q * MR_RK + 3] = (T)(1.0 / (0.5 * (da + db)));
    rk[q * MR_RK + 4] = (T)(1.0 / (k == 0 ? da : (k == g.nz - 1 ? db : da + db)));
  }
}

// The smaller of two differences of one sign, else 0 (minmod)
template <typename T>
__device__ __forceinline__ T minmod_pair(T a, T b) {
  const T m = (fabs(b) < fabs(a)) ? b : a;
  return (a * b <= T(0)) ? T(0) : m;
}
// The difference of a cell's two MUSCL face values along one direction, over
// the sign of the velocity: |uf| times it is uf (f+ - f-).  dp, dm: the
// differences to the neighbours in + and - direction; N the upwind neighbour and
// F the one beyond it.  Of the two limiters one is of dp and dm whichever way
// the wind blows, so a cell needs three differences and two limiters where face
// by face it took four to six differences and as many selections.
template <typename T>
__device__ __forceinline__ T muscl_diff(T dp, T dm, T C, T N, T F, bool up) {
  const T h = up ? T(0.5) : T(-0.5);
  const T d = up ? N - F : F - N;
  const T a = C + h * minmod_pair(dp, dm);
  const T b = N + h * minmod_pair(up ? dm : dp, d);
  return a - b;
}
