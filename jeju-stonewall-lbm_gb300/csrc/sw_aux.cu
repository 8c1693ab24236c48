// sw_aux.cu -- k_init, k_macro / k_accum, tile classification and layout transposes.
//
// This translation unit is compiled with --fmad=false: these kernels run once
// (or every few steps) and evaluate every expression in source order, so their
// float32 results equal the reference's operation sequence exactly (k_init for
// the same random stream, k_macro for the same f).
#include <cooperative_groups.h>

#include "sw_aux.cuh"

namespace sw {

// ---------------------------------------------------------------- random stream
// PCG hash (Jarzynski & Olano, JCGT 2020), used as rand_init(seed, offset) =
// pcg(seed + pcg(offset)) and randf(state) = (pcg(state) >> 8) / 2^24 -- the
// form of the wp.rand_init / wp.randf calls in lbm3d.py:48-52.
__device__ __forceinline__ uint32_t pcg_hash(uint32_t s) {
  uint32_t b = s * 747796405u + 2891336453u;
  uint32_t c = ((b >> ((b >> 28u) + 4u)) ^ b) * 277803737u;
  return (c >> 22u) ^ c;
}
__device__ __forceinline__ float randf(uint32_t &st) {
  st = pcg_hash(st);
  return (float)(st >> 8) * (1.0f / 16777216.0f);
}
// Standard normals by Box-Muller, in float (FP64 is slow on this part; the
// oracle's double-precision version agrees to float rounding).
__device__ __forceinline__ float gauss_pair(uint32_t &st, float *second) {
  const float u1 = 1.0f - randf(st);  // (0, 1]
  const float u2 = randf(st);
  const float r = sqrtf(-2.0f * logf(u1));
  float sn, cs;
  sincosf(6.2831853071795865f * u2, &sn, &cs);
  if (second) *second = r * sn;
  return r * cs;
}

// Velocity of k_init at a cell (lbm3d.py:45-52): the perturbed inlet speed, rest at solids.
template <typename R>
__device__ __forceinline__ void init_velocity(bool fluid, int x, int y, int z, const float *uin, float noise, int seed,
                                              int noise_kind, R &ux, R &uy, R &uz) {
  ux = uy = uz = R(0.0);
  if (!fluid) return;
  const uint32_t off = ((uint32_t)x * 7919u + (uint32_t)y) * 7907u + (uint32_t)z;
  uint32_t st = pcg_hash((uint32_t)seed + pcg_hash(off));
  const R u0 = (R)uin[z];
  const R nz_ = (R)noise;
  if (noise_kind == SW_NOISE_UNIFORM) {
    ux = u0 * (R(1.0) + nz_ * (R(2.0) * (R)randf(st) - R(1.0)));
    uy = u0 * nz_ * (R(2.0) * (R)randf(st) - R(1.0));
    uz = u0 * nz_ * (R(2.0) * (R)randf(st) - R(1.0));
  } else {
    float g2 = 0.0f;
    const float g1 = gauss_pair(st, &g2);
    const float g3 = gauss_pair(st, nullptr);
    ux = u0 * (R(1.0) + nz_ * (R)g1);
    uy = u0 * nz_ * (R)g2;
    uz = u0 * nz_ * (R)g3;
  }
}

// feq_i (lbm3d.py:33-36) at rho = 1 for all populations, in feq_i's order for
// each: put(Int<i>, value).  The terms of c_a = 0 are left out (they add a zero)
// and the members of a pair share (c.u)^2.
template <typename R, typename Put>
__device__ __forceinline__ void init_populations(R ux, R uy, R uz, Put &&put) {
  const R k = R(1.5) * (ux * ux + uy * uy + uz * uz);
  put(Int<0>{}, W<R>(0) * ((R(1.0) + R(0.0)) - k));
  static_for<0, 9>([&](auto P) {
    constexpr int i = 2 * decltype(P)::value + 1;
    constexpr int cx = CX(i), cy = CY(i), cz = CZ(i);
    R cu;
    if constexpr (cx != 0 && cy != 0) cu = (cx > 0 ? ux : -ux) + (cy > 0 ? uy : -uy);
    else if constexpr (cx != 0 && cz != 0) cu = (cx > 0 ? ux : -ux) + (cz > 0 ? uz : -uz);
    else if constexpr (cy != 0 && cz != 0) cu = (cy > 0 ? uy : -uy) + (cz > 0 ? uz : -uz);
    else if constexpr (cx != 0) cu = cx > 0 ? ux : -ux;
    else if constexpr (cy != 0) cu = cy > 0 ? uy : -uy;
    else cu = cz > 0 ? uz : -uz;
    cu = R(3.0) * cu;
    const R h = R(0.5) * cu * cu;
    put(Int<i>{}, W<R>(i) * (R(1.0) + cu + h - k));
    put(Int<i + 1>{}, W<R>(i) * (R(1.0) - cu + h - k));
  });
}

// k_init, lbm3d.py:39-54.  CPT cells per thread along x: two in the 16-bit types,
// stored as one 32-bit word a population.  Bound by the stores and, with
// Gaussian noise, as much by its logarithms and sines; 32-bit index arithmetic
// (a plane has fewer than 2^31 cells) and the shared pair terms took a
// 640x128x128 fp16 lattice from 173 to 137 us.
template <int DT, int CPT>
__global__ void __launch_bounds__(256) k_init(Geom g, typename Store<DT>::T *f, const uint8_t *flag, const float *uin,
                                              float noise, int seed, int noise_kind) {
  using S = Store<DT>;
  using T = typename S::T;
  using R = typename S::R;
  const uint32_t c = (blockIdx.x * 256u + threadIdx.x) * CPT;
  if (c >= (uint32_t)g.plane) return;
  const uint32_t row = c / (uint32_t)g.pitch;
  const int x = (int)(c - row * (uint32_t)g.pitch);
  const int z = (int)(row / (uint32_t)g.ny), y = (int)(row - (uint32_t)z * (uint32_t)g.ny);
  if (x >= g.nx) return;
  const size_t plane = (size_t)g.plane;
  T v[CPT][Q];
#pragma unroll
  for (int j = 0; j < CPT; ++j) {
    R ux, uy, uz;
    init_velocity<R>(x + j < g.nx && flag[c + j] == 0, x + j, y, z, uin, noise, seed, noise_kind, ux, uy, uz);
    init_populations<R>(ux, uy, uz, [&](auto I, R w) {
      constexpr int i = decltype(I)::value;
      v[j][i] = S::template enc<i>(w);
    });
  }
  static_for<0, Q>([&](auto I) {
    constexpr int i = decltype(I)::value;
    T *o = f + (size_t)i * plane + c;
    if constexpr (CPT == 2) {
      if (x + 1 < g.nx) {
        struct alignas(2 * sizeof(T)) Pair { T a, b; };
        *reinterpret_cast<Pair *>(o) = Pair{v[0][i], v[1][i]};
        return;
      }
    }
    *o = v[0][i];
  });
}

// k_macro (lbm3d.py:158-182) with an optional fused k_accum (lbm3d.py:185-188) in double.
template <int DT>
__global__ void k_macro(Geom g, const typename Store<DT>::T *f, const uint8_t *flag, float *u, double *acc) {
  using S = Store<DT>;
  using R = typename S::R;
  const long long c = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= g.plane) return;
  if ((int)(c % g.pitch) >= g.nx) return;
  const size_t P = (size_t)g.plane;
  R out[4];
  if (flag[c] != 0) {
    out[0] = R(1.0); out[1] = R(0.0); out[2] = R(0.0); out[3] = R(0.0);
  } else {
    R rho = R(0.0), mx = R(0.0), my = R(0.0), mz = R(0.0);
    static_for<0, Q>([&](auto I) {
      constexpr int i = decltype(I)::value;
      const R v = S::template dec<i>(f[(size_t)i * P + c]);
      rho += v;
      mx += v * R(CX(i));
      my += v * R(CY(i));
      mz += v * R(CZ(i));
    });
    out[0] = rho; out[1] = mx / rho; out[2] = my / rho; out[3] = mz / rho;
  }
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    if (u) u[k * P + c] = (float)out[k];
    if (acc) acc[k * P + c] += (double)out[k];
  }
}

__global__ void k_accum(Geom g, const float *u, double *acc) {
  const long long c = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= 4 * g.plane) return;
  if ((int)(c % g.pitch) >= g.nx) return;
  acc[c] += (double)u[c];
}

// The 32 flags of a row segment as bit masks: not fluid, and stone.
struct SegMask {
  uint32_t solid, wall;
};
// bit k of the result: byte k of w is not zero
__device__ __forceinline__ uint32_t nonzero_bytes(uint32_t w) {
  const uint32_t t = ((((w & 0x7f7f7f7fu) + 0x7f7f7f7fu) | w) >> 7) & 0x01010101u;
  return (t * 0x10204080u) >> 28;
}
template <bool ALIGNED> __device__ __forceinline__ SegMask seg_mask(const uint8_t *seg) {
  uint32_t w[8];
  if constexpr (ALIGNED) {
    const uint4 a = __ldg(reinterpret_cast<const uint4 *>(seg)), b = __ldg(reinterpret_cast<const uint4 *>(seg) + 1);
    w[0] = a.x, w[1] = a.y, w[2] = a.z, w[3] = a.w, w[4] = b.x, w[5] = b.y, w[6] = b.z, w[7] = b.w;
  } else {
#pragma unroll
    for (int k = 0; k < 8; ++k)
      w[k] = seg[4 * k] | (uint32_t)seg[4 * k + 1] << 8 | (uint32_t)seg[4 * k + 2] << 16 | (uint32_t)seg[4 * k + 3] << 24;
  }
  SegMask m{0u, 0u};
  if (((w[0] | w[1]) | (w[2] | w[3])) | ((w[4] | w[5]) | (w[6] | w[7]))) {   // (most segments are all fluid)
#pragma unroll
    for (int k = 0; k < 8; ++k) {
      m.solid |= nonzero_bytes(w[k]) << (4 * k);
      m.wall |= (nonzero_bytes(w[k] ^ 0x01010101u) ^ 15u) << (4 * k);
    }
  }
  return m;
}

// Segment classification for the step kernel (see TILE_* in sw_common.cuh).
// Mirrors the pull-source mapping of the step (lbm3d.py:77-88).  One thread per
// segment: the nine source rows' 32 flags each become two bit masks, shifted
// along x for the sources at x - 1 and x + 1, so a segment takes 18 16-byte
// loads instead of 19 byte loads per cell: 640x128x128, 506 -> 13 us.
template <bool ALIGNED>
__global__ void __launch_bounds__(256) k_build_tiles(Geom g, const uint8_t *flag, uint8_t *tiles) {
  const uint32_t nseg = (uint32_t)(g.plane / SEG);
  const uint32_t seg = blockIdx.x * 256u + threadIdx.x;
  if (seg >= nseg) return;
  const uint32_t row = seg / (uint32_t)g.nseg_x;
  const int sx = (int)(seg - row * (uint32_t)g.nseg_x);
  const int z = (int)(row / (uint32_t)g.ny), y = (int)(row - (uint32_t)z * (uint32_t)g.ny);
  const int x0 = sx * SEG, left = g.nx - x0;                          // cells of the row from here on
  const uint32_t live = left >= SEG ? 0xffffffffu : (1u << left) - 1u;
  const int ys[3] = {y == 0 ? g.ny - 1 : y - 1, y, y == g.ny - 1 ? 0 : y + 1};
  const int zs[3] = {z - 1, z, z == g.nz - 1 ? z : z + 1};            // the top copies its own level
  uint32_t solid = 0u, wall = 0u, own = 0u;                           // sources of each cell, ORed
#pragma unroll
  for (int dz = 0; dz < 3; ++dz) {
    if (zs[dz] < 0) {                                                 // below the bottom plane: ground
      solid = 0xffffffffu;
      continue;
    }
#pragma unroll
    for (int dy = 0; dy < 3; ++dy) {
      const uint8_t *p = flag + (((size_t)zs[dz] * g.ny + ys[dy]) * g.pitch + x0);
      const SegMask m = seg_mask<ALIGNED>(p);
      if (dz == 1 && dy == 1) own = m.solid;
      else solid |= m.solid, wall |= m.wall;                          // the source at x
      if (dz == 1 || dy == 1) {                                       // sources at x - 1 and x + 1
        const uint8_t before = x0 > 0 ? p[-1] : (uint8_t)0;           // (the inlet does not pull)
        const uint8_t after = left > SEG ? p[SEG] : (uint8_t)0;
        uint32_t sn = (m.solid >> 1) | (after != 0 ? 0x80000000u : 0u), wn = (m.wall >> 1) | (after == SW_WALL ? 0x80000000u : 0u);
        if (left <= SEG) {                                            // the outlet copies column nx - 1
          const uint32_t last = 1u << (left - 1);
          sn = (sn & ~last) | (m.solid & last);
          wn = (wn & ~last) | (m.wall & last);
        }
        solid |= sn | (m.solid << 1) | (before != 0 ? 1u : 0u);
        wall |= wn | (m.wall << 1) | (before == SW_WALL ? 1u : 0u);
      }
    }
  }
  const uint32_t fluid = live & ~own;
  const uint32_t pulls = x0 == 0 ? fluid & ~1u : fluid;               // inlet cells do not pull
  tiles[seg] = (uint8_t)((fluid ? 0 : TILE_ALL_SOLID) | ((live & own) | (pulls & solid) ? TILE_CHECK : 0) |
                         (pulls & wall ? TILE_FORCE : 0));
}

// ---------------------------------------------------------------- x <-> z transposes
// Reference layout a[k][x][y][z] (z fastest) <-> device layout b[k][z][y][pitch].
// One block moves a 64 x 32 tile of the (x, z) plane of one (k, y), eight elements
// per thread in flight on either side.  Bound by DRAM; with one element in flight
// per row step (32 x 32 tiles) and the weight of k found per element, a float32
// 480x96x96 lattice took 240 us each way, now 139.
constexpr int kTileX = 64, kTileZ = 32, kTileThreads = 256;
template <typename A, typename B, typename Conv>
__global__ void __launch_bounds__(kTileThreads) k_ref_to_dev(Geom g, const A *a, B *b, Conv make) {
  __shared__ A t[kTileX][kTileZ + 1];
  const int ky = blockIdx.x;             // k * ny + y
  const int k = ky / g.ny, y = ky % g.ny;
  const int x0 = blockIdx.y * kTileX, z0 = blockIdx.z * kTileZ;
  const auto conv = make(k);
  constexpr int kRows = kTileThreads / kTileZ, N = kTileX / kRows;
  {
    const int dz = threadIdx.x % kTileZ, dx = threadIdx.x / kTileZ, z = z0 + dz;
    const A *src = a + (size_t)k * g.nx * g.ny * g.nz + ((size_t)(x0 + dx) * g.ny + y) * g.nz + z;
    A v[N];
#pragma unroll
    for (int j = 0; j < N; ++j)
      if (x0 + dx + j * kRows < g.nx && z < g.nz) v[j] = __ldg(src + (size_t)j * kRows * g.ny * g.nz);
#pragma unroll
    for (int j = 0; j < N; ++j) t[dx + j * kRows][dz] = v[j];
  }
  __syncthreads();
  constexpr int kLevels = kTileThreads / kTileX, M = kTileZ / kLevels;
  const int dx = threadIdx.x % kTileX, dz = threadIdx.x / kTileX, x = x0 + dx;
  if (x >= g.pitch) return;
  B *dst = b + (size_t)k * g.plane + ((size_t)(z0 + dz) * g.ny + y) * g.pitch + x;
#pragma unroll
  for (int j = 0; j < M; ++j)
    if (z0 + dz + j * kLevels < g.nz)
      dst[(size_t)j * kLevels * g.ny * g.pitch] = x < g.nx ? conv(t[dx][dz + j * kLevels]) : conv.pad();
}

template <typename B, typename A, typename Conv>
__global__ void __launch_bounds__(kTileThreads) k_dev_to_ref(Geom g, const B *b, A *a, Conv make) {
  __shared__ A t[kTileX][kTileZ + 1];
  const int ky = blockIdx.x;
  const int k = ky / g.ny, y = ky % g.ny;
  const int x0 = blockIdx.y * kTileX, z0 = blockIdx.z * kTileZ;
  const auto conv = make(k);
  {
    constexpr int kLevels = kTileThreads / kTileX, M = kTileZ / kLevels;
    const int dx = threadIdx.x % kTileX, dz = threadIdx.x / kTileX, x = x0 + dx;
    const B *src = b + (size_t)k * g.plane + ((size_t)(z0 + dz) * g.ny + y) * g.pitch + x;
    B v[M];
#pragma unroll
    for (int j = 0; j < M; ++j)
      if (x < g.nx && z0 + dz + j * kLevels < g.nz) v[j] = __ldg(src + (size_t)j * kLevels * g.ny * g.pitch);
#pragma unroll
    for (int j = 0; j < M; ++j) t[dx][dz + j * kLevels] = conv(v[j]);
  }
  __syncthreads();
  constexpr int kRows = kTileThreads / kTileZ, N = kTileX / kRows;
  const int dz = threadIdx.x % kTileZ, dx = threadIdx.x / kTileZ, z = z0 + dz;
  if (z >= g.nz) return;
  A *dst = a + (size_t)k * g.nx * g.ny * g.nz + ((size_t)(x0 + dx) * g.ny + y) * g.nz + z;
#pragma unroll
  for (int j = 0; j < N; ++j)
    if (x0 + dx + j * kRows < g.nx) dst[(size_t)j * kRows * g.ny * g.nz] = t[dx + j * kRows][dz];
}

// The weight of population k, as W<R>(k).
template <typename R> __device__ __forceinline__ R weight_of(int k) {
  return k == 0 ? W<R>(0) : k < 7 ? W<R>(1) : W<R>(7);
}
// Converters between a reference-layout value and the stored value of population k,
// made once per block (Store::enc and Store::dec with the weight at run time).
template <int DT, typename A> struct EncF {
  using S = Store<DT>;
  struct Of {
    typename S::R w;
    __device__ typename S::T operator()(A v) const {
      if constexpr (S::kShift) return S::from_shifted((typename S::R)v - w);
      else return (typename S::R)v;
    }
    __device__ typename S::T pad() const {
      if constexpr (S::kShift) return S::from_shifted(w - w);
      else return w;
    }
  };
  __device__ Of operator()(int k) const { return {weight_of<typename S::R>(k)}; }
};
template <int DT, typename A> struct DecF {
  using S = Store<DT>;
  struct Of {
    typename S::R w;
    __device__ A operator()(typename S::T v) const {
      if constexpr (S::kShift) return (A)(w + S::to_shifted(v));
      else return (A)v;
    }
  };
  __device__ Of operator()(int k) const { return {weight_of<typename S::R>(k)}; }
};
template <typename A> struct Ident {
  struct Of {
    __device__ A operator()(A v) const { return v; }
    __device__ A pad() const { return A(0); }
  };
  __device__ Of operator()(int) const { return {}; }
};

inline dim3 tgrid(const Geom &g, int nk, int xext) {
  return dim3((unsigned)(nk * g.ny), (unsigned)((xext + kTileX - 1) / kTileX), (unsigned)((g.nz + kTileZ - 1) / kTileZ));
}

template <int DT>
cudaError_t pack_f_t(const Geom &g, int ref_dtype, const void *ref, void *f, cudaStream_t s) {
  using T = typename Store<DT>::T;
  if (ref_dtype == SW_F32)
    k_ref_to_dev<<<tgrid(g, Q, g.pitch), kTileThreads, 0, s>>>(g, (const float *)ref, (T *)f, EncF<DT, float>{});
  else
    k_ref_to_dev<<<tgrid(g, Q, g.pitch), kTileThreads, 0, s>>>(g, (const double *)ref, (T *)f, EncF<DT, double>{});
  return cudaGetLastError();
}
template <int DT>
cudaError_t unpack_f_t(const Geom &g, int ref_dtype, const void *f, void *ref, cudaStream_t s) {
  using T = typename Store<DT>::T;
  if (ref_dtype == SW_F32)
    k_dev_to_ref<<<tgrid(g, Q, g.nx), kTileThreads, 0, s>>>(g, (const T *)f, (float *)ref, DecF<DT, float>{});
  else
    k_dev_to_ref<<<tgrid(g, Q, g.nx), kTileThreads, 0, s>>>(g, (const T *)f, (double *)ref, DecF<DT, double>{});
  return cudaGetLastError();
}

template <int DT>
cudaError_t init_t(const Geom &g, void *f, const uint8_t *flag, const float *uin, float noise, int seed, int kind,
                   cudaStream_t s) {
  constexpr int CPT = sizeof(typename Store<DT>::T) == 2 ? 2 : 1;
  const long long blocks = (g.plane / CPT + 255) / 256;
  k_init<DT, CPT><<<(unsigned)blocks, 256, 0, s>>>(g, (typename Store<DT>::T *)f, flag, uin, noise, seed, kind);
  return cudaGetLastError();
}
template <int DT>
cudaError_t macro_t(const Geom &g, const void *f, const uint8_t *flag, float *u, double *acc, cudaStream_t s) {
  const long long blocks = (g.plane + 255) / 256;
  k_macro<DT><<<(unsigned)blocks, 256, 0, s>>>(g, (const typename Store<DT>::T *)f, flag, u, acc);
  return cudaGetLastError();
}

#define SW_DISPATCH(dtype, CALL)                         \
  switch (dtype) {                                       \
    case SW_F32: { constexpr int DT = SW_F32; return CALL; } \
    case SW_F64: { constexpr int DT = SW_F64; return CALL; } \
    case SW_F16_SHIFT: { constexpr int DT = SW_F16_SHIFT; return CALL; } \
    case SW_BF16_SHIFT: { constexpr int DT = SW_BF16_SHIFT; return CALL; } \
    default: return cudaErrorInvalidValue;               \
  }

cudaError_t aux_init(const Geom &g, int dtype, void *f, const uint8_t *flag, const float *uin, float noise, int seed,
                     int kind, cudaStream_t s) {
  SW_DISPATCH(dtype, init_t<DT>(g, f, flag, uin, noise, seed, kind, s));
}
cudaError_t aux_macro(const Geom &g, int dtype, const void *f, const uint8_t *flag, float *u, double *acc,
                      cudaStream_t s) {
  SW_DISPATCH(dtype, macro_t<DT>(g, f, flag, u, acc, s));
}
cudaError_t aux_accum(const Geom &g, const float *u, double *acc, cudaStream_t s) {
  const long long blocks = (4 * g.plane + 255) / 256;
  k_accum<<<(unsigned)blocks, 256, 0, s>>>(g, u, acc);
  return cudaGetLastError();
}
cudaError_t aux_pack_f(const Geom &g, int dtype, int ref_dtype, const void *ref, void *f, cudaStream_t s) {
  SW_DISPATCH(dtype, pack_f_t<DT>(g, ref_dtype, ref, f, s));
}
cudaError_t aux_unpack_f(const Geom &g, int dtype, int ref_dtype, const void *f, void *ref, cudaStream_t s) {
  SW_DISPATCH(dtype, unpack_f_t<DT>(g, ref_dtype, f, ref, s));
}
cudaError_t aux_pack_flag(const Geom &g, const uint8_t *ref, uint8_t *flag, cudaStream_t s) {
  k_ref_to_dev<<<tgrid(g, 1, g.pitch), kTileThreads, 0, s>>>(g, ref, flag, Ident<uint8_t>{});
  return cudaGetLastError();
}
cudaError_t aux_unpack_u(const Geom &g, const float *u, float *ref, cudaStream_t s) {
  k_dev_to_ref<<<tgrid(g, 4, g.nx), kTileThreads, 0, s>>>(g, u, ref, Ident<float>{});
  return cudaGetLastError();
}
cudaError_t aux_unpack_acc(const Geom &g, const double *acc, double *ref, cudaStream_t s) {
  k_dev_to_ref<<<tgrid(g, 4, g.nx), kTileThreads, 0, s>>>(g, acc, ref, Ident<double>{});
  return cudaGetLastError();
}
cudaError_t aux_build_tiles(const Geom &g, const uint8_t *flag, uint8_t *tiles, cudaStream_t s) {
  const unsigned blocks = (unsigned)((g.plane / SEG + 255) / 256);
  if (((uintptr_t)flag & 15u) == 0) k_build_tiles<true><<<blocks, 256, 0, s>>>(g, flag, tiles);
  else k_build_tiles<false><<<blocks, 256, 0, s>>>(g, flag, tiles);     // rows start on 32-byte offsets of it
  return cudaGetLastError();
}

__global__ void k_force_to_f64(const long long *fx, double *out, long long n) {
  const long long k = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (k < n) out[k] = (double)fx[k] * (1.0 / FORCE_SCALE);
}
cudaError_t aux_force_to_f64(const long long *fx, double *out, long long n, cudaStream_t s) {
  if (n <= 0) return cudaSuccess;
  k_force_to_f64<<<(unsigned)((n + 255) / 256), 256, 0, s>>>(fx, out, n);
  return cudaGetLastError();
}

// ---------------------------------------------------------------- wall-load coefficients
// lbm3d.py:396-407: per step t, Fx = sum_z F_x(z), Fz = sum_z F_z(z) and the
// overturning moment M = sum_z F_x(z) (z - 1/2) about the wall base, as
// Cd = Fx / (q A), Cl = Fz / (q A), Cm = M / (q A H), q A = U_H^2 / 2 * H ny.
// Eight lanes per step (a row of 16-byte levels is read 128 bytes at a time).
// The sums over the levels are exact: the halves of the fixed-point values are
// added as 64-bit integers and become doubles once per lane, because the FP64
// pipe retires two operations per clock and SM, conversions included (nine of
// them per level bounded the first form: 20 000 x 128 levels 100 us, now
// 20 us).  kCoefLevels levels at a time keep the integer sums below 2^62.
constexpr int kCoefLevels = 1 << 16;
__global__ void __launch_bounds__(256) k_coefficients(const long long *force, long long n_steps, int nz, double qa,
                                                      double H, double *coef) {
  const long long t = ((long long)blockIdx.x * 256 + threadIdx.x) >> 3;
  const int lane = threadIdx.x & 7;
  double sum[3] = {0.0, 0.0, 0.0};                           // Fx, Fz, 2 M (in units of 1 / FORCE_SCALE)
  if (t < n_steps) {
    const longlong2 *row = reinterpret_cast<const longlong2 *>(force) + t * nz;
    for (int z0 = 0; z0 < nz; z0 += kCoefLevels) {
      const int n = nz - z0 < kCoefLevels ? nz - z0 : kCoefLevels;
      long long xh = 0, xl = 0, zh = 0, zl = 0, mh = 0, ml = 0;
#pragma unroll 4
      for (int z = lane; z < n; z += 8) {
        const longlong2 v = __ldg(row + z0 + z);
        const int h = (int)(v.x >> 32), w = 2 * z - 1;
        const uint32_t l = (uint32_t)v.x;
        xh += h;
        xl += l;
        zh += (int)(v.y >> 32);
        zl += (uint32_t)v.y;
        mh += (long long)h * w;
        ml += (long long)l * w;
      }
      const double fx = __fma_rn((double)xh, 4294967296.0, (double)xl);
      sum[0] += fx;
      sum[1] += __fma_rn((double)zh, 4294967296.0, (double)zl);
      sum[2] += __fma_rn((double)mh, 4294967296.0, (double)ml);
      if (z0 > 0) sum[2] += 2.0 * (double)z0 * fx;           // (uniform: rows this long are rare)
    }
  }
#pragma unroll
  for (int o = 4; o > 0; o >>= 1) {
#pragma unroll
    for (int k = 0; k < 3; ++k) sum[k] += __shfl_xor_sync(0xffffffffu, sum[k], o);
  }
  // lane k writes coefficient k: Cd, Cl, Cm (one division per warp)
  const double scale = lane == 2 ? 0.5 / FORCE_SCALE : 1.0 / FORCE_SCALE;
  const double den = lane == 2 ? qa * H : qa, num = lane == 0 ? sum[0] : lane == 1 ? sum[1] : sum[2];
  if (t < n_steps && lane < 3) coef[lane * n_steps + t] = num * scale / den;
}

// postprocess.py:65-82 over the steps t >= n_spin of the coefficient series:
// stats = mean Cd, max Cd, std Cd (about the mean, two passes), mean Cm, max Cm,
// mean Cl; NaN when no step is left.  One cluster of blocks, partial results
// exchanged through distributed shared memory, fixed reduction order.  Bound by
// one SM's FP64 pipe as a single block (62 us for 20 000 steps, 16 us with
// eight); the maxima compare bit patterns as integers for the same reason.
constexpr int kStatThreads = 256, kStatBlocks = 8;
struct StatPart {
  double cd, cm, cl, dev;
  long long max_cd, max_cm;
};
// doubles in the order of their values as signed integers; NaN as -infinity,
// which a maximum starts from
constexpr long long ordered_floor = (long long)0x800fffffffffffffull;
__device__ __forceinline__ long long ordered(double v) {
  const long long b = __double_as_longlong(v);
  const long long k = b ^ ((b >> 63) & 0x7fffffffffffffffll);
  return (b & 0x7fffffffffffffffll) > 0x7ff0000000000000ll ? ordered_floor : k;
}
__device__ __forceinline__ double unordered(long long k) {
  return __longlong_as_double(k ^ ((k >> 63) & 0x7fffffffffffffffll));
}
// warp sums of this block in sh, added in warp order by every thread
__device__ __forceinline__ double block_sum(double v, double *sh) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = v;
  __syncthreads();
  if (threadIdx.x == 0)
    for (int w = 1; w < kStatThreads / 32; ++w) v += sh[w];
  __syncthreads();
  return v;                                                  // thread 0's is the block's
}
__device__ __forceinline__ long long block_max(long long v, long long *sh) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    const long long w = __shfl_xor_sync(0xffffffffu, v, o);
    v = w > v ? w : v;
  }
  if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = v;
  __syncthreads();
  if (threadIdx.x == 0)
    for (int w = 1; w < kStatThreads / 32; ++w) v = sh[w] > v ? sh[w] : v;
  __syncthreads();
  return v;
}
__global__ void __cluster_dims__(kStatBlocks) __launch_bounds__(kStatThreads)
    k_coef_stats(const double *coef, long long n_steps, long long n_spin, double *stats) {
  namespace cg = cooperative_groups;
  __shared__ StatPart part;
  __shared__ double sh[kStatThreads / 32];
  __shared__ long long shk[kStatThreads / 32];
  cg::cluster_group cluster = cg::this_cluster();
  const double *cd = coef, *cl = coef + n_steps, *cm = coef + 2 * n_steps;
  const long long n = n_steps - n_spin;
  if (n <= 0) {                                              // the same in every block
    if (blockIdx.x == 0 && threadIdx.x < 6) stats[threadIdx.x] = __longlong_as_double(0x7ff8000000000000ll);
    return;
  }
  const long long first = n_spin + (long long)blockIdx.x * kStatThreads + threadIdx.x;
  constexpr long long stride = (long long)kStatBlocks * kStatThreads;
  double s_cd = 0.0, s_cm = 0.0, s_cl = 0.0;
  long long m_cd = ordered_floor, m_cm = ordered_floor;
#pragma unroll 4
  for (long long t = first; t < n_steps; t += stride) {
    const double a = cd[t], b = cm[t];
    s_cd += a;
    s_cm += b;
    s_cl += cl[t];
    const long long ka = ordered(a), kb = ordered(b);
    m_cd = ka > m_cd ? ka : m_cd;
    m_cm = kb > m_cm ? kb : m_cm;
  }
  s_cd = block_sum(s_cd, sh);
  s_cm = block_sum(s_cm, sh);
  s_cl = block_sum(s_cl, sh);
  m_cd = block_max(m_cd, shk);
  m_cm = block_max(m_cm, shk);
  if (threadIdx.x == 0) part = {s_cd, s_cm, s_cl, 0.0, m_cd, m_cm};
  cluster.sync();
  double mean_cd = 0.0;
  for (int r = 0; r < kStatBlocks; ++r) mean_cd += cluster.map_shared_rank(&part, r)->cd;
  mean_cd = mean_cd / (double)n;
  double s_dev = 0.0;
#pragma unroll 4
  for (long long t = first; t < n_steps; t += stride) {
    const double d = cd[t] - mean_cd;
    s_dev += d * d;
  }
  s_dev = block_sum(s_dev, sh);
  if (threadIdx.x == 0) part.dev = s_dev;
  cluster.sync();
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    StatPart all = part;
    for (int r = 1; r < kStatBlocks; ++r) {
      const StatPart *o = cluster.map_shared_rank(&part, r);
      all.cm += o->cm;
      all.cl += o->cl;
      all.dev += o->dev;
      all.max_cd = o->max_cd > all.max_cd ? o->max_cd : all.max_cd;
      all.max_cm = o->max_cm > all.max_cm ? o->max_cm : all.max_cm;
    }
    stats[0] = mean_cd;
    stats[1] = unordered(all.max_cd);
    stats[2] = sqrt(all.dev / (double)n);
    stats[3] = all.cm / (double)n;
    stats[4] = unordered(all.max_cm);
    stats[5] = all.cl / (double)n;
  }
  cluster.sync();                                            // the other blocks' shared memory until read
}

cudaError_t aux_coefficients(const long long *force, long long n_steps, int nz, double qa, double H, double *coef,
                             cudaStream_t s) {
  if (n_steps <= 0) return cudaSuccess;
  const long long threads = n_steps * 8;
  k_coefficients<<<(unsigned)((threads + 255) / 256), 256, 0, s>>>(force, n_steps, nz, qa, H, coef);
  return cudaGetLastError();
}
cudaError_t aux_coef_stats(const double *coef, long long n_steps, long long n_spin, double *stats, cudaStream_t s) {
  k_coef_stats<<<kStatBlocks, kStatThreads, 0, s>>>(coef, n_steps, n_spin, stats);
  return cudaGetLastError();
}

// ---------------------------------------------------------------- recirculation area
// export3d.py:169-184 on the every-2nd-cell mean field (lbm3d.py:412): the box
// of cells (2 (i0 + i), 2 j, 2 k), i < I, j < J, k < K, holds u_x of the time
// mean (sums / n_acc in float64, rounded to float) or 0.05 at non-fluid cells,
// divided by U_H in float; level k = 0 takes level 1's value; one 3-point box
// blur with edge clamping along i, then j, then k ((a + b) + c, then / 3, in
// float); the reverse-flow cells are those left below zero.  Built without FMA
// contraction (the file's --fmad=false) and with explicitly rounded operations,
// so the count equals the float32 NumPy restatement's.  Scratch layout
// [k][j][i].
struct RecircBox {
  int i0, I, J, K;
};
__global__ void k_recirc_gather(Geom g, RecircBox b, const double *acc, double n, const uint8_t *flag, float uh,
                                float *out) {
  const long long e = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (e >= (long long)b.I * b.J * b.K) return;
  const int i = (int)(e % b.I), j = (int)((e / b.I) % b.J), k = (int)(e / ((long long)b.I * b.J));
  const int x = 2 * (b.i0 + i), y = 2 * j, z = 2 * (k == 0 ? 1 : k);
  const size_t c = ((size_t)z * g.ny + y) * g.pitch + x;
  const float v = flag[c] != 0 ? 0.05f : __double2float_rn(__ddiv_rn(acc[(size_t)g.plane + c], n));
  out[e] = __fdiv_rn(v, uh);
}
// AXIS 0: i, 1: j, 2: k.  With COUNT the result is not stored: each cell below
// zero adds one to *count (one atomic per warp).
template <int AXIS, bool COUNT>
__global__ void k_recirc_blur(RecircBox b, const float *in, float *out, unsigned long long *count) {
  const long long e = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  const long long n = (long long)b.I * b.J * b.K;
  bool neg = false;
  if (e < n) {
    const int i = (int)(e % b.I), j = (int)((e / b.I) % b.J), k = (int)(e / ((long long)b.I * b.J));
    const int at = AXIS == 0 ? i : AXIS == 1 ? j : k;
    const int len = AXIS == 0 ? b.I : AXIS == 1 ? b.J : b.K;
    const long long step = AXIS == 0 ? 1 : AXIS == 1 ? (long long)b.I : (long long)b.I * b.J;
    const float lo = in[e - (at > 0 ? step : 0)], mid = in[e], hi = in[e + (at + 1 < len ? step : 0)];
    const float v = __fdiv_rn(__fadd_rn(__fadd_rn(lo, mid), hi), 3.0f);
    if (COUNT) neg = v < 0.0f;
    else out[e] = v;
  }
  if (COUNT) {
    const unsigned m = __ballot_sync(0xffffffffu, neg);
    if ((threadIdx.x & 31) == 0 && m) atomicAdd(count, (unsigned long long)__popc(m));
  }
}
cudaError_t aux_recirc_count(const Geom &g, int i0, int I, int J, int K, const double *acc, long long n_acc,
                             const uint8_t *flag, float uh, float *scratch, long long *count, cudaStream_t s) {
  const RecircBox b{i0, I, J, K};
  const long long n = (long long)I * J * K;
  float *a = scratch, *t = scratch + n;
  unsigned long long *cnt = reinterpret_cast<unsigned long long *>(count);
  cudaError_t e = cudaMemsetAsync(cnt, 0, sizeof(*cnt), s);
  if (e != cudaSuccess) return e;
  const unsigned blocks = (unsigned)((n + 255) / 256);
  k_recirc_gather<<<blocks, 256, 0, s>>>(g, b, acc, (double)(n_acc > 0 ? n_acc : 1), flag, uh, a);
  k_recirc_blur<0, false><<<blocks, 256, 0, s>>>(b, a, t, nullptr);
  k_recirc_blur<1, false><<<blocks, 256, 0, s>>>(b, t, a, nullptr);
  k_recirc_blur<2, true><<<blocks, 256, 0, s>>>(b, a, nullptr, cnt);
  return cudaGetLastError();
}

// ---------------------------------------------------------------- viewer payload
// k_slice_xz / k_slice_xy (lbm3d.py:191-200): the macro field u (device layout
// [4][nz][ny][pitch]) at y = y0 or z = z0, written in the reference layout
// out[c][x][z] / out[c][x][y].
__global__ void k_slice_xz(Geom g, const float *u, int y0, float *out) {
  const long long k = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= 4ll * g.nx * g.nz) return;
  const int z = (int)(k % g.nz), x = (int)((k / g.nz) % g.nx), c = (int)(k / ((long long)g.nz * g.nx));
  out[k] = u[(size_t)c * g.plane + ((size_t)z * g.ny + y0) * g.pitch + x];
}
__global__ void k_slice_xy(Geom g, const float *u, int z0, float *out) {
  const long long k = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= 4ll * g.nx * g.ny) return;
  const int y = (int)(k % g.ny), x = (int)((k / g.ny) % g.nx), c = (int)(k / ((long long)g.ny * g.nx));
  out[k] = u[(size_t)c * g.plane + ((size_t)z0 * g.ny + y) * g.pitch + x];
}

// Q-criterion at one cell (q_at, lbm3d.py:203-222): -1/2 A_ij A_ji of the
// central-difference velocity gradient, 0 next to any non-fluid cell; y
// periodic.  Float32 in the reference's evaluation order (this translation
// unit is compiled without multiply-add contraction).
__device__ float q_at(const Geom &g, const float *u, const uint8_t *flag, int x, int y, int z) {
  const int yp = (y + 1) % g.ny, ym = (y - 1 + g.ny) % g.ny;
  auto fl = [&](int xx, int yy, int zz) { return flag[((size_t)zz * g.ny + yy) * g.pitch + xx]; };
  if (fl(x, y, z) != 0 || fl(x + 1, y, z) != 0 || fl(x - 1, y, z) != 0 || fl(x, yp, z) != 0 || fl(x, ym, z) != 0 ||
      fl(x, y, z + 1) != 0 || fl(x, y, z - 1) != 0)
    return 0.0f;
  auto U = [&](int c, int xx, int yy, int zz) { return u[(size_t)c * g.plane + ((size_t)zz * g.ny + yy) * g.pitch + xx]; };
  const float a11 = 0.5f * (U(1, x + 1, y, z) - U(1, x - 1, y, z));
  const float a12 = 0.5f * (U(1, x, yp, z) - U(1, x, ym, z));
  const float a13 = 0.5f * (U(1, x, y, z + 1) - U(1, x, y, z - 1));
  const float a21 = 0.5f * (U(2, x + 1, y, z) - U(2, x - 1, y, z));
  const float a22 = 0.5f * (U(2, x, yp, z) - U(2, x, ym, z));
  const float a23 = 0.5f * (U(2, x, y, z + 1) - U(2, x, y, z - 1));
  const float a31 = 0.5f * (U(3, x + 1, y, z) - U(3, x - 1, y, z));
  const float a32 = 0.5f * (U(3, x, yp, z) - U(3, x, ym, z));
  const float a33 = 0.5f * (U(3, x, y, z + 1) - U(3, x, y, z - 1));
  return -0.5f * (a11 * a11 + a22 * a22 + a33 * a33 + 2.0f * (a12 * a21 + a13 * a31 + a23 * a32));
}

// k_qcoarse (lbm3d.py:225-238): max of max(Q, 0) over ds^3 blocks of the crop
// starting at (x0, 0, 0).  A block of threads takes `nb` neighbouring output
// voxels of one (j, k): its threads run along x over their nb * ds cells, so the
// 25 loads of a cell are coalesced (one thread per voxel, with neighbouring
// threads ds levels apart, took 597 us for the 120x53x33 frame of an
// 800x160x321 grid; this takes 72 us), and the maxima of a voxel meet in
// shared memory as integers (they are not negative).
constexpr int kQThreads = 128;
__global__ void __launch_bounds__(kQThreads) k_qcoarse(Geom g, const float *u, const uint8_t *flag, int x0, int ds,
                                                       int di, int dj, int dk, int nb, float *out) {
  __shared__ int best[kQThreads];
  const unsigned nbx = (unsigned)((di + nb - 1) / nb), jk = blockIdx.x / nbx;
  const int i0 = (int)(blockIdx.x - jk * nbx) * nb;
  const int j = (int)(jk / (unsigned)dk), k = (int)(jk - (unsigned)j * dk);
  const int n = min(nb, di - i0);                            // voxels here (nb <= kQThreads)
  if ((int)threadIdx.x < n) best[threadIdx.x] = 0;
  __syncthreads();
  for (int t = threadIdx.x; t < n * ds; t += kQThreads) {
    const int x = x0 + i0 * ds + t;
    float m = 0.0f;
    if (x >= 1 && x < g.nx - 1)
      for (int c = 0; c < ds; ++c) {
        const int z = k * ds + c;
        if (z < 1 || z >= g.nz - 1) continue;
        for (int b = 0; b < ds; ++b) m = fmaxf(m, q_at(g, u, flag, x, j * ds + b, z));
      }
    if (m > 0.0f) atomicMax(&best[t / ds], __float_as_int(m));
  }
  __syncthreads();
  if ((int)threadIdx.x < n) out[((long long)(i0 + (int)threadIdx.x) * dj + j) * dk + k] = __int_as_float(best[threadIdx.x]);
}

// The planes of a snapshot (lbm3d.py:371-375): ux, uy, uz at y = y0 as
// [3][nx][nz], then at z = z0 as [3][nx][ny], rounded to half precision.  One
// component per blockIdx.y: a plane of one has fewer cells than 2^31, three may not.
__global__ void k_snapshot(Geom g, const float *u, int y0, int z0, __half *out) {
  const long long e = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  const long long xz = (long long)g.nx * g.nz, xy = (long long)g.nx * g.ny;
  if (e >= xz + xy) return;
  const bool side = e < xz;
  const uint32_t c = blockIdx.y, r = (uint32_t)(side ? e : e - xz), n = (uint32_t)(side ? g.nz : g.ny);
  const uint32_t x = r / n, w = r - x * n;
  const size_t row = side ? (size_t)w * g.ny + y0 : (size_t)z0 * g.ny + w;
  __half *plane = side ? out + c * xz : out + 3 * xz + c * xy;
  plane[r] = __float2half_rn(u[(size_t)(c + 1) * g.plane + row * g.pitch + x]);
}

// The log quantisation of a Q frame (lbm3d.py:317-318) by its level boundaries:
// out = how many of the 255 ascending levels are <= min(q * scale, qmax).
__global__ void __launch_bounds__(256) k_quantise(const float *q, long long n, float scale, float qmax,
                                                  const float *levels, uint8_t *out) {
  __shared__ float lev[256];
  lev[threadIdx.x] = threadIdx.x < 255 ? levels[threadIdx.x] : __int_as_float(0x7f800000);
  __syncthreads();
  const long long e = (long long)blockIdx.x * 256 + threadIdx.x;
  if (e >= n) return;
  const float v = fminf(__fmul_rn(q[e], scale), qmax);
  int lo = 0;                                                // levels[0..lo) <= v
#pragma unroll
  for (int step = 128; step > 0; step >>= 1)
    if (lev[lo + step - 1] <= v) lo += step;
  out[e] = (uint8_t)lo;
}

cudaError_t aux_slice_xz(const Geom &g, const float *u, int y0, float *out, cudaStream_t s) {
  const long long n = 4ll * g.nx * g.nz;
  k_slice_xz<<<(unsigned)((n + 255) / 256), 256, 0, s>>>(g, u, y0, out);
  return cudaGetLastError();
}
cudaError_t aux_slice_xy(const Geom &g, const float *u, int z0, float *out, cudaStream_t s) {
  const long long n = 4ll * g.nx * g.ny;
  k_slice_xy<<<(unsigned)((n + 255) / 256), 256, 0, s>>>(g, u, z0, out);
  return cudaGetLastError();
}
cudaError_t aux_qcoarse(const Geom &g, const float *u, const uint8_t *flag, int x0, int ds, int di, int dj, int dk,
                        float *out, cudaStream_t s) {
  if ((long long)di * dj * dk == 0) return cudaSuccess;
  const int nb = ds < kQThreads ? kQThreads / ds : 1;        // as many voxels as a block has cells for
  const long long blocks = (long long)((di + nb - 1) / nb) * dj * dk;
  k_qcoarse<<<(unsigned)blocks, kQThreads, 0, s>>>(g, u, flag, x0, ds, di, dj, dk, nb, out);
  return cudaGetLastError();
}
cudaError_t aux_snapshot(const Geom &g, const float *u, int y0, int z0, void *out, cudaStream_t s) {
  const long long n = (long long)g.nx * ((long long)g.nz + g.ny);
  k_snapshot<<<dim3((unsigned)((n + 255) / 256), 3), 256, 0, s>>>(g, u, y0, z0, static_cast<__half *>(out));
  return cudaGetLastError();
}
cudaError_t aux_quantise(const float *q, long long n, float scale, float qmax, const float *levels, uint8_t *out,
                         cudaStream_t s) {
  if (n <= 0) return cudaSuccess;
  k_quantise<<<(unsigned)((n + 255) / 256), 256, 0, s>>>(q, n, scale, qmax, levels, out);
  return cudaGetLastError();
}

}  // namespace sw
