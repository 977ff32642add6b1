// yz_pairs.cu -- inverse (y,z) transform of two neighbouring window planes x, x + 1 of a rotation at
// once, with the window minimum: the planes are the two members of every register pair (packed FP32,
// pair_fft.cuh), so a butterfly's loads, stores, address arithmetic, twiddles and issue slots are
// shared by both. The arithmetic per plane is that of the single-plane kernels (k_yz_inv_argmin,
// k_yz_octet): radix stages R1 and 8 over the digit-reversed positions of y, rows (2p, 2p + 1)
// packed as one complex line over z, keys of (energy, linear index); results are bit-identical.
//
// B holds the two planes' values of a spectral column side by side (re x, re x+1, im x, im x+1: 16
// bytes), either as plane pairs (FP32 x pass) or as plane quads (one-column Hankel x pass, whose
// stores must fill 32-byte sectors).
//
// CTA = a rotation and a part of its plane pairs, looped. An octet of 8 lanes owns a line (a kz
// column for y, a row pair for z): lane t takes block t in the first stage and the groups np = t,
// t + 8, ... in the second; the exchange between them goes through the line's own storage in the
// plane buffer, with __syncwarp only, so that a pair of planes has two CTA barriers (y -> z, z -> the
// next y). Banks, in 16-byte units of which a quarter-warp must hit 8 different ones: in the y pass a
// quarter-warp is 4 neighbouring columns of 2 blocks or groups (its loads from B then fall in 2 lines
// instead of 8, which cost 25 L1 wavefronts each), rows and blocks lying 4 mod 8 units apart; in the
// z pass it is one octet, a line's positions swizzled within its row pair.
//
// Measured on a B200 against the single-plane kernels (two smallest keys, plane quads; ms per 1e5
// rotations): 64^3 42.9 -> 31.7, 96^3 259 -> 132, 128^3 672 -> 362; FP32 form (plane pairs): 64^3 30.2 ->
// 28.2, 96^3 221 -> 131, 128^3 526 -> 328. About 2.9 k warp instructions per plane at 64^3 (7.3 k before);
// what bounds it now is the shared-memory and L1 data path beside the CTA barriers.
//
// The smallest key (two smallest: TOP2) is carried over the CTA's planes and reduced once at its
// end; a bound in shared memory, lowered by each warp that sees smaller energies, keeps all but a
// few lanes from building keys.
#include <cuda_runtime.h>
#include <stdint.h>

#include <algorithm>

#include "cdk_internal.h"
#include "pair_fft.cuh"
#include "window_keys.cuh"

namespace cdk {
namespace {

// Threads per CTA: octets for all kz columns in one round. CTAs per SM: at 64^3 four (56 registers)
// measured 33.5 ms per 1e5 rotations against 31.7 with three (72 registers)
template <int N>
struct YzShape {
  static constexpr int NZH = N / 2 + 1;
  static constexpr int T = (NZH * 8 + 31) / 32 * 32;  // 160, 288, 416, 544
  static constexpr int CTAS = N == 32 ? 6 : N == 64 ? 3 : N == 96 ? 2 : 1;
  // units of 16 bytes between rows, and between blocks of R1 rows: both 4 mod 8
  static constexpr int ROW = (NZH + 3) / 8 * 8 + 4;
  static constexpr int BLOCK = (N / 8) * ROW + 4;
  static constexpr size_t SMEM = sizeof(float4) * ((N / 8) * 7 + 8 * BLOCK);
  static_assert(ROW >= NZH && ROW % 8 == 4 && BLOCK % 8 == 4, "row and block strides");
};

// Twiddle products v[k] conj(w^(np k)), k = 1..7, of both planes; table [np][k - 1] of (c, c, s, s)
template <int N>
__device__ __forceinline__ void yz_twiddle(cpair* v, const float4* tw, int np) {
#pragma unroll
  for (int k = 1; k < 8; ++k) {
    const float4 w = tw[np * 7 + k - 1];
    const pair_t c = pk(w.x, w.y), s = pk(w.z, w.w);
    const float2 y = unpk(v[k].y), t = unpk(p_mul(v[k].x, s));
    v[k].x = p_fma(v[k].x, c, p_mul(v[k].y, s));
    v[k].y = pk(__fmaf_rn(y.x, w.x, -t.x), __fmaf_rn(y.y, w.y, -t.y));
  }
}

// min that keeps a NaN
__device__ __forceinline__ float min_nan(float a, float b) {
  float r;
  asm("min.NaN.f32 %0, %1, %2;" : "=f"(r) : "f"(a), "f"(b));
  return r;
}

template <int N, bool TOP2, bool QUADS>
__global__ void __launch_bounds__(YzShape<N>::T, YzShape<N>::CTAS) k_yz_pairs(const __grid_constant__ WaveArgs a) {
  constexpr int NZH = N / 2 + 1, NCOL = N * NZH, R1 = N / 8, T = YzShape<N>::T;
  constexpr int ROW = YzShape<N>::ROW, BLOCK = YzShape<N>::BLOCK;
  constexpr int NG = (R1 + 7) / 8;  // second-stage groups per lane
  static_assert(T / 8 >= N / 2, "an octet per row pair");
  extern __shared__ __align__(16) unsigned char smem_raw[];
  float4* tw = reinterpret_cast<float4*>(smem_raw);
  float4* O = tw + R1 * 7;
  // order_key of an energy that at least one (TOP2: two) of the CTA's values so far does not exceed:
  // a value strictly above it cannot enter
  __shared__ unsigned int s_bound;
  const int r = blockIdx.y, part = blockIdx.x, parts = gridDim.x;
  const RotRec* rec = a.rec + r;
  if (!rec->valid) return;
  const int Wx = rec->W[0], Wy = rec->W[1], Wz = rec->W[2];
  const int pairs = (Wx + 1) / 2, npairs = (Wy + 1) / 2;
  const int tid = threadIdx.x, lane = tid & 31;
  // y: octets of lanes 4 apart, so that a quarter-warp holds 4 neighbouring columns of 2 blocks
  const int ty = lane >> 2, gy = (tid >> 5) * 4 + (lane & 3);
  const int t = tid & 7, g = tid >> 3;  // z: octets of consecutive lanes
  for (int i = tid; i < R1 * 7; i += T) {
    const float2 w = a.tw[(i / 7) * (i % 7 + 1)];
    tw[i] = make_float4(w.x, w.x, w.y, w.y);
  }
  if (tid == 0) s_bound = order_key(INFINITY);
  auto ld = [](const float4* p) {
    const float4 f = *p;
    return cpair{pk(f.x, f.y), pk(f.z, f.w)};
  };
  auto st = [](float4* p, cpair v) {
    const float2 x = unpk(v.x), y = unpk(v.y);
    *p = make_float4(x.x, x.y, y.x, y.y);
  };
  constexpr int BS = QUADS ? 2 * b_quad_rots(N) : 1;  // float4 per column
  const bool has_col = gy < NZH;
  const int c0 = ty * R1 * NZH + (has_col ? gy : 0);  // column of the block's first row
  const float4* src0 = reinterpret_cast<const float4*>(a.B) +
                       (QUADS ? b_quad_index<N>(r, c0) : (size_t)r * (N / 2) * NCOL + c0);
  float4* const col = O + (has_col ? gy : 0);
  const int sw = R1 % 8 == 0 ? t : t >> 1;  // swizzle of a line's positions t R1 + m -> t R1 + (m ^ sw)
  const float inv = 1.0f / (float)((double)N * N * N);
  unsigned long long best = ~0ull, best2 = ~0ull;
  __syncthreads();
#pragma unroll 1
  for (int p = part; p < pairs; p += parts) {
    // y of column gy: first stage (radix R1, no twiddles) over block ty's positions
    if (has_col) {
      const float4* src = QUADS ? src0 + (size_t)(p >> 1) * (NCOL * BS) + (p & 1) : src0 + (size_t)p * NCOL;
      cpair v[R1];
#pragma unroll
      for (int j = 0; j < R1; ++j) v[j] = ld(src + j * NZH * BS);
      PairRadix<R1, +1>::run(v);
#pragma unroll
      for (int j = 0; j < R1; ++j) st(col + ty * BLOCK + j * ROW, v[j]);
    }
    __syncwarp();
    // second stage (radix 8): the groups' 8 positions become the natural rows np + R1 j in place
#pragma unroll
    for (int q = 0; q < NG; ++q) {
      const int np = ty + 8 * q;
      if (has_col && np < R1) {
        cpair u[8];
#pragma unroll
        for (int b = 0; b < 8; ++b) u[b] = ld(col + b * BLOCK + np * ROW);
        yz_twiddle<N>(u, tw, np);
        PairRadix<8, +1>::run(u);
#pragma unroll
        for (int j = 0; j < 8; ++j) st(col + j * BLOCK + np * ROW, u[j]);
      }
    }
    __syncthreads();
    // z of row pair g: rows (2g, 2g + 1) as one complex line with its Hermitian extension
    if ((g & ~3) < npairs) {  // warp-uniform: one of the warp's octets has a row pair
      const bool act = g < npairs;
      const int y = 2 * (act ? g : 0);
      float4* const A = O + (y / R1) * BLOCK + (y % R1) * ROW;
      const float4* const Bv = A + ROW;
      {
        cpair z[R1];
#pragma unroll
        for (int j = 0; j < R1; ++j) {
          const int k = t + 8 * j;
          const int m = j < R1 / 2 ? k : N - k;
          const cpair ak = ld(A + m), bk = ld(Bv + m);
          if (j < R1 / 2) z[j] = cpair{p_sub(ak.x, bk.y), p_add(ak.y, bk.x)};
          else z[j] = cpair{p_add(ak.x, bk.y), p_sub(bk.x, ak.y)};
          if ((j == 0 || j == R1 / 2) && t == 0) z[j] = cpair{ak.x, bk.x};  // k = 0, N / 2
        }
        __syncwarp();  // the octet has read its rows: their slots become the exchange
        PairRadix<R1, +1>::run(z);
        if (act) {
#pragma unroll
          for (int j = 0; j < R1; ++j) st(A + t * R1 + (j ^ sw), z[j]);
        }
        __syncwarp();
      }
      const int x = 2 * p;
      const bool row1 = y + 1 < Wy, plane1 = x + 1 < Wx;
#pragma unroll
      for (int q = 0; q < NG; ++q) {
        const int np = t + 8 * q;
        const bool on = act && np < R1;
        cpair u[8];
#pragma unroll
        for (int b = 0; b < 8; ++b) u[b] = ld(A + b * R1 + ((on ? np : 0) ^ (R1 % 8 == 0 ? b : b >> 1)));
        yz_twiddle<N>(u, tw, on ? np : 0);
        PairRadix<8, +1>::run(u);
        // energies of z = np + R1 j: rows y (real parts) and y + 1 (imaginary parts), planes x, x + 1
        float lo = INFINITY;
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          if (on && np + R1 * j < Wz) {
            const float2 e0 = unpk(u[j].x), e1 = unpk(u[j].y);
            float m = row1 ? min_nan(e0.x, e1.x) : e0.x;
            if (plane1) m = min_nan(m, row1 ? min_nan(e0.y, e1.y) : e0.y);
            lo = min_nan(lo, m);
          }
        }
        lo *= inv;
        const unsigned int seen = *(volatile unsigned int*)&s_bound;
        float bound = key_to_float(seen);
        if (__any_sync(0xffffffffu, on && !(lo > bound))) {
          // the bound that this warp's lines give: two (TOP2) lanes hold an energy no larger
          const unsigned int k = on ? order_key(lo) : 0xffffffffu;
          unsigned int m = __reduce_min_sync(0xffffffffu, k);
          if (TOP2 && __popc(__ballot_sync(0xffffffffu, k == m)) < 2)
            m = __reduce_min_sync(0xffffffffu, k == m ? 0xffffffffu : k);
          if (m < seen) {
            bound = key_to_float(m);
            if (lane == 0) atomicMin(&s_bound, m);
          }
          if (on && !(lo > bound)) {
            const unsigned int lin = (unsigned int)((x * N + y) * N + np);
            auto keep = [&](float e, unsigned int at) {
              e *= inv;
              if (e > bound) return;
              const unsigned long long key = ((unsigned long long)order_key(e) << 32) | at;
              if constexpr (TOP2) top2_insert(key, best, best2);
              else best = key < best ? key : best;
            };
#pragma unroll
            for (int j = 0; j < 8; ++j) {
              if (np + R1 * j < Wz) {
                const float2 e0 = unpk(u[j].x), e1 = unpk(u[j].y);
                const unsigned int at = lin + (unsigned int)(R1 * j);
                keep(e0.x, at);
                if (row1) keep(e1.x, at + N);
                if (plane1) {
                  keep(e0.y, at + N * N);
                  if (row1) keep(e1.y, at + N * N + N);
                }
              }
            }
          }
        }
      }
    }
    __syncthreads();
  }
  // the CTA's smallest keys; the plane buffer is free
  warp_keep_min<TOP2>(best, best2);
  unsigned long long* s_best = reinterpret_cast<unsigned long long*>(O);
  constexpr int NW = T / 32;
  if ((tid & 31) == 0) {
    s_best[tid >> 5] = best;
    if constexpr (TOP2) s_best[NW + (tid >> 5)] = best2;
  }
  __syncthreads();
  if (tid < 32) {
    best = tid < NW ? s_best[tid] : ~0ull;
    if constexpr (TOP2) best2 = tid < NW ? s_best[NW + tid] : ~0ull;
    warp_keep_min<TOP2>(best, best2);
    if (tid == 0) {
      atomicMin(a.keys + r, best);
      if constexpr (TOP2) {
        a.keys2[((size_t)r * N + part) * 2] = best;
        a.keys2[((size_t)r * N + part) * 2 + 1] = best2;
      }
    }
  }
}

// CTAs per rotation: about 16 rounds of CTAs over the device, so that the last one costs little,
// each with at least two plane pairs
template <int N>
int yz_parts(int nrot) {
  const long want = 148l * YzShape<N>::CTAS * 16;
  return (int)std::max<long>(1, std::min<long>(N / 4, (want + nrot - 1) / nrot));
}

template <int N>
cudaError_t launch_t(const WaveArgs& a, cudaStream_t s) {
  const bool quads = a.bpairs == 4;
  auto kern = a.keys2 ? (quads ? k_yz_pairs<N, true, true> : k_yz_pairs<N, true, false>)
                      : (quads ? k_yz_pairs<N, false, true> : k_yz_pairs<N, false, false>);
  const cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)YzShape<N>::SMEM);
  if (e != cudaSuccess) return e;
  kern<<<dim3(yz_parts<N>(a.nrot), a.nrot), YzShape<N>::T, YzShape<N>::SMEM, s>>>(a);
  return cudaGetLastError();
}

}  // namespace

int yz_pairs_key_slots(const WaveArgs& a) {
  switch (a.n) {
    case 32: return yz_parts<32>(a.nrot);
    case 64: return yz_parts<64>(a.nrot);
    case 96: return yz_parts<96>(a.nrot);
    default: return yz_parts<128>(a.nrot);
  }
}

cudaError_t launch_yz_pairs(const WaveArgs& a, cudaStream_t s) {
  if (a.bpairs != 2 && a.bpairs != 4) return cudaErrorInvalidValue;
  switch (a.n) {
    case 32: return launch_t<32>(a, s);
    case 64: return launch_t<64>(a, s);
    case 96: return launch_t<96>(a, s);
    case 128: return launch_t<128>(a, s);
    default: return cudaErrorInvalidValue;
  }
}

}  // namespace cdk
