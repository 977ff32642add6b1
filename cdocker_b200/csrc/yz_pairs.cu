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
// k_yz_pairs (k_yz_quads, for plane quads at n <= 64, is described there): CTA = a rotation and a part of
// its plane pairs, looped. An octet of 8 lanes owns a line (a kz
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
  static constexpr size_t SMEM = sizeof(float2) * (N / 8) * 7 + sizeof(float4) * 8 * BLOCK;
  static_assert(ROW >= NZH && ROW % 8 == 4 && BLOCK % 8 == 4, "row and block strides");
};

// Twiddle products v[k] conj(w^(np k)), k = 1..7, of both planes; table [np][k - 1] of (c, s): loads of 8
// bytes and not the doubled pairs (c, c, s, s) cost half the wavefronts (inverse pass 96^3 FP32 1.31 ->
// 1.25 ms, 128^3 3.38 -> 3.21)
template <int N>
__device__ __forceinline__ void yz_twiddle(cpair* v, const float2* tw, int np) {
#pragma unroll
  for (int k = 1; k < 8; ++k) {
    const float2 w = tw[np * 7 + k - 1];
    const pair_t c = pk(w.x, w.x), s = pk(w.y, w.y);
    const float2 y = unpk(v[k].y), t = unpk(p_mul(v[k].x, s));
    v[k].x = p_fma(v[k].x, c, p_mul(v[k].y, s));
    v[k].y = pk(__fmaf_rn(y.x, w.x, -t.x), __fmaf_rn(y.y, w.x, -t.y));
  }
}

// min that keeps a NaN
__device__ __forceinline__ float min_nan(float a, float b) {
  float r;
  asm("min.NaN.f32 %0, %1, %2;" : "=f"(r) : "f"(a), "f"(b));
  return r;
}

// Energies of z = np + R1 j, j < 8, of rows y (real parts) and y + 1 (imaginary parts) and planes x, x + 1,
// into the thread's smallest key (TOP2: two smallest). Called by whole warps; on: the lane has values.
// s_bound: order_key of an energy that at least one (TOP2: two) of the CTA's values so far does not
// exceed: a value strictly above it cannot enter.
template <int N, bool TOP2>
__device__ __forceinline__ void yz_keep(const cpair* u, bool on, int np, int x, int y, bool row1, bool plane1, int Wz,
                                        float inv, int lane, unsigned int* s_bound, unsigned long long& best,
                                        unsigned long long& best2) {
  constexpr int R1 = N / 8;
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
  const unsigned int seen = *(volatile unsigned int*)s_bound;
  float bound = key_to_float(seen);
  if (__any_sync(0xffffffffu, on && !(lo > bound))) {
    // the bound that this warp's lines give: two (TOP2) lanes hold an energy no larger
    const unsigned int k = on ? order_key(lo) : 0xffffffffu;
    unsigned int m = __reduce_min_sync(0xffffffffu, k);
    if (TOP2 && __popc(__ballot_sync(0xffffffffu, k == m)) < 2)
      m = __reduce_min_sync(0xffffffffu, k == m ? 0xffffffffu : k);
    if (m < seen) {
      bound = key_to_float(m);
      if (lane == 0) atomicMin(s_bound, m);
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

// The CTA's smallest keys, reduced in the plane buffer (free by now) and stored
template <int N, int NW, bool TOP2>
__device__ __forceinline__ void yz_store(const WaveArgs& a, int r, int part, void* buffer, unsigned long long best,
                                         unsigned long long best2) {
  const int tid = threadIdx.x;
  warp_keep_min<TOP2>(best, best2);
  unsigned long long* s_best = static_cast<unsigned long long*>(buffer);
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

template <int N, bool TOP2, bool QUADS>
__global__ void __launch_bounds__(YzShape<N>::T, YzShape<N>::CTAS) k_yz_pairs(const __grid_constant__ WaveArgs a) {
  constexpr int NZH = N / 2 + 1, NCOL = N * NZH, R1 = N / 8, T = YzShape<N>::T;
  constexpr int ROW = YzShape<N>::ROW, BLOCK = YzShape<N>::BLOCK;
  constexpr int NG = (R1 + 7) / 8;  // second-stage groups per lane
  static_assert(T / 8 >= N / 2 && R1 * 7 % 2 == 0, "an octet per row pair; the plane buffer aligned");
  extern __shared__ __align__(16) unsigned char smem_raw[];
  float2* tw = reinterpret_cast<float2*>(smem_raw);
  float4* O = reinterpret_cast<float4*>(tw + R1 * 7);
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
  for (int i = tid; i < R1 * 7; i += T) tw[i] = a.tw[(i / 7) * (i % 7 + 1)];
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
        yz_keep<N, TOP2>(u, on, np, x, y, row1, plane1, Wz, inv, lane, &s_bound, best, best2);
      }
    }
    __syncthreads();
  }
  yz_store<N, T / 32, TOP2>(a, r, part, O, best, best2);
}

// Plane quads of single rotations (n <= 64: the one-column Hankel x pass): a CTA loads a quad's four
// planes, contiguous in B, into its plane buffer with eight bulk copies (one per row, issued lane by lane,
// kept a warp busy for thousands of cycles: 64^3 28.2 -> QNOW), so no load goes through the
// LSU -- there a 16-byte load, whose lanes took half of 32 sectors in 8 or more lines, cost 24 L1 cycles,
// 42 % of the L1 time at 64^3 -- and transforms both pairs in place between the same two barriers. Three
// CTAs per SM at 64^3 hide each other's copies. Units of 16 bytes (one pair of one column) lie column by
// column, pair by pair; a quarter-warp is 2 columns x 2 pairs x 2 blocks in y and 4 positions x 2 pairs in
// z, 8 different banks with the strides below. ms per 1e5 rotations (two smallest
// keys): 64^3 33.3 -> 28.8, 32^3 5.6 -> 4.4 against k_yz_pairs over the same quads; over plane pairs (FP32 x
// pass, two shorter copies per row) the same scheme lost, 30.6 against 28.0 at 64^3.
template <int N>
struct YzQuadShape {
  static constexpr int NZH = N / 2 + 1;
  static constexpr int T = N == 32 ? 160 : 288;
  static constexpr int CTAS = N == 32 ? 6 : 3;
  static constexpr int ROW = 2 * NZH;              // 2 mod 8: a block of N / 8 rows as it lies in B
  static constexpr int BLOCK = (N / 8) * ROW + 4;  // 4 mod 8
  static constexpr size_t SMEM = sizeof(float2) * (N / 8) * 7 + sizeof(float4) * 8 * BLOCK;
  static_assert(ROW % 8 == 2 && BLOCK % 8 == 4, "row and block strides");
  static_assert(2 * ROW >= 2 * N, "a row pair holds a line of both pairs");
};

constexpr long kYzWaitLimit = 1l << 22;

template <int N, bool TOP2>
__global__ void __launch_bounds__(YzQuadShape<N>::T, YzQuadShape<N>::CTAS) k_yz_quads(const __grid_constant__ WaveArgs a) {
  using S = YzQuadShape<N>;
  constexpr int NZH = S::NZH, R1 = N / 8, T = S::T, NW = T / 32, ROW = S::ROW, BLOCK = S::BLOCK;
  static_assert(R1 <= 8 && b_quad_rots(N) == 1, "one second-stage group per lane, rotations apart");
  extern __shared__ __align__(16) unsigned char smem_raw[];
  float2* tw = reinterpret_cast<float2*>(smem_raw);
  float4* O = reinterpret_cast<float4*>(tw + R1 * 7);
  __shared__ unsigned int s_bound;
  __shared__ __align__(8) uint64_t s_full;
  __shared__ int s_fail;
  const int r = blockIdx.y, part = blockIdx.x, parts = gridDim.x;
  const RotRec* rec = a.rec + r;
  if (!rec->valid) return;
  const int Wx = rec->W[0], Wy = rec->W[1], Wz = rec->W[2];
  const int quads = (Wx + 3) / 4, npairs = (Wy + 1) / 2;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const uint32_t full = (uint32_t)__cvta_generic_to_shared(&s_full);
  for (int i = tid; i < R1 * 7; i += T) tw[i] = a.tw[(i / 7) * (i % 7 + 1)];
  if (tid == 0) {
    s_bound = order_key(INFINITY);
    s_fail = 0;
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(full));
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  auto ld = [](const float4* p) {
    const float4 f = *p;
    return cpair{pk(f.x, f.y), pk(f.z, f.w)};
  };
  auto st = [](float4* p, cpair v) {
    const float2 x = unpk(v.x), y = unpk(v.y);
    *p = make_float4(x.x, x.y, y.x, y.y);
  };
  // one thread: the quad's eight blocks into the plane buffer
  auto load_quad = [&](int p) {
    constexpr uint32_t bytes = R1 * NZH * 32;
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%1], %0;" ::"r"(bytes * 8), "r"(full) : "memory");
    const float4* src = reinterpret_cast<const float4*>(a.B) + b_quad_index<N>(r, 0) + (size_t)p * (N * NZH * 2);
#pragma unroll 1
    for (int b = 0; b < 8; ++b)
      asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                       (uint32_t)__cvta_generic_to_shared(O + b * BLOCK)),
                   "l"(src + b * (R1 * ROW)), "r"(bytes), "r"(full)
                   : "memory");
  };
  auto wait_quad = [&](uint32_t parity) {
    for (long i = 0; i < kYzWaitLimit; ++i) {
      uint32_t done;
      asm volatile(
          "{\n\t.reg .pred p;\n\t"
          "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
          "selp.u32 %0, 1, 0, p;\n\t}"
          : "=r"(done)
          : "r"(full), "r"(parity)
          : "memory");
      if (done) return;
      if (i > 32) {
        if (*(volatile int*)&s_fail) return;  // another thread gave up
        __nanosleep(40);
      }
    }
    *(volatile int*)&s_fail = 1;
  };
  const int q = lane & 1;                          // the lane's pair of the quad
  const int ty = lane >> 2;                        // y: block; columns 2u, 2u + 1 of unit u
  // and group: the quarter-warp's two groups 2 rows, 4 units mod 8, apart
  const int np = (ty & 4) | ((ty & 1) << 1) | ((ty >> 1) & 1);
  const int t = (lane >> 1) & 7, g2 = lane >> 4;   // z: place in the line; row pairs 2w, 2w + 1 of unit w
  constexpr int SW = R1 - 1;  // swizzle of a line's positions b R1 + m -> b R1 + (m ^ (b & SW))
  const float inv = 1.0f / (float)((double)N * N * N);
  unsigned long long best = ~0ull, best2 = ~0ull;
  __syncthreads();
  if (tid == 0 && part < quads) load_quad(part);
  uint32_t parity = 0;
#pragma unroll 1
  for (int p = part; p < quads; p += parts, parity ^= 1u) {
    wait_quad(parity);
    // y: both stages of columns 2u, 2u + 1 and both pairs by one warp
#pragma unroll 1
    for (int u = warp; u < (NZH + 1) / 2; u += NW) {
      const int c = 2 * u + ((lane >> 1) & 1);
      const bool has_col = c < NZH;
      float4* const col = O + (has_col ? 2 * c + q : 0);
      if (has_col) {
        cpair v[R1];
#pragma unroll
        for (int j = 0; j < R1; ++j) v[j] = ld(col + ty * BLOCK + j * ROW);
        PairRadix<R1, +1>::run(v);
#pragma unroll
        for (int j = 0; j < R1; ++j) st(col + ty * BLOCK + j * ROW, v[j]);
      }
      __syncwarp();
      if (has_col && np < R1) {
        cpair v[8];
#pragma unroll
        for (int b = 0; b < 8; ++b) v[b] = ld(col + b * BLOCK + np * ROW);
        yz_twiddle<N>(v, tw, np);
        PairRadix<8, +1>::run(v);
#pragma unroll
        for (int j = 0; j < 8; ++j) st(col + j * BLOCK + np * ROW, v[j]);
      }
    }
    __syncthreads();
    // z: rows (2g, 2g + 1) as one complex line with its Hermitian extension
    const int x = 4 * p + 2 * q;
    const bool pair = x < Wx, plane1 = x + 1 < Wx;
#pragma unroll 1
    for (int w = warp; 2 * w < npairs; w += NW) {
      const int g = 2 * w + g2;
      const bool act = g < npairs && pair;
      const int y = 2 * (g < npairs ? g : 0);
      float4* const A = O + (y / R1) * BLOCK + (y % R1) * ROW + q;
      const float4* const Bv = A + ROW;
      {
        cpair z[R1];
#pragma unroll
        for (int j = 0; j < R1; ++j) {
          const int k = t + 8 * j;
          const int m = j < R1 / 2 ? k : N - k;
          const cpair ak = ld(A + 2 * m), bk = ld(Bv + 2 * m);
          if (j < R1 / 2) z[j] = cpair{p_sub(ak.x, bk.y), p_add(ak.y, bk.x)};
          else z[j] = cpair{p_add(ak.x, bk.y), p_sub(bk.x, ak.y)};
          if ((j == 0 || j == R1 / 2) && t == 0) z[j] = cpair{ak.x, bk.x};  // k = 0, N / 2
        }
        __syncwarp();  // the warp has read its rows: their slots become the exchange
        PairRadix<R1, +1>::run(z);
        if (g < npairs) {
#pragma unroll
          for (int j = 0; j < R1; ++j) st(A + 2 * (t * R1 + (j ^ (t & SW))), z[j]);
        }
        __syncwarp();
      }
      const bool on = act && t < R1;
      cpair v[8];
#pragma unroll
      for (int b = 0; b < 8; ++b) v[b] = ld(A + 2 * (b * R1 + ((t & SW) ^ (b & SW))));
      yz_twiddle<N>(v, tw, t & SW);
      PairRadix<8, +1>::run(v);
      yz_keep<N, TOP2>(v, on, t & SW, x, y, y + 1 < Wy, plane1, Wz, inv, lane, &s_bound, best, best2);
    }
    // the next quad's copies (async proxy) follow every read and write of this one
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    __syncthreads();
    if (tid == 0 && p + parts < quads) load_quad(p + parts);
  }
  yz_store<N, NW, TOP2>(a, r, part, O, best, best2);
  if (tid == 0 && s_fail) {
    atomicOr(a.fault, 1);
    s_fail = 0;
    wait_quad(parity ^ 1u);  // a copy still in flight lands before the CTA leaves
  }
}

// CTAs per rotation: about 16 rounds of CTAs over the device, so that the last one costs little,
// each with at least two plane pairs
template <int N>
int yz_parts(int nrot) {
  const long want = 148l * YzShape<N>::CTAS * 16;
  return (int)std::max<long>(1, std::min<long>(N / 4, (want + nrot - 1) / nrot));
}

// Over quads of single rotations (n <= 64) k_yz_quads, else k_yz_pairs: both sides above
template <int N>
cudaError_t launch_t(const WaveArgs& a, cudaStream_t s) {
  constexpr bool SINGLE = b_quad_rots(N) == 1;
  if (a.bpairs == 2 && a.keys2) return cudaErrorInvalidValue;  // plane pairs are the FP32 form's: one key
  void (*kern)(WaveArgs) = k_yz_pairs<N, false, false>;
  size_t sm = YzShape<N>::SMEM;
  int threads = YzShape<N>::T;
  if (a.bpairs == 4) {
    if constexpr (SINGLE) {
      kern = a.keys2 ? k_yz_quads<N, true> : k_yz_quads<N, false>;
      sm = YzQuadShape<N>::SMEM;
      threads = YzQuadShape<N>::T;
    } else {
      kern = a.keys2 ? k_yz_pairs<N, true, true> : k_yz_pairs<N, false, true>;
    }
  }
  const cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm);
  if (e != cudaSuccess) return e;
  kern<<<dim3(yz_parts<N>(a.nrot), a.nrot), threads, sm, s>>>(a);
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
