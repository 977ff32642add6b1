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
// k_yz_pairs, n >= 96 (k_yz_two, n <= 64, takes two pairs at once and is described there): CTA = a rotation
// and a part of its plane pairs, looped. An octet of 8 lanes owns a line (a kz column for y, a row pair for
// z): lane t takes a block in the first stage and the groups np, np + 8, ... in the second; the exchange
// between them goes through the line's own storage in the plane buffer, with __syncwarp only, so that a
// pair of planes has two CTA barriers (y -> z, z -> the next y). Banks, in 16-byte units of which a
// quarter-warp must hit 8 different ones: in the y pass a quarter-warp is 4 neighbouring columns of 2
// blocks or groups, 4 mod 8 units apart; in the z pass it is one octet, a line's positions swizzled within
// its row pair. Plane pairs are copied into the plane buffer by eight bulk copies, so that their loads do
// not go through the LSU; quads of two rotations side by side are loaded by the y pass (the copies would
// bring both rotations).
//
// Measured on a B200, inverse pass, against the single-plane kernels of before (ms per 1e5 rotations): over
// quads with the two smallest keys 64^3 42.9 -> 25.2, 96^3 259 -> 130, 128^3 672 -> 350; over plane pairs 64^3
// 30.2 -> 23.2, 96^3 221 -> 119, 128^3 526 -> 306 (96^3 1.25 -> 1.19 and 128^3 3.21 -> 3.06 ms per 1,000 by the
// bulk copies). What bounds it now is the shared-memory data path (70 % at 64^3) beside the CTA barriers;
// at 128^3, where the plane buffer allows one CTA per SM, the barriers and the load latency.
//
// The smallest key (two smallest: TOP2) is carried over the CTA's planes and reduced once at its
// end; a bound in shared memory, lowered by each warp that sees smaller energies, keeps all but a
// few lanes from building keys.
#include <cuda_runtime.h>
#include <stdint.h>

#include <algorithm>

#include "cdk_internal.h"
#include "copy_turns.cuh"
#include "pair_fft.cuh"
#include "window_keys.cuh"

namespace cdk {
namespace {

// Threads per CTA: octets for all kz columns in one round
template <int N, bool QUADS>
struct YzShape {
  static constexpr int NZH = N / 2 + 1;
  static constexpr int T = (NZH * 8 + 31) / 32 * 32;  // 416, 544
  static constexpr int CTAS = N == 96 ? 2 : 1;
  // units of 16 bytes between rows (plane pairs: a block of N / 8 rows as it lies in B; quads: 4 mod 8) and
  // between blocks
  static constexpr int ROW = QUADS ? (NZH + 3) / 8 * 8 + 4 : NZH;
  static constexpr int BLOCK = ((N / 8) * ROW + 3) / 8 * 8 + 4;
  static constexpr size_t SMEM = sizeof(float2) * (N / 8) * 7 + sizeof(float4) * 8 * BLOCK;
  static_assert(ROW >= NZH && ROW % 8 == (QUADS ? 4 : 1) && BLOCK % 8 == 4 && 2 * ROW >= N, "row and block strides");
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

constexpr long kYzWaitLimit = 1l << 22;

// Bounded wait for a phase of the CTA's copies; fail is set when it gives up
__device__ __forceinline__ void yz_wait(uint32_t bar, uint32_t parity, volatile int* fail) {
  for (long i = 0; i < kYzWaitLimit; ++i) {
    uint32_t done;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(done)
        : "r"(bar), "r"(parity)
        : "memory");
    if (done) return;
    if (i > 32) {
      if (*fail) return;  // another thread gave up
      __nanosleep(40);
    }
  }
  *fail = 1;
}

// One thread: 8 COPIES bulk copies of bytes each into the plane buffer: copy i from src + (i & 7) sb + (i >> 3) sq
// to dst + (i & 7) db + (i >> 3) dq, completing on bar
template <int COPIES>
__device__ __forceinline__ void yz_load(float4* dst, const float4* src, uint32_t bytes, int db, int dq, int sb, int sq,
                                        uint32_t bar) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%1], %0;" ::"r"(bytes * COPIES * 8), "r"(bar) : "memory");
#pragma unroll 1
  for (int i = 0; i < 8 * COPIES; ++i) {
    const int b = i & 7, q = i >> 3;
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                     (uint32_t)__cvta_generic_to_shared(dst + b * db + q * dq)),
                 "l"(src + (size_t)b * sb + (size_t)q * sq), "r"(bytes), "r"(bar)
                 : "memory");
  }
}

// The operations of copy_turns from a kernel's lambdas
template <class Load, class Wait, class Columns, class Failed, class Rows, class Drain>
struct YzTurns {
  Load load;
  Wait wait;
  Columns columns;
  Failed failed;
  Rows rows;
  Drain drain;
};
template <class... F>
__device__ __forceinline__ YzTurns<F...> yz_turns(F... f) {
  return {f...};
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

// A CTA whose copies did not come: reports it and leaves no keys
template <int N, bool TOP2>
__device__ __forceinline__ void yz_give_up(const WaveArgs& a, int r, int part) {
  if (threadIdx.x != 0) return;
  atomicOr(a.fault, 1);
  if constexpr (TOP2) a.keys2[((size_t)r * N + part) * 2] = a.keys2[((size_t)r * N + part) * 2 + 1] = ~0ull;
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
__global__ void __launch_bounds__(YzShape<N, QUADS>::T, YzShape<N, QUADS>::CTAS) k_yz_pairs(const __grid_constant__ WaveArgs a) {
  constexpr int NZH = N / 2 + 1, NCOL = N * NZH, R1 = N / 8, T = YzShape<N, QUADS>::T;
  constexpr int ROW = YzShape<N, QUADS>::ROW, BLOCK = YzShape<N, QUADS>::BLOCK;
  constexpr int NG = (R1 + 7) / 8;  // second-stage groups per lane
  static_assert(T / 8 >= N / 2 && R1 * 7 % 2 == 0, "an octet per row pair; the plane buffer aligned");
  extern __shared__ __align__(16) unsigned char smem_raw[];
  float2* tw = reinterpret_cast<float2*>(smem_raw);
  float4* O = reinterpret_cast<float4*>(tw + R1 * 7);
  // order_key of an energy that at least one (TOP2: two) of the CTA's values so far does not exceed:
  // a value strictly above it cannot enter
  __shared__ unsigned int s_bound;
  __shared__ __align__(8) uint64_t s_full;  // plane pairs: their copies
  __shared__ int s_fail;
  const uint32_t full = (uint32_t)__cvta_generic_to_shared(&s_full);
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
  if (tid == 0) {
    s_bound = order_key(INFINITY);
    s_fail = 0;
    if constexpr (!QUADS) {
      asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(full));
      asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
  }
  auto ld = [](const float4* p) {
    const float4 f = *p;
    return cpair{pk(f.x, f.y), pk(f.z, f.w)};
  };
  auto st = [](float4* p, cpair v) {
    const float2 x = unpk(v.x), y = unpk(v.y);
    *p = make_float4(x.x, x.y, y.x, y.y);
  };
  constexpr int BS = 2 * b_quad_rots(N);  // quads: float4 per column
  const bool has_col = gy < NZH;
  const int c0 = ty * R1 * NZH + (has_col ? gy : 0);  // column of the block's first row
  const float4* src0 = reinterpret_cast<const float4*>(a.B) +
                       (QUADS ? b_quad_index<N>(r, c0) : (size_t)r * (N / 2) * NCOL);
  float4* const col = O + (has_col ? gy : 0);
  const int sw = R1 % 8 == 0 ? t : t >> 1;  // swizzle of a line's positions t R1 + m -> t R1 + (m ^ sw)
  const float inv = 1.0f / (float)((double)N * N * N);
  unsigned long long best = ~0ull, best2 = ~0ull;
  // plane pairs, one thread: the eight blocks into the plane buffer
  auto load = [&](int p) {
    if (!QUADS && tid == 0) yz_load<1>(O, src0 + (size_t)p * NCOL, R1 * NZH * 16, BLOCK, 0, R1 * NZH, 0, full);
  };
  auto wait = [&](uint32_t parity) {
    if constexpr (!QUADS) yz_wait(full, parity, &s_fail);
  };
  auto failed = [&] { return !QUADS && *(volatile int*)&s_fail != 0; };
  auto drain = [&](uint32_t parity) {
    int gave_up = 0;
    if (!QUADS && tid == 0) yz_wait(full, parity, &gave_up);
  };
  auto columns = [&](int p) {
    // y of column gy: first stage (radix R1, no twiddles) over block ty's positions
    if (has_col) {
      cpair v[R1];
      if constexpr (QUADS) {
        const float4* src = src0 + (size_t)(p >> 1) * (NCOL * BS) + (p & 1);
#pragma unroll
        for (int j = 0; j < R1; ++j) v[j] = ld(src + j * NZH * BS);
      } else {
#pragma unroll
        for (int j = 0; j < R1; ++j) v[j] = ld(col + ty * BLOCK + j * ROW);
      }
      PairRadix<R1, +1>::run(v);
#pragma unroll
      for (int j = 0; j < R1; ++j) st(col + ty * BLOCK + j * ROW, v[j]);
    }
    __syncwarp();
    // second stage (radix 8): the groups' 8 positions become the natural rows np + R1 j in place
#pragma unroll
    for (int q = 0; q < NG; ++q) {
      // plane pairs: a quarter-warp's two groups 4 rows apart (4 units mod 8)
      const int np = (QUADS ? ty : (ty & 1) * 4 + (ty >> 1)) + 8 * q;
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
  };
  auto rows = [&](int p) {
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
    // the next pair's copies (async proxy) follow every read and write of this one
    if constexpr (!QUADS) asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    __syncthreads();
  };
  __syncthreads();
  auto turns = yz_turns(load, wait, columns, failed, rows, drain);
  if (copy_turns(part, parts, pairs, turns)) yz_store<N, T / 32, TOP2>(a, r, part, O, best, best2);
  else yz_give_up<N, TOP2>(a, r, part);
}

// Two plane pairs at once (n <= 64): a CTA brings them into its plane buffer with bulk copies, so no load
// goes through the LSU -- there a 16-byte load, whose lanes took half of 32 sectors in 8 or more lines, cost
// 24 L1 cycles, 42 % of the L1 time at 64^3 -- and transforms both in place between the same two barriers.
// Three CTAs per SM at 64^3 hide each other's copies. Eight copies (plane pairs: sixteen), a block of N / 8
// rows each, from one thread: one per row, issued lane by lane, kept a warp busy for thousands of cycles
// (64^3 28.2 -> 25.2 ms per 1e5 rotations). A quarter-warp is 2 columns x 2 pairs x 2 blocks in y and 4
// positions x 2 pairs in z, 8 different banks with the strides below. Against one pair at a time, ms per 1e5
// rotations: quads, two smallest keys, 64^3 33.3 -> 25.2, 32^3 5.6 -> 3.9; plane pairs 64^3 27.5 -> 23.2. Threads
// per CTA (192, 256, 288, 320 at 64^3) make no difference: it is bound by the shared-memory data path.
template <int N, bool QUADS>
struct YzTwoShape {
  static constexpr int NZH = N / 2 + 1, R1 = N / 8;
  static constexpr int T = N == 32 ? 160 : 288;
  static constexpr int CTAS = N == 32 ? 6 : 3;
  // units of 16 bytes between columns, rows (2 or 1 mod 8: a block of N / 8 rows as it lies in B), a block's
  // pairs (plane pairs: 4 mod 8) and blocks (4 mod 8, plane pairs 2)
  static constexpr int COL = QUADS ? 2 : 1;
  static constexpr int ROW = COL * NZH;
  static constexpr int PAIR = QUADS ? 1 : (R1 * ROW + 3) / 8 * 8 + 4;
  static constexpr int BLOCK = QUADS ? R1 * ROW + 4 : (PAIR + R1 * ROW + 5) / 8 * 8 + 2;
  static constexpr size_t SMEM = sizeof(float2) * (N / 8) * 7 + sizeof(float4) * 8 * BLOCK;
  static_assert(QUADS ? ROW % 8 == 2 && BLOCK % 8 == 4
                      : ROW % 8 == 1 && PAIR % 8 == 4 && BLOCK % 8 == 2 && PAIR >= R1 * ROW && BLOCK >= PAIR + R1 * ROW,
                "strides");
  static_assert(2 * ROW >= COL * N, "a row pair holds its lines");
};

template <int N, bool TOP2, bool QUADS>
__global__ void __launch_bounds__(YzTwoShape<N, QUADS>::T, YzTwoShape<N, QUADS>::CTAS)
    k_yz_two(const __grid_constant__ WaveArgs a) {
  using S = YzTwoShape<N, QUADS>;
  constexpr int NZH = S::NZH, R1 = N / 8, T = S::T, NW = T / 32, ROW = S::ROW, BLOCK = S::BLOCK;
  static_assert(R1 <= 8 && (!QUADS || b_quad_rots(N) == 1), "one second-stage group per lane, rotations apart");
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
  // one thread: the eight blocks of both pairs into the plane buffer
  auto load = [&](int p) {
    constexpr int COPIES = QUADS ? 1 : 2;  // per block
    const float4* src = reinterpret_cast<const float4*>(a.B) + ((size_t)r * (N / 4) + p) * (N * NZH * 2);
    if (tid == 0) yz_load<COPIES>(O, src, R1 * NZH * 32 / COPIES, BLOCK, S::PAIR, R1 * ROW, N * NZH, full);
  };
  auto wait = [&](uint32_t parity) { yz_wait(full, parity, &s_fail); };
  auto failed = [&] { return *(volatile int*)&s_fail != 0; };
  auto drain = [&](uint32_t parity) {
    int gave_up = 0;
    if (tid == 0) yz_wait(full, parity, &gave_up);
  };
  const int q = lane & 1;                          // the lane's pair of the quad
  const int ty = lane >> 2;                        // y: block; columns 2u, 2u + 1 of unit u
  // and group: the quarter-warp's two groups 2 rows, 4 units mod 8, apart
  const int np = (ty & 4) | ((ty & 1) << 1) | ((ty >> 1) & 1);
  const int t = (lane >> 1) & 7, g2 = lane >> 4;   // z: place in the line; row pairs 2w, 2w + 1 of unit w
  constexpr int SW = R1 - 1;  // swizzle of a line's positions b R1 + m -> b R1 + (m ^ (b & SW))
  const float inv = 1.0f / (float)((double)N * N * N);
  unsigned long long best = ~0ull, best2 = ~0ull;
  auto columns = [&](int p) {
    // y: both stages of columns 2u, 2u + 1 and both pairs by one warp
#pragma unroll 1
    for (int u = warp; u < (NZH + 1) / 2; u += NW) {
      const int c = 2 * u + ((lane >> 1) & 1);
      const bool has_col = c < NZH;
      float4* const col = O + q * S::PAIR + (has_col ? c * S::COL : 0);
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
  };
  auto rows = [&](int p) {
    // z: rows (2g, 2g + 1) as one complex line with its Hermitian extension
    const int x = 4 * p + 2 * q;
    const bool pair = x < Wx, plane1 = x + 1 < Wx;
#pragma unroll 1
    for (int w = warp; 2 * w < npairs; w += NW) {
      const int g = 2 * w + g2;
      const bool act = g < npairs && pair;
      const int y = 2 * (g < npairs ? g : 0);
      float4* const A = O + (y / R1) * BLOCK + (y % R1) * ROW + q * S::PAIR;
      const float4* const Bv = A + ROW;
      {
        cpair z[R1];
#pragma unroll
        for (int j = 0; j < R1; ++j) {
          const int k = t + 8 * j;
          const int m = j < R1 / 2 ? k : N - k;
          const cpair ak = ld(A + m * S::COL), bk = ld(Bv + m * S::COL);
          if (j < R1 / 2) z[j] = cpair{p_sub(ak.x, bk.y), p_add(ak.y, bk.x)};
          else z[j] = cpair{p_add(ak.x, bk.y), p_sub(bk.x, ak.y)};
          if ((j == 0 || j == R1 / 2) && t == 0) z[j] = cpair{ak.x, bk.x};  // k = 0, N / 2
        }
        __syncwarp();  // the warp has read its rows: their slots become the exchange
        PairRadix<R1, +1>::run(z);
        if (g < npairs) {
#pragma unroll
          for (int j = 0; j < R1; ++j) st(A + S::COL * (t * R1 + (j ^ (t & SW))), z[j]);
        }
        __syncwarp();
      }
      const bool on = act && t < R1;
      cpair v[8];
#pragma unroll
      for (int b = 0; b < 8; ++b) v[b] = ld(A + S::COL * (b * R1 + ((t & SW) ^ (b & SW))));
      yz_twiddle<N>(v, tw, t & SW);
      PairRadix<8, +1>::run(v);
      yz_keep<N, TOP2>(v, on, t & SW, x, y, y + 1 < Wy, plane1, Wz, inv, lane, &s_bound, best, best2);
    }
    // the next quad's copies (async proxy) follow every read and write of this one
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    __syncthreads();
  };
  __syncthreads();
  auto turns = yz_turns(load, wait, columns, failed, rows, drain);
  if (copy_turns(part, parts, quads, turns)) yz_store<N, NW, TOP2>(a, r, part, O, best, best2);
  else yz_give_up<N, TOP2>(a, r, part);
}

// CTAs per rotation: about 16 rounds of CTAs over the device, so that the last one costs little,
// each with at least two plane pairs
template <int N>
int yz_parts(int nrot) {
  const long want = 148l * (N == 32 ? 6 : N == 64 ? 3 : N == 96 ? 2 : 1) * 16;
  return (int)std::max<long>(1, std::min<long>(N / 4, (want + nrot - 1) / nrot));
}

// n <= 64: k_yz_two, else k_yz_pairs (both sides above; the plane buffer of two pairs would leave one CTA
// per SM at n = 96 and does not fit at 128). Two smallest keys only over quads: plane pairs are the FP32
// form's.
template <int N>
cudaError_t launch_t(const WaveArgs& a, cudaStream_t s) {
  const bool quads = a.bpairs == 4;
  if (!quads && a.keys2) return cudaErrorInvalidValue;
  void (*kern)(WaveArgs);
  size_t sm;
  int threads;
  if constexpr (N <= 64) {
    kern = a.keys2 ? k_yz_two<N, true, true> : quads ? k_yz_two<N, false, true> : k_yz_two<N, false, false>;
    sm = quads ? YzTwoShape<N, true>::SMEM : YzTwoShape<N, false>::SMEM;
    threads = YzTwoShape<N, true>::T;
  } else {
    kern = a.keys2 ? k_yz_pairs<N, true, true> : quads ? k_yz_pairs<N, false, true> : k_yz_pairs<N, false, false>;
    sm = quads ? YzShape<N, true>::SMEM : YzShape<N, false>::SMEM;
    threads = YzShape<N, true>::T;
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
