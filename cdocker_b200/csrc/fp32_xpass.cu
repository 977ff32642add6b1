// fp32_xpass.cu -- the FP32 form's x pass: per spectral column the forward DFT along x of every
// channel's ligand planes, the conjugate product with the resident receptor spectrum summed over
// the channels, and the inverse DFT, of which only the translation window's rows are written
// (src/kernel.cu ConjMult + SumGrids and the x dimension of the transforms around them).
//
// The transform of length N = 8 R1 runs as a radix-8 and a radix-R1 stage. Here a thread owns,
// for one column of one rotation, the first-stage outputs q = QQ and QQ + 4 (QQ = its warp of
// four): it evaluates them straight from the ligand's planes x = np + R1 j, of which only
// j < JN = ceil(box / R1) can be non-zero (2 or 3 of the 8), and the second stage, the product
// and the channel sum of those outputs then stay in its registers: the forward transforms need no
// exchange at all. One exchange through shared memory per rotation feeds the last inverse stage.
// The outputs q and q + 4 differ in one sign before their twiddles, so the two live in one
// register pair each and most of the arithmetic is packed (pair_fft.cuh).
//
// What bounds it: latency at one CTA of 16 warps per SM (registers, receptor tile and rings). At 64^3, box
// of 22 planes, issue is 63 % active, the shared-memory path 67 %, the FMA pipe 50 %; a warp waits, per issue,
// 1.1 for fixed latencies, 0.8 for shared loads, 0.7 each for the FP32 pipe and the channel's barrier (per
// thread and channel about 430 instructions, 226 floating point, 42 shared loads). Measured on a B200, K = 9,
// against k_xpass_block (block_xpass.cu), which exchanges between the stages for every channel and spends its
// issue slots on shared-memory traffic and block barriers: 32^3, 500 rotations 0.373 -> 0.145 ms; 64^3, 5,000
// rotations 15.1 -> 7.2 ms; 96^3, 999 rotations 10.7 -> 4.2 ms; 128^3, 1,000 rotations 26.1 -> 11.1 ms; results
// bit-identical. That kernel takes the waves where it is the faster (xpass_block_stages below).
//
// CTA = 8 columns x a chunk of rotations; its 8-column tile of the receptor spectra stays in
// shared memory. 8 columns and not 16 or 32: the tile fits beside the rings at every n and K <=
// 16, a spectra load is shared by the warp's four rotations, and 64-byte row pieces still fill
// whole sectors. G groups of 128 threads (7 at n = 32, 4 at 64, 3 above: the registers of the second
// stage; at 32^3 seven measured 0.145 ms against 0.162 with four, 500 rotations, and 0.99 against 1.12,
// 4,000; at 64^3 five, at 96 registers, gained nothing) each take every G-th set of 4 rotations; a warp's lanes are 8 columns x 4
// rotations. A set's channels are streamed through a ring of nst stages by 16-byte cp.async (one
// stage: the planes 0 .. R1 JN - 1 of one channel, the untouched ones zero-filled by the copy),
// one 128-thread barrier per channel.
//
// Order of the sums: a rotation's active channels alternate between two partial sums (even and
// odd rank), added at the end; ascending channels within each. The even sum waits in the group's
// exchange buffer while the odd one accumulates.
#include <cuda_runtime.h>
#include <stdint.h>

#include <algorithm>
#include <cmath>

#include "cdk_internal.h"
#include "pair_fft.cuh"

namespace cdk {
namespace {

constexpr int XP_COLS = 8;                    // columns per CTA
constexpr int XP_SET = 32 / XP_COLS;          // rotations per set (a warp's lanes: 8 x 4)
constexpr int XP_MAX_CHUNK = 128;             // rotations per CTA
constexpr int XP_MIN_CHUNK = 32;
constexpr size_t kXpSmemCap = 227 * 1024 - 512;

template <int N>
struct XpShape {
  static constexpr int R1 = N / 8;
  static constexpr int GMAX = N == 32 ? 7 : N == 64 ? 4 : 3;  // groups of 128 threads
};

// twiddles w_N^(np q) of the output pairs (q, q + 4), q = 0..3, in the kernel's parameters: real,
// imaginary and negated imaginary parts as register pairs
template <int N>
struct XpTwiddles {
  pair_t x[N / 8][4], y[N / 8][4], ny[N / 8][4];
};

// what the kernel needs of a rotation's record
struct XpRec {
  uint8_t lo[KMAX], cnt[KMAX];  // per channel: first touched plane and their number (0: none)
  uint16_t act, even;           // active channels; those of even rank among them
  int W0;                       // x window; 0: not a valid rotation
};
// A set's channels in order: ne of the even partial sum, then no of the odd one; a step is the
// channel, plus kXpWide when its planes need the launch's JM inputs per first-stage output.
// uniform: all its valid rotations have the same channels in the same sums.
constexpr int kXpWide = 0x80;
struct XpSet {
  uint8_t ne, no, uniform, pad;
  uint8_t step[2 * KMAX];
};

// inputs per first-stage output: the launch's JM, or JL where a channel's planes allow it
__host__ __device__ constexpr int xp_low(int jm) { return jm == 8 ? 4 : jm - 1; }

// First forward stage: outputs QQ (low half) and QQ + 4 (high half) of the radix-8 DFT over
// x[j], j < JN (the others are zero), times the twiddles; Radix<8, -1> and c_mul of fft.cuh with the
// terms that are zero left out.
template <int N, int JN, int QQ>
__device__ __forceinline__ void xp_stage1(const float2* st, const XpTwiddles<N>& tw, cpair* v) {
  constexpr int R1 = N / 8;
  const float r2 = 0.70710678118654752440f;
#pragma unroll
  for (int np = 0; np < R1; ++np) {
    float2 x[JN];
#pragma unroll
    for (int j = 0; j < JN; ++j) x[j] = st[(np + R1 * j) * 32];
    float2 lo, hi;
    if constexpr (JN == 1) {
      lo = hi = x[0];
    } else {
      // u_j = x_j + x_(j+4) (even outputs) or x_j - x_(j+4) (odd outputs)
      float2 u[4];
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        if (j + 4 < JN)
          u[j] = QQ % 2 == 0 ? make_float2(__fadd_rn(x[j].x, x[j + 4 < JN ? j + 4 : 0].x), __fadd_rn(x[j].y, x[j + 4 < JN ? j + 4 : 0].y))
                             : make_float2(__fsub_rn(x[j].x, x[j + 4 < JN ? j + 4 : 0].x), __fsub_rn(x[j].y, x[j + 4 < JN ? j + 4 : 0].y));
        else
          u[j] = j < JN ? x[j < JN ? j : 0] : make_float2(0.f, 0.f);
      }
      float2 s = u[0], t;
      if constexpr (QQ == 0) {
        if (JN > 2) s = make_float2(__fadd_rn(s.x, u[2].x), __fadd_rn(s.y, u[2].y));
        t = JN > 3 ? make_float2(__fadd_rn(u[1].x, u[3].x), __fadd_rn(u[1].y, u[3].y)) : u[1];
      } else if constexpr (QQ == 2) {
        if (JN > 2) s = make_float2(__fsub_rn(s.x, u[2].x), __fsub_rn(s.y, u[2].y));
        const float2 e = JN > 3 ? make_float2(__fsub_rn(u[1].x, u[3].x), __fsub_rn(u[1].y, u[3].y)) : u[1];
        t = make_float2(e.y, -e.x);
      } else {
        const float2 t1 = make_float2(__fadd_rn(u[1].x, u[1].y), __fsub_rn(u[1].y, u[1].x));
        float2 m;
        if (JN > 3) {
          const float2 m3 = make_float2(__fmul_rn(r2, __fsub_rn(u[3].y, u[3].x)), __fmul_rn(-r2, __fadd_rn(u[3].y, u[3].x)));
          m = QQ == 1 ? make_float2(__fmaf_rn(r2, t1.x, m3.x), __fmaf_rn(r2, t1.y, m3.y))
                      : make_float2(__fmaf_rn(r2, t1.x, -m3.x), __fmaf_rn(r2, t1.y, -m3.y));
        } else {
          m = make_float2(__fmul_rn(r2, t1.x), __fmul_rn(r2, t1.y));
        }
        if constexpr (QQ == 1) {
          if (JN > 2) s = make_float2(__fadd_rn(s.x, u[2].y), __fsub_rn(s.y, u[2].x));
          t = m;
        } else {
          if (JN > 2) s = make_float2(__fsub_rn(s.x, u[2].y), __fadd_rn(s.y, u[2].x));
          t = make_float2(m.y, -m.x);
        }
      }
      lo = make_float2(__fadd_rn(s.x, t.x), __fadd_rn(s.y, t.y));
      hi = make_float2(__fsub_rn(s.x, t.x), __fsub_rn(s.y, t.y));
    }
    if (np == 0) {
      v[np] = {pk(lo.x, hi.x), pk(lo.y, hi.y)};
    } else if constexpr (QQ == 0) {
      // output 0 has no twiddle
      const float2 wx = unpk(tw.x[np][0]), wy = unpk(tw.y[np][0]);
      const float hx = __fmaf_rn(hi.x, wx.y, -__fmul_rn(hi.y, wy.y)), hy = __fmaf_rn(hi.y, wx.y, __fmul_rn(hi.x, wy.y));
      v[np] = {pk(lo.x, hx), pk(lo.y, hy)};
    } else {
      const pair_t ax = pk(lo.x, hi.x), ay = pk(lo.y, hi.y);
      v[np] = {p_fma(ax, tw.x[np][QQ], p_mul(ay, tw.ny[np][QQ])), p_fma(ay, tw.x[np][QQ], p_mul(ax, tw.y[np][QQ]))};
    }
  }
}

// Last inverse stage: the radix-8 DFT (Radix<8, +1>) of the twiddled q-outputs e[qq] = (q = qq,
// q = qq + 4)
template <int N>
__device__ __forceinline__ void xp_last(const float4* e, const XpTwiddles<N>& tw, int np, float2* o) {
  const float r2 = 0.70710678118654752440f;
  float2 u[4], w[4];
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    const pair_t ax = pk(e[q].x, e[q].y), ay = pk(e[q].z, e[q].w);
    // c_mulc: (x wx + y wy, y wx - x wy)
    const float2 tx = unpk(p_fma(ax, tw.x[np][q], p_mul(ay, tw.y[np][q])));
    const float2 ty = unpk(p_fma(ay, tw.x[np][q], p_mul(ax, tw.ny[np][q])));
    const float2 a = q == 0 ? make_float2(e[0].x, e[0].z) : make_float2(tx.x, ty.x);
    u[q] = make_float2(__fadd_rn(a.x, tx.y), __fadd_rn(a.y, ty.y));
    w[q] = make_float2(__fsub_rn(a.x, tx.y), __fsub_rn(a.y, ty.y));
  }
  auto add = [](float2 a, float2 b) { return make_float2(__fadd_rn(a.x, b.x), __fadd_rn(a.y, b.y)); };
  auto sub = [](float2 a, float2 b) { return make_float2(__fsub_rn(a.x, b.x), __fsub_rn(a.y, b.y)); };
  {
    const float2 s02 = add(u[0], u[2]), d02 = sub(u[0], u[2]), s13 = add(u[1], u[3]), e13 = sub(u[1], u[3]);
    o[0] = add(s02, s13);
    o[4] = sub(s02, s13);
    o[2] = make_float2(__fsub_rn(d02.x, e13.y), __fadd_rn(d02.y, e13.x));
    o[6] = make_float2(__fadd_rn(d02.x, e13.y), __fsub_rn(d02.y, e13.x));
  }
  const float2 t1 = make_float2(__fsub_rn(w[1].x, w[1].y), __fadd_rn(w[1].y, w[1].x));
  const float2 m3 = make_float2(__fmul_rn(-r2, __fadd_rn(w[3].x, w[3].y)), __fmul_rn(r2, __fsub_rn(w[3].x, w[3].y)));
  const float2 s13 = make_float2(__fmaf_rn(r2, t1.x, m3.x), __fmaf_rn(r2, t1.y, m3.y));
  const float2 e13 = make_float2(__fmaf_rn(r2, t1.x, -m3.x), __fmaf_rn(r2, t1.y, -m3.y));
  const float2 s02 = make_float2(__fsub_rn(w[0].x, w[2].y), __fadd_rn(w[0].y, w[2].x));
  const float2 d02 = make_float2(__fadd_rn(w[0].x, w[2].y), __fsub_rn(w[0].y, w[2].x));
  o[1] = add(s02, s13);
  o[5] = sub(s02, s13);
  o[3] = make_float2(__fsub_rn(d02.x, e13.y), __fadd_rn(d02.y, e13.x));
  o[7] = make_float2(__fadd_rn(d02.x, e13.y), __fsub_rn(d02.y, e13.x));
}

struct XpShared {
  const float4* P;     // [K][R1][4][8] receptor spectra: (re q, re q+4, im q, im q+4)
  const XpRec* recs;   // the chunk's rotations
  const XpSet* sets;
  float4* exch;        // the group's exchange buffer [R1][4][32]
  float2* ring;        // the group's ring [nst][planes][32]
};

// stage 1 of output pair qq (uniform over the warp): only this part of the loop is specialised by the
// pair, so that the loop's code stays small (the whole loop four times over missed the instruction
// cache: half of the issue cycles)
template <int N, int JN>
__device__ __forceinline__ void xp_stage1_of(int qq, const float2* st, const XpTwiddles<N>& tw, cpair* v) {
  if (qq == 0) xp_stage1<N, JN, 0>(st, tw, v);
  else if (qq == 1) xp_stage1<N, JN, 1>(st, tw, v);
  else if (qq == 2) xp_stage1<N, JN, 2>(st, tw, v);
  else xp_stage1<N, JN, 3>(st, tw, v);
}

template <int N, int JM>
__device__ __forceinline__ void xp_body(const WaveArgs& a, const XpTwiddles<N>& tw, const XpShared& sh, int grp, int G,
                                        int nst, int r_begin, int nsets, int c0, int QQ) {
  constexpr int R1 = N / 8, NCOL = N * (N / 2 + 1), JL = xp_low(JM);
  constexpr int PLANES = R1 * JM;
  const int t = threadIdx.x & 127, lane = t & 31;
  const int col = lane % XP_COLS, rot = lane / XP_COLS;
  const int bar = grp + 1;
  auto group_sync = [&] {
    __syncwarp();
    asm volatile("bar.sync %0, 128;" ::"r"(bar) : "memory");
  };
  // the group's next set with active channels, from s on (nsets: none)
  auto next_set = [&](int s) {
    while (s < nsets && sh.sets[s].ne == 0) s += G;
    return min(s, nsets);
  };
  // copy role: 16 bytes (2 columns) of rotation t / 4 % 4, planes t / 16, t / 16 + 8, ...
  const int f_rot = (t >> 2) & 3, f_p0 = t >> 4;
  const uint32_t f_dst = (uint32_t)__cvta_generic_to_shared(sh.ring) + (uint32_t)(f_p0 * 256 + (t & 15) * 16);
  const float2* f_base = a.A + ((size_t)r_begin * a.K * a.Lb + f_p0) * NCOL + c0 + 2 * (t & 3);
  const uint32_t chan = (uint32_t)a.Lb * NCOL;  // float2 per channel of a rotation
  int f_set = next_set(grp), f_i = 0;
  auto fetch = [&](int slot) {
    if (f_set < nsets) {
      const XpSet& S = sh.sets[f_set];
      const int b = S.step[f_i], k = b & (KMAX - 1);
      const XpRec& rc = sh.recs[f_set * XP_SET + f_rot];
      const int d = f_p0 - rc.lo[k];
      const unsigned int cnt = rc.cnt[k];
      const float2* src = f_base + (size_t)((f_set * XP_SET + f_rot) * a.K + k) * chan;
      const uint32_t dst = f_dst + (uint32_t)slot * (PLANES * 256);
#pragma unroll
      for (int i = 0; i < (PLANES + 7) / 8; ++i) {
        if (8 * i >= R1 * JL && !(b & kXpWide)) break;
        if (PLANES % 8 && 8 * i + 8 > PLANES && f_p0 + 8 * i >= PLANES) break;
        // zero-fills an untouched plane (no byte of its source is read)
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst + 8 * i * 256),
                     "l"(src + (size_t)8 * i * NCOL), "r"((unsigned int)(d + 8 * i) < cnt ? 16 : 0)
                     : "memory");
      }
      if (++f_i == S.ne + S.no) {
        f_i = 0;
        f_set = next_set(f_set + G);
      }
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  for (int i = 0; i + 1 < nst; ++i) fetch(i);
  int slot = 0;
  cpair acc[R1];
  // one channel into acc
  auto step = [&](const XpSet& S, int b, bool lane_on) {
    // this stage's copies have landed, for every thread of the group after the barrier, which
    // also frees the slot of the stage before for the next copies
    if (nst == 3) asm volatile("cp.async.wait_group 1;" ::: "memory");
    else asm volatile("cp.async.wait_group 0;" ::: "memory");
    group_sync();
    fetch(slot == 0 ? nst - 1 : slot - 1);
    const float2* st = sh.ring + (uint32_t)slot * (PLANES * 32) + lane;
    if (++slot == nst) slot = 0;
    cpair v[R1];
    if (b & kXpWide) xp_stage1_of<N, JM>(QQ, st, tw, v);
    else xp_stage1_of<N, JL>(QQ, st, tw, v);
    PairRadix<R1, -1>::run(v);
    // conj(L) P into the partial sum; in a set of different ligands the lanes whose rotation has
    // this channel in the other sum or not at all sit out
    const float4* P = sh.P + ((b & (KMAX - 1)) * R1 * 4 + QQ) * XP_COLS + col;
    if (S.uniform || lane_on) {
#pragma unroll
      for (int j = 0; j < R1; ++j) {
        const float4 p = P[j * 4 * XP_COLS];
        const float2 x = unpk(v[j].x), y = unpk(v[j].y);
        acc[j].x = p_add(acc[j].x, p_fma(v[j].x, pk(p.x, p.y), p_mul(v[j].y, pk(p.z, p.w))));
        acc[j].y = p_add(acc[j].y, pk(__fmaf_rn(x.x, p.z, -__fmul_rn(y.x, p.x)), __fmaf_rn(x.y, p.w, -__fmul_rn(y.y, p.y))));
      }
    }
  };
  float4* ex = sh.exch + QQ * 32 + lane;  // this thread's slots [j * 128]
  for (int s = next_set(grp); s < nsets; s = next_set(s + G)) {
    const XpSet& S = sh.sets[s];
    const XpRec& rc = sh.recs[s * XP_SET + rot];
    const int ne = S.ne, ns = ne + S.no;
#pragma unroll
    for (int j = 0; j < R1; ++j) acc[j] = {0ull, 0ull};
#pragma unroll 1
    for (int i = 0; i < ns; ++i) {
      if (i == ne) {
        // the even partial sum to this thread's own slots of the exchange buffer (its readers of
        // the previous set are past a channel barrier of this one)
#pragma unroll
        for (int j = 0; j < R1; ++j) {
          const float2 x = unpk(acc[j].x), y = unpk(acc[j].y);
          ex[j * 128] = make_float4(x.x, x.y, y.x, y.y);
          acc[j] = {0ull, 0ull};
        }
      }
      const int b = S.step[i];
      step(S, b, (((i < ne ? rc.even : rc.act & ~rc.even) >> (b & (KMAX - 1))) & 1) != 0);
    }
    if (ns > ne) {
#pragma unroll
      for (int j = 0; j < R1; ++j) {
        const float4 e = ex[j * 128];
        acc[j] = {p_add(pk(e.x, e.y), acc[j].x), p_add(pk(e.z, e.w), acc[j].y)};
      }
    }
    PairRadix<R1, +1>::run(acc);
#pragma unroll
    for (int j = 0; j < R1; ++j) {
      const float2 x = unpk(acc[j].x), y = unpk(acc[j].y);
      ex[j * 128] = make_float4(x.x, x.y, y.x, y.y);
    }
    group_sync();
    const int W0 = rc.W0;
    float2* dst = a.B + (size_t)(r_begin + s * XP_SET + rot) * N * NCOL + c0 + col;
    // planes np and np + 1 (np even) of each j together: one 16-byte store in the paired layout
#pragma unroll 1
    for (int np = 2 * QQ; np < R1; np += 8) {
      float2 o[2][8];
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        float4 e[4];
#pragma unroll
        for (int q = 0; q < 4; ++q) e[q] = sh.exch[((np + h) * 4 + q) * 32 + lane];
        xp_last<N>(e, tw, np + h, o[h]);
      }
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        const int x = np + R1 * j;
        if (a.bpairs) {
          if (x < W0)
            *reinterpret_cast<float4*>(dst + (size_t)x * NCOL + c0 + col) =
                make_float4(o[0][j].x, o[1][j].x, o[0][j].y, o[1][j].y);
        } else {
          if (x < W0) dst[(size_t)x * NCOL] = o[0][j];
          if (x + 1 < W0) dst[(size_t)(x + 1) * NCOL] = o[1][j];
        }
      }
    }
  }
  asm volatile("cp.async.wait_all;" ::: "memory");
}

// shared memory of a CTA: the receptor tile, the chunk's records and sets, and per group the
// exchange buffer and the ring
struct XpLayout {
  uint32_t recs, sets, groups, exch, group, total;
};
__host__ __device__ inline XpLayout xp_layout(int n, int K, int G, int nst, int planes, int chunk) {
  XpLayout L;
  L.recs = (uint32_t)K * (n / 8) * 4 * XP_COLS * 16;
  L.sets = L.recs + (uint32_t)chunk * sizeof(XpRec);
  L.groups = (L.sets + (uint32_t)(chunk / XP_SET) * sizeof(XpSet) + 127u) & ~127u;
  L.exch = (uint32_t)(n / 8) * 4 * 32 * 16;
  L.group = L.exch + (uint32_t)nst * planes * 256;
  L.total = L.groups + (uint32_t)G * L.group;
  return L;
}

template <int N, int JM>
__global__ void __launch_bounds__(128 * XpShape<N>::GMAX, 1)
    k_xpass_pairs(const __grid_constant__ WaveArgs a, const __grid_constant__ XpTwiddles<N> tw, int chunk, int nst) {
  constexpr int R1 = N / 8, NCOL = N * (N / 2 + 1);
  extern __shared__ __align__(128) unsigned char smem_raw[];
  const int G = blockDim.x >> 7;
  const int tid = threadIdx.x;
  const XpLayout L = xp_layout(N, a.K, G, nst, R1 * JM, chunk);
  float4* P = reinterpret_cast<float4*>(smem_raw);
  XpRec* recs = reinterpret_cast<XpRec*>(smem_raw + L.recs);
  XpSet* sets = reinterpret_cast<XpSet*>(smem_raw + L.sets);
  const int c0 = blockIdx.x * XP_COLS;
  const int r_begin = blockIdx.y * chunk;
  const int nrot = min(chunk, a.nrot - r_begin);
  const int nsets = (nrot + XP_SET - 1) / XP_SET;
  for (int i = tid; i < nsets * XP_SET; i += blockDim.x) {
    XpRec& r = recs[i];
    const RotRec* rec = a.rec + r_begin + i;
    const bool valid = i < nrot && rec->valid;
    unsigned int act = 0, even = 0;
    int rank = 0;
    for (int k = 0; k < KMAX; ++k) {
      const bool on = valid && k < a.K && rec->xlo[k] <= rec->xhi[k];
      r.lo[k] = on ? (uint8_t)rec->xlo[k] : 0;
      r.cnt[k] = on ? (uint8_t)(rec->xhi[k] - rec->xlo[k] + 1) : 0;
      if (on) {
        act |= 1u << k;
        if (!(rank++ & 1)) even |= 1u << k;
      }
    }
    r.act = (uint16_t)act;
    r.even = (uint16_t)even;
    r.W0 = valid ? rec->W[0] : 0;
  }
  // receptor tile: position q R1 + j of column c0 + c
  float* Pf = reinterpret_cast<float*>(P);
  for (int i = tid; i < a.K * N * XP_COLS; i += blockDim.x) {
    const int c = i % XP_COLS, pos = (i / XP_COLS) % N, k = i / (XP_COLS * N);
    const int q = pos / R1, j = pos % R1;
    const float2 p = a.phat[((size_t)pos * a.K + k) * NCOL + c0 + c];
    float* d = Pf + (((size_t)(k * R1 + j) * 4 + (q & 3)) * XP_COLS + c) * 4 + (q >> 2);
    d[0] = p.x;
    d[2] = p.y;
  }
  __syncthreads();
  for (int i = tid; i < nsets; i += blockDim.x) {
    XpSet& S = sets[i];
    const XpRec* rc = recs + i * XP_SET;
    unsigned int em = 0, om = 0, first = 0;
    bool uniform = true;
    for (int r = 0; r < XP_SET; ++r) {
      em |= rc[r].even;
      om |= rc[r].act & ~rc[r].even;
      if (rc[r].act == 0) continue;  // not valid (or no atoms): its lanes are never stored
      if (first == 0) first = rc[r].act;
      uniform = uniform && rc[r].act == first;
    }
    int n = 0;
    for (int half = 0; half < 2; ++half) {
      for (int k = 0; k < KMAX; ++k) {
        if (!(((half ? om : em) >> k) & 1)) continue;
        int top = 0;
        for (int r = 0; r < XP_SET; ++r) top = max(top, (int)rc[r].lo[k] + (int)rc[r].cnt[k]);
        S.step[n++] = (uint8_t)(k | (top > R1 * xp_low(JM) ? kXpWide : 0));
      }
      if (half) S.no = (uint8_t)(n - S.ne);
      else S.ne = (uint8_t)n;
    }
    S.uniform = uniform;
  }
  __syncthreads();
  const int grp = tid >> 7;
  XpShared sh;
  sh.P = P;
  sh.recs = recs;
  sh.sets = sets;
  sh.exch = reinterpret_cast<float4*>(smem_raw + L.groups + (uint32_t)grp * L.group);
  sh.ring = reinterpret_cast<float2*>(reinterpret_cast<unsigned char*>(sh.exch) + L.exch);
  xp_body<N, JM>(a, tw, sh, grp, G, nst, r_begin, nsets, c0, __shfl_sync(0xffffffffu, (tid >> 5) & 3, 0));
}

template <int N>
const XpTwiddles<N>& xp_twiddles() {
  static const XpTwiddles<N> t = [] {
    XpTwiddles<N> w;
    auto bits = [](float lo, float hi) {
      union {
        float f[2];
        pair_t p;
      } u;
      u.f[0] = lo;
      u.f[1] = hi;
      return u.p;
    };
    for (int np = 0; np < N / 8; ++np)
      for (int q = 0; q < 4; ++q) {
        // the context's twiddle table: exp(-2 pi i j / N) rounded to float
        auto c = [](int j) { return (float)std::cos(-2.0 * M_PI * j / N); };
        auto s = [](int j) { return (float)std::sin(-2.0 * M_PI * j / N); };
        const int j0 = np * q, j1 = np * (q + 4);
        w.x[np][q] = bits(c(j0), c(j1));
        w.y[np][q] = bits(s(j0), s(j1));
        w.ny[np][q] = bits(-s(j0), -s(j1));
      }
    return w;
  }();
  return t;
}

// Rotations per CTA when the caller names none: the chunk with the fewest estimated rounds of
// sets over the device's SMs (one CTA each), each CTA charged three sets for its receptor tile
// and its pipeline's start.
int xp_chunk(int ncol, int nrot, int G, int most, int sms) {
  int best = XP_SET * G;
  double best_cost = 1e30;
  for (int c = XP_SET * G; c <= most; c += XP_SET * G) {
    const long ctas = (long)(ncol / XP_COLS) * ((nrot + c - 1) / c);
    const double cost = (double)((ctas + sms - 1) / sms) * (std::min(c, nrot) / (double)(XP_SET * G) + 3.0);
    if (cost < best_cost - 1e-9) {
      best_cost = cost;
      best = c;
    }
  }
  return best;
}

struct XpPlan {
  int jm, G, nst, chunk;
  size_t smem;
};

// The launch's shape: JM covers the ligand box; the most groups, then the deeper ring, that
// shared memory holds beside the records of the longest chunk, else (n = 128, K = 16, boxes of more
// than 64 planes) of a short one: every n, K <= 16 and box has a shape
bool xp_plan(const WaveArgs& a, XpPlan* p) {
  const int R1 = a.n / 8, ncol = a.n * (a.n / 2 + 1);
  const int jn = (a.Lb + R1 - 1) / R1;
  p->jm = jn <= 2 ? 2 : jn <= 4 ? jn : 8;
  p->G = a.n == 32 ? XpShape<32>::GMAX : a.n == 64 ? XpShape<64>::GMAX : XpShape<128>::GMAX;
  p->nst = 3;
  int most = XP_MAX_CHUNK;
  while (xp_layout(a.n, a.K, p->G, p->nst, R1 * p->jm, most).total > kXpSmemCap) {
    if (p->nst == 3) p->nst = 2;
    else if (p->G > 1) --p->G, p->nst = 3;
    else if (most > XP_MIN_CHUNK) most = XP_MIN_CHUNK;
    else return false;
  }
  int dev = 0, sms = 0;
  if (cudaGetDevice(&dev) != cudaSuccess ||
      cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || sms < 1)
    sms = 148;
  p->chunk = a.chunk > 0 ? std::min(most, (a.chunk + XP_SET - 1) / XP_SET * XP_SET)
                         : xp_chunk(ncol, a.nrot, p->G, most, sms);
  p->smem = xp_layout(a.n, a.K, p->G, p->nst, R1 * p->jm, p->chunk).total;
  return true;
}

template <int N, int JM>
cudaError_t launch_xp_jm(const WaveArgs& a, const XpPlan& p, cudaStream_t s) {
  auto kern = k_xpass_pairs<N, JM>;
  // the most that any shape asks for and not this launch's: the attribute is the process's, and another
  // thread's smaller shape, set between this call and the launch, would refuse it
  const cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kXpSmemCap);
  if (e != cudaSuccess) return e;
  constexpr int NCOL = N * (N / 2 + 1);
  kern<<<dim3(NCOL / XP_COLS, (a.nrot + p.chunk - 1) / p.chunk), 128 * p.G, p.smem, s>>>(a, xp_twiddles<N>(), p.chunk,
                                                                                        p.nst);
  return cudaGetLastError();
}

template <int N>
cudaError_t launch_xp(const WaveArgs& a, const XpPlan& p, cudaStream_t s) {
  switch (p.jm) {
    case 2: return launch_xp_jm<N, 2>(a, p, s);
    case 3: return launch_xp_jm<N, 3>(a, p, s);
    case 4: return launch_xp_jm<N, 4>(a, p, s);
    default: return launch_xp_jm<N, 8>(a, p, s);
  }
}

}  // namespace

// Waves that k_xpass_block (block_xpass.cu) searches faster, x pass and inverse pass together; k_xpass_pairs is
// the faster on the other side. Measured, time of the former over the latter:
//   few rotations: a set of four is not full, and the pairs' receptor tile, records and rings take the whole SM
//     before the first one. Boxes up to n/2, K = 2 to 16: n = 32, 3 rotations 0.89-1.08, 4 0.98-1.20
//     (K = 2: 5 0.96-1.0, 6 1.09); 64, 5 0.81-0.97, 8 1.0-1.24; 96, 5 0.68-1.02, 8 0.95-1.41; 128, 3 0.77-0.99,
//     4 0.89-1.23. Larger boxes (eight inputs per first-stage output): 64, 7 rotations about 0.9, 16
//     1.16-1.6; 96, 8 0.62-1.03, 16 0.95-1.2 (K >= 10 0.76-1.1, 32 0.9-1.4); 128, 4 0.6-0.9, 16 0.8-1.4.
//   128^3, boxes far above n/2: beside the receptor tile one group of warps is left per SM. K = 5 to 9, any number of
//     rotations: boxes of 79 planes 1.04-1.14, 86 0.78-1.04, 95 0.77-0.96, 111 0.56-0.7; K = 12, 16 (the block
//     kernel at one CTA per SM): 86 1.16-1.44, 95 0.85-1.14, 102 0.83-0.92; K <= 3 (two groups) 1.3-1.5.
bool xpass_block_stages(const WaveArgs& a) {
  const bool wide = a.Lb > a.n / 2;
  switch (a.n) {
    case 32: return a.nrot <= (a.K <= 2 ? 5 : 3);
    case 64: return a.nrot <= (wide ? 7 : 5);
    case 96: return a.nrot <= (!wide ? 5 : a.K < 10 ? 15 : 24);
    default: return a.nrot <= (wide ? 8 : 3) || (a.K >= 5 && a.Lb > (a.K < 10 ? 80 : 88));
  }
}

void xpass_b_layout(WaveArgs& a) {
  a.bpairs = a.keys2 || a.yz_block_stages || xpass_block_stages(a) ? 0 : 2;
}

bool xpass_col_tile_ok(int n, int col_tile) { return col_tile == 8 || (n <= 64 && col_tile == 16); }

int xpass_rotations_per_cta(const WaveArgs& a) {
  if (!a.bpairs && xpass_block_stages(a)) return kXpassBlockRotations;
  XpPlan p;
  return xp_plan(a, &p) ? p.chunk : 0;
}

int xpass_columns_per_cta(const WaveArgs& a) {
  return !a.bpairs && xpass_block_stages(a) ? xpass_block_columns(a.n, a.K) : XP_COLS;
}

cudaError_t launch_xpass(const WaveArgs& a, cudaStream_t s) {
  XpPlan p;
  if (!a.A || !a.B || a.K < 1 || a.K > KMAX || a.Lb < 1 || a.Lb > a.n || a.nrot < 1 ||
      !xpass_col_tile_ok(a.n, a.col_tile) || !xp_plan(a, &p))
    return cudaErrorInvalidValue;
  if (!a.bpairs && xpass_block_stages(a)) return launch_xpass_block(a, s);
  switch (a.n) {
    case 32: return launch_xp<32>(a, p, s);
    case 64: return launch_xp<64>(a, p, s);
    case 96: return launch_xp<96>(a, p, s);
    case 128: return launch_xp<128>(a, p, s);
    default: return cudaErrorInvalidValue;
  }
}

}  // namespace cdk
