// block_xpass.cu -- the FP32 form's x pass for waves of a few rotations and for the largest boxes: block-wide
// radix stages, a rotation at a time. The same sums in the same order as k_xpass_pairs (fp32_xpass.cu), so
// the same bits; which of the two runs is xpass_block_stages' rule.
//
// A CTA holds a quarter to half of an SM's shared memory and starts on its first rotation as soon as its
// receptor tile is there; k_xpass_pairs takes the whole SM, fills lanes with sets of four rotations and pays for
// its rings and records first.
#include <cuda_runtime.h>
#include <stdint.h>

#include "cdk_internal.h"
#include "fft.cuh"

namespace cdk {
namespace {

// Two-stage plans (N = R0*R1), fused stage by stage; CT spectral columns per CTA:
//   phase A  first forward stage straight from A in global memory (only the x planes a
//            channel touches are read; the rest are known zeros), two channels per round;
//            the next round's loads are issued before this round's phase B to hide latency
//   phase B  second forward stage + conj(L_k) * P_k accumulated in registers over all
//            channels (receptor tile resident in shared memory for the CTA's rotations)
//   combine  pair sum through one shuffle, first inverse stage
//   phase C  last inverse stage, written straight to B for x inside the window
template <int N, int CT>
__global__ void __launch_bounds__(256, 2) k_xpass_block(const __grid_constant__ WaveArgs a, int rot_per_cta) {
  constexpr int NZH = N / 2 + 1;
  constexpr int NCOL = N * NZH;
  constexpr int R0 = FFTPlan<N>::R0, R1 = FFTPlan<N>::R1, M1 = N / R0;
  constexpr int NA = 2 * CT * M1;  // phase-A items
  constexpr int NB = 2 * CT * R0;  // phase-B items
  static_assert(FFTPlan<N>::NS == 2, "two-stage plans only");
  static_assert(NA <= 256 && NB <= 256, "one item per thread");
  static_assert(NCOL % CT == 0, "column tiles must divide the half spectrum");
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int K = a.K;
  float2* tw = reinterpret_cast<float2*>(smem_raw);
  int* s_ch = reinterpret_cast<int*>(tw + N);               // [KMAX] channel ids, [KMAX] count
  short* s_rng = reinterpret_cast<short*>(s_ch + 2 * KMAX);  // [KMAX][2] x range per slot
  float2* Ps = reinterpret_cast<float2*>(s_rng + 4 * KMAX);  // [N][K][CT]
  float2* Wb = Ps + (size_t)N * K * CT;                      // [N][2][CT]
  float2* S = Wb + (size_t)N * 2 * CT;                       // [N][CT]
  const int c0 = blockIdx.x * CT;
  const int tid = threadIdx.x;
  for (int i = tid; i < N; i += 256) tw[i] = a.tw[i];
  for (int i = tid; i < N * K * CT; i += 256) {
    const int c = i % CT, t = i / CT;  // t = pos*K + k
    Ps[i] = a.phat[(size_t)t * NCOL + c0 + c];
  }
  // per-thread roles
  const int a_c = tid % CT, a_half = (tid / CT) & 1, a_np = tid / (2 * CT);
  const int b_half = tid & 1, b_c = (tid >> 1) % CT, b_b = (tid >> 1) / CT;
  const int r_begin = blockIdx.y * rot_per_cta;
  const int r_end = min(a.nrot, r_begin + rot_per_cta);
  for (int r = r_begin; r < r_end; ++r) {
    const RotRec* rec = a.rec + r;
    if (!rec->valid) continue;
    __syncthreads();  // previous rotation is done with s_ch / Wb / S
    if (tid == 0) {
      int nk = 0;
      for (int k = 0; k < K; ++k)
        if (rec->xlo[k] <= rec->xhi[k]) {
          s_rng[2 * nk] = rec->xlo[k];
          s_rng[2 * nk + 1] = rec->xhi[k];
          s_ch[nk++] = k;
        }
      s_ch[KMAX] = nk;
    }
    __syncthreads();
    const int nk = s_ch[KMAX];
    const float2* Ar = a.A + ((size_t)r * K) * a.Lb * NCOL + c0 + a_c;
    // raw loads of one round (channels kk0, kk0+1) for this thread's phase-A item
    auto load_round = [&](int kk0, float2* v) {
      const int kk = kk0 + a_half;
      if (tid < NA && kk < nk) {
        const int k = s_ch[kk];
        const int lo = s_rng[2 * kk], hi = s_rng[2 * kk + 1];
        const float2* src = Ar + (size_t)k * a.Lb * NCOL;
#pragma unroll
        for (int j = 0; j < R0; ++j) {
          const int x = a_np + j * M1;
          v[j] = (x >= lo && x <= hi) ? src[(size_t)x * NCOL] : make_float2(0.f, 0.f);
        }
      } else {
#pragma unroll
        for (int j = 0; j < R0; ++j) v[j] = make_float2(0.f, 0.f);
      }
    };
    float2 acc[R1];
#pragma unroll
    for (int j = 0; j < R1; ++j) acc[j] = make_float2(0.f, 0.f);
    float2 va[R0];
    load_round(0, va);
    for (int k0 = 0; k0 < nk; k0 += 2) {
      // phase A: first forward stage into Wb
      if (tid < NA) {
        Radix<R0, -1>::run(va);
#pragma unroll
        for (int q = 1; q < R0; ++q) va[q] = c_mul(va[q], tw[a_np * q]);
#pragma unroll
        for (int q = 0; q < R0; ++q) Wb[((a_np + q * M1) * 2 + a_half) * CT + a_c] = va[q];
      }
      __syncthreads();
      if (k0 + 2 < nk) load_round(k0 + 2, va);  // in flight during phase B
      // phase B: second forward stage and the conjugate product, accumulated
      const int kk = k0 + b_half;
      if (tid < NB && kk < nk) {
        const int k = s_ch[kk];
        float2 v[R1];
#pragma unroll
        for (int j = 0; j < R1; ++j) v[j] = Wb[((b_b * R1 + j) * 2 + b_half) * CT + b_c];
        Radix<R1, -1>::run(v);
#pragma unroll
        for (int q = 0; q < R1; ++q) {
          const float2 p = Ps[((b_b * R1 + q) * K + k) * CT + b_c];
          acc[q].x += v[q].x * p.x + v[q].y * p.y;
          acc[q].y += v[q].x * p.y - v[q].y * p.x;
        }
      }
      __syncthreads();
    }
    // combine the pair (lanes tid, tid^1), first inverse stage, into S
    if (tid < ((NB + 31) & ~31)) {
      float2 v[R1];
#pragma unroll
      for (int j = 0; j < R1; ++j) {
        v[j].x = acc[j].x + __shfl_xor_sync(0xffffffffu, acc[j].x, 1);
        v[j].y = acc[j].y + __shfl_xor_sync(0xffffffffu, acc[j].y, 1);
      }
      if (tid < NB && b_half == 0) {
        Radix<R1, +1>::run(v);
#pragma unroll
        for (int j = 0; j < R1; ++j) S[(b_b * R1 + j) * CT + b_c] = v[j];
      }
    }
    __syncthreads();
    // phase C: last inverse stage, window rows only
    const int Wx = rec->W[0];
    if (tid < CT * M1) {
      const int c = tid % CT, np = tid / CT;
      float2 v[R0];
#pragma unroll
      for (int q = 0; q < R0; ++q) {
        v[q] = S[(np + q * M1) * CT + c];
        if (q > 0) v[q] = c_mulc(v[q], tw[np * q]);
      }
      Radix<R0, +1>::run(v);
      float2* dst = a.B + (size_t)r * N * NCOL + c0 + c;
#pragma unroll
      for (int j = 0; j < R0; ++j) {
        const int x = np + j * M1;
        if (x < Wx) dst[(size_t)x * NCOL] = v[j];
      }
    }
  }
}

constexpr size_t block_smem(int n, int ct, int K) {
  return sizeof(float2) * n + sizeof(int) * 2 * KMAX + sizeof(short) * 4 * KMAX + sizeof(float2) * (size_t)n * ct * (K + 3);
}

template <int N, int CT>
cudaError_t launch_ct(const WaveArgs& a, cudaStream_t s) {
  auto kern = k_xpass_block<N, CT>;
  // the most that any K asks for: the attribute is the process's (other threads' contexts)
  const cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)block_smem(N, CT, KMAX));
  if (e != cudaSuccess) return e;
  constexpr int NCOL = N * (N / 2 + 1);
  // a receptor tile serves 32 rotations, which leaves enough CTAs for the scheduler
  constexpr int per = kXpassBlockRotations;
  kern<<<dim3(NCOL / CT, (a.nrot + per - 1) / per), 256, block_smem(N, CT, a.K), s>>>(a, per);
  return cudaGetLastError();
}

template <int N>
cudaError_t launch_n(const WaveArgs& a, cudaStream_t s) {
  if constexpr (N <= 64) {
    if (xpass_block_columns(N, a.K) == 16) return launch_ct<N, 16>(a, s);
  }
  return launch_ct<N, 8>(a, s);
}

}  // namespace

// 16 columns where the buffers stay within about 110 KB (two CTAs per SM), else 8
int xpass_block_columns(int n, int K) { return n <= 64 && block_smem(n, 16, K) <= 110 * 1024 ? 16 : 8; }

cudaError_t launch_xpass_block(const WaveArgs& a, cudaStream_t s) {
  switch (a.n) {
    case 32: return launch_n<32>(a, s);
    case 64: return launch_n<64>(a, s);
    case 96: return launch_n<96>(a, s);
    case 128: return launch_n<128>(a, s);
    default: return cudaErrorInvalidValue;
  }
}

}  // namespace cdk
