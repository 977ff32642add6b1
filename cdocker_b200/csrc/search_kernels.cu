// search_kernels.cu -- the FP32 FFT translational-rotational search on sm_100a.
//
// One wave of rotations runs five kernels, all on one stream:
//   prep          rotate atoms (reference op order, no contraction), bounding box, windows,
//                 per-channel x-plane ranges          (src/Rotate.cpp, GetMin/MaxCoors.cpp)
//   spread_yz     per rotation (up to 96 atoms): the (y,z) spectra of the planes its atoms touch as
//                 sums of separable spectra of their trilinear weights -> A; larger ligands, per
//                 (rotation, channel, x plane): spread the atoms into shared memory (FillLigandGrid's
//                 arithmetic), then the 2-D real-to-complex FFT   (src/FillLigandGrid.cpp)
//   xpass         (fp32_xpass.cu; block_xpass.cu for a few rotations) per spectral column tile: FFT along x
//                 of every channel, the conjugate product with the resident receptor spectra summed over
//                 channels, and the inverse FFT along x, keeping only the translation window -> B
//                                                       (src/kernel.cu ConjMult + SumGrids)
//   yz_inv_argmin (yz_pairs.cu) per (rotation, planes x, x + 1 in window): inverse FFT over y, complex-
//                 to-real over z, min / first argmin over the window, folded into one 64-bit key per
//                 rotation                (src/TranRotaConfSearchNoMini.cu:429-464)
//   finalize      keys -> minE, (i,j,k)
// The energy grid never leaves shared memory. Spectra stay in the digit-reversed order the
// in-place FFT stages produce; the receptor spectra are computed by the same stages, so
// the pointwise product lines up without any permutation.
#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include <algorithm>

#include "cdk_internal.h"
#include "fft.cuh"
#include "pair_fft.cuh"
#include "window_keys.cuh"

namespace cdk {

namespace {

// (a, b) -> packed bf16x2 hi = rn(a), rn(b) and lo = rn(a - hi), rn(b - hi); a in the low half
__device__ __forceinline__ void split_bf16x2(float a, float b, uint32_t& hi, uint32_t& lo) {
  const __nv_bfloat162 h = __floats2bfloat162_rn(a, b);
  const float2 hf = __bfloat1622float2(h);
  const __nv_bfloat162 l = __floats2bfloat162_rn(a - hf.x, b - hf.y);
  hi = *reinterpret_cast<const uint32_t*>(&h);
  lo = *reinterpret_cast<const uint32_t*>(&l);
}

// one 32-byte store (p 32-byte aligned): words w0..w3 then w4..w7
__device__ __forceinline__ void st_v8u(void* p, uint4 lo, uint4 hi) {
  asm volatile("st.global.v8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"l"(p), "r"(lo.x), "r"(lo.y),
               "r"(lo.z), "r"(lo.w), "r"(hi.x), "r"(hi.y), "r"(hi.z), "r"(hi.w)
               : "memory");
}

// Tiled ligand rows (WaveArgs.lop_tiled): (tile r / 128, channel k, chunk jc) is a row set of
// 128 rotations x ncol columns; rotation m = r % 128 keeps its columns side by side, so the lanes
// of a warp (consecutive columns) write one contiguous run. Rows are in natural order: the x
// pass's tensor copies gather column c of the 128 rotations and apply the tensor cores' swizzle.
__device__ __forceinline__ unsigned char* tiled_row(const WaveArgs& a, int r, int k, int jc, int c, int row_bytes) {
  const int ncol = a.n * (a.n / 2 + 1);
  const size_t set = ((size_t)(r / kTileRot) * a.K + k) * 4 + jc;
  return a.lop + ((set * kTileRot + (size_t)(r % kTileRot)) * ncol + c) * (size_t)row_bytes;
}

// split-FP16: one 32-byte row [re | im] of the 8 planes
__device__ __forceinline__ void tiled_row_store(const WaveArgs& a, int r, int k, int jc, int c, uint4 re, uint4 im) {
  st_v8u(tiled_row(a, r, k, jc, c, 32), re, im);
}

// split-BF16: one 64-byte row [hi re | hi im | lo re | lo im]; the x pass reads the lo part 32
// bytes into the same rows. rows[0..3]: hi re, hi im, lo re, lo im.
__device__ __forceinline__ void tiled_row_store64(const WaveArgs& a, int r, int k, int jc, int c, const uint4* rows) {
  uint4* dst = reinterpret_cast<uint4*>(tiled_row(a, r, k, jc, c, 64));
  st_v8u(dst, rows[0], rows[1]);
  st_v8u(dst + 2, rows[2], rows[3]);
}


// ---------------------------------------------------------------------------------------
// exact-order float rotation (src/QuaternionMultiply.cpp:3-11, src/Rotate.cpp:4-27)
__device__ __forceinline__ void qmul_rn(const float* l, const float* r, float* o) {
  o[0] = __fsub_rn(__fsub_rn(__fsub_rn(__fmul_rn(l[0], r[0]), __fmul_rn(l[1], r[1])),
                             __fmul_rn(l[2], r[2])),
                   __fmul_rn(l[3], r[3]));
  o[1] = __fsub_rn(__fadd_rn(__fadd_rn(__fmul_rn(l[0], r[1]), __fmul_rn(l[1], r[0])),
                             __fmul_rn(l[2], r[3])),
                   __fmul_rn(l[3], r[2]));
  o[2] = __fadd_rn(__fadd_rn(__fsub_rn(__fmul_rn(l[0], r[2]), __fmul_rn(l[1], r[3])),
                             __fmul_rn(l[2], r[0])),
                   __fmul_rn(l[3], r[1]));
  o[3] = __fadd_rn(__fsub_rn(__fadd_rn(__fmul_rn(l[0], r[3]), __fmul_rn(l[1], r[2])),
                             __fmul_rn(l[2], r[1])),
                   __fmul_rn(l[3], r[0]));
}

__device__ __forceinline__ void rotate_rn(const float* q, float vx, float vy, float vz,
                                          float* out) {
  float qc[4] = {q[0], -q[1], -q[2], -q[3]};
  float qv[4] = {0.0f, vx, vy, vz};
  float t1[4], t2[4];
  qmul_rn(q, qv, t1);
  qmul_rn(t1, qc, t2);
  out[0] = t2[1];
  out[1] = t2[2];
  out[2] = t2[3];
}

// cell index of a coordinate, FillLigandGrid's double arithmetic (src/FillLigandGrid.cpp:28-30)
__device__ __forceinline__ int cell_of(float x, float mn, float h) {
  return (int)__ddiv_rn(__dsub_rn((double)x, (double)mn), (double)h);
}
// ratio within the cell (src/FillLigandGrid.cpp:33-35): `index * spacing` is a float product
__device__ __forceinline__ double ratio_of(float x, float mn, float h, int i) {
  return __ddiv_rn(__dsub_rn(__dsub_rn((double)x, (double)mn), (double)__fmul_rn((float)i, h)),
                   (double)h);
}

// ---------------------------------------------------------------------------------------
// prep: one warp per rotation
__global__ void __launch_bounds__(128) k_prep(WaveArgs a) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int r = blockIdx.x * 4 + warp;
  __shared__ int s_lo[4][KMAX], s_hi[4][KMAX], s_ext[4][3];
  if (lane < KMAX) {
    s_lo[warp][lane] = 0x7fff;
    s_hi[warp][lane] = -1;
  }
  if (lane < 3) s_ext[warp][lane] = 0;
  __syncwarp();
  if (r >= a.nrot) return;
  const RotDesc rd = a.rots[r];
  const ConfDesc cd = a.confs[rd.conf];
  const int nA = min(cd.n_atoms, a.max_atoms);
  const float* xyz = a.coords + (size_t)cd.coord_off * 3;
  float mn[3] = {INFINITY, INFINITY, INFINITY}, mx[3] = {-INFINITY, -INFINITY, -INFINITY};
  for (int i = lane; i < nA; i += 32) {
    float p[3];
    rotate_rn(rd.q, xyz[i * 3 + 0], xyz[i * 3 + 1], xyz[i * 3 + 2], p);
    a.rot_xyz[(size_t)r * a.max_atoms + i] = make_float4(p[0], p[1], p[2], 0.0f);
#pragma unroll
    for (int d = 0; d < 3; ++d) {
      mn[d] = fminf(mn[d], p[d]);
      mx[d] = fmaxf(mx[d], p[d]);
    }
  }
#pragma unroll
  for (int d = 0; d < 3; ++d)
    for (int o = 16; o > 0; o >>= 1) {
      mn[d] = fminf(mn[d], __shfl_xor_sync(0xffffffffu, mn[d], o));
      mx[d] = fmaxf(mx[d], __shfl_xor_sync(0xffffffffu, mx[d], o));
    }
  const float h = a.spacing;
  int W[3];
#pragma unroll
  for (int d = 0; d < 3; ++d) W[d] = a.n - (int)__fdiv_rn(__fsub_rn(mx[d], mn[d]), h) - 2;
  const bool valid = nA > 0 && W[0] > 0 && W[1] > 0 && W[2] > 0;
  __syncwarp();
  // per-channel x range and touched extents
  const AtomParam* prm = a.params + cd.param_off;
  const int elec = a.K - 1;
  for (int i = lane; i < nA; i += 32) {
    float4 p = a.rot_xyz[(size_t)r * a.max_atoms + i];
    int ci[3] = {cell_of(p.x, mn[0], h), cell_of(p.y, mn[1], h), cell_of(p.z, mn[2], h)};
    const int sl = prm[i].slot;
    if (sl >= 0 && sl < elec) {
      atomicMin(&s_lo[warp][sl], ci[0]);
      atomicMax(&s_hi[warp][sl], ci[0] + 1);
    }
    atomicMin(&s_lo[warp][elec], ci[0]);
    atomicMax(&s_hi[warp][elec], ci[0] + 1);
#pragma unroll
    for (int d = 0; d < 3; ++d) atomicMax(&s_ext[warp][d], ci[d] + 2);
  }
  __syncwarp();
  bool range_bad = false;
  if (a.f16 && a.range_err) {
    // split-FP16 form: |A(x, ky, kz)| <= sum over the channel's atoms of |s_a| (x weights and
    // |Fy|, |Fz| are at most 1), so the scaled ligand rows fit FP16 when this bound does
    bool bad = false;
    if (lane < a.K) {
      float bound = 0.f;
      for (int i = 0; i < nA; ++i) {
        if (lane == elec) bound += fabsf(prm[i].charge);
        else if (prm[i].slot == lane) bound += fabsf(prm[i].w_vdw);
      }
      bad = bound * a.lscale[lane] > 60000.f;
    }
    range_bad = __any_sync(0xffffffffu, bad);
    if (range_bad && lane == 0) atomicOr(a.range_err, 1);
  }
  RotRec* rec = a.rec + r;
  if (lane < KMAX) {
    const bool used = lane < a.K && s_hi[warp][lane] >= 0;
    rec->xlo[lane] = used ? (short)s_lo[warp][lane] : (short)1;
    rec->xhi[lane] = used ? (short)s_hi[warp][lane] : (short)0;
  }
  if (lane == 0) {
    // err 1: the x planes of a channel leave the planned box, or y/z cells the grid;
    // err 2: a scaled ligand value would leave the FP16 range (split-FP16 form). Either makes
    // the rotation invalid (no kernel after this one touches it)
    int err = 0;
    if (valid && (s_ext[warp][0] - 1 >= a.Lb || s_ext[warp][1] > a.n || s_ext[warp][2] > a.n))
      err = 1;
    else if (valid && range_bad)
      err = 2;
#pragma unroll
    for (int d = 0; d < 3; ++d) {
      rec->mn[d] = mn[d];
      rec->W[d] = W[d];
    }
    rec->ext_y = s_ext[warp][1];
    rec->valid = (valid && !err) ? 1 : 0;
    rec->err = err;
    rec->nA = nA;
    rec->param_off = cd.param_off;
    a.keys[r] = ~0ull;
  }
}

// ---------------------------------------------------------------------------------------
// shared helpers for the (y,z) plane transforms
//   P: packed real rows, pair p holds rows 2p (real part) and 2p+1 (imag part), stride n+1
//   O: half spectrum over z, [y][kz] with stride nzh (row y, col kz)

// z: R2C of `npairs` packed row pairs in P, then split into O rows (2p, 2p+1)
template <int N>
__device__ __forceinline__ void plane_forward(float2* P, float2* O, int npairs,
                                              const float2* tw) {
  constexpr int NZH = N / 2 + 1;
  const int tid = threadIdx.x, nthr = blockDim.x;
  fft_lines<N, false>(P, npairs, N + 1, 1, tw, tid, nthr);
  for (int i = tid; i < (N / 2) * NZH; i += nthr) {
    const int p = i / NZH, kz = i - p * NZH;
    float2 A = make_float2(0.f, 0.f), Bv = make_float2(0.f, 0.f);
    if (p < npairs) {
      const float2 zk = P[p * (N + 1) + fft_pos<N>(kz)];
      const float2 zn = P[p * (N + 1) + fft_pos<N>((N - kz) % N)];
      A = make_float2(0.5f * (zk.x + zn.x), 0.5f * (zk.y - zn.y));
      Bv = make_float2(0.5f * (zk.y + zn.y), -0.5f * (zk.x - zn.x));
    }
    O[(2 * p) * NZH + kz] = A;
    O[(2 * p + 1) * NZH + kz] = Bv;
  }
  __syncthreads();
  // y: complex FFT on the nzh columns
  fft_lines<N, false>(O, NZH, 1, NZH, tw, tid, nthr);
}

// ---------------------------------------------------------------------------------------
// an atom on the plane being spread: y and z cells and ratios, its weight times the x weight
struct SpreadAtom {
  double yr, zr, w;
  int yi, zi;
};

// spread + forward (y,z) transform of one (rotation, channel, x plane)
template <int N>
__global__ void __launch_bounds__(256) k_spread_yz(WaveArgs a) {
  constexpr int NZH = N / 2 + 1;
  constexpr int NCOL = N * NZH;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  float2* tw = reinterpret_cast<float2*>(smem_raw);
  float2* O = tw + N;
  float2* P = O + N * NZH;
  const int x = blockIdx.x, k = blockIdx.y, r = blockIdx.z;
  const RotRec* rec = a.rec + r;
  if (!rec->valid) return;
  const int xlo = rec->xlo[k], xhi = rec->xhi[k];
  if (x < xlo || x > xhi) return;
  const int tid = threadIdx.x, nthr = blockDim.x;
  for (int i = tid; i < N; i += nthr) tw[i] = a.tw[i];
  const int npairs = min(N / 2, (rec->ext_y + 1) / 2);
  float* Pf = reinterpret_cast<float*>(P);
  for (int i = tid; i < npairs * (N + 1); i += nthr) P[i] = make_float2(0.f, 0.f);
  __syncthreads();
  // spread the atoms touching plane x (src/FillLigandGrid.cpp:24-66 vdW, :75-118 elec). The cells
  // and ratios of up to 256 atoms at a time by a thread each, compacted in ascending order; then
  // warp 0 adds the atoms one after another, the four (y,z) corners of an atom in four lanes (they
  // never share a cell), the weights of eight atoms computed together, each add rounded back to
  // float from double as in the reference: the plane is bit-identical to FillLigandGrid's and the
  // search is deterministic whatever the batch around a rotation. (With the divisions of an atom's
  // cells and ratios in warp 0's loop as well, 2.14 against 1.98 ms per 1,000 rotations of a 100-atom
  // ligand at 64^3.)
  __shared__ int s_warp[8];
  __shared__ SpreadAtom s_at[256];
  const AtomParam* prm = a.params + rec->param_off;
  const float mn0 = rec->mn[0], mn1 = rec->mn[1], mn2 = rec->mn[2];
  const float h = a.spacing;
  const bool elec = (k == a.K - 1);
  const int nA = rec->nA;
  for (int base = 0; base < nA; base += 256) {
    const int i = base + tid, lane = tid & 31;
    bool touch = false;
    int xi = 0;
    float4 p;
    AtomParam ap;
    if (i < nA) {
      ap = prm[i];
      if (elec || ap.slot == k) {
        p = a.rot_xyz[(size_t)r * a.max_atoms + i];
        xi = cell_of(p.x, mn0, h);
        touch = (xi == x) || (xi + 1 == x);
      }
    }
    const unsigned int m = __ballot_sync(0xffffffffu, touch);
    if (lane == 0) s_warp[tid >> 5] = __popc(m);
    __syncthreads();
    int at = 0, cnt = 0;
    for (int w = 0; w < 8; ++w) {
      if (w < (tid >> 5)) at += s_warp[w];
      cnt += s_warp[w];
    }
    if (touch) {
      const double xr = ratio_of(p.x, mn0, h, xi);
      SpreadAtom sa;
      sa.yi = cell_of(p.y, mn1, h);
      sa.zi = cell_of(p.z, mn2, h);
      sa.yr = ratio_of(p.y, mn1, h, sa.yi);
      sa.zr = ratio_of(p.z, mn2, h, sa.zi);
      sa.w = __dmul_rn(elec ? (double)ap.charge : (double)ap.w_vdw, (xi == x) ? __dsub_rn(1.0, xr) : xr);
      s_at[at + __popc(m & ((1u << lane) - 1))] = sa;
    }
    __syncthreads();
    if (tid < 32) {
      for (int j0 = 0; j0 < cnt; j0 += 8) {
        const int j = j0 + (lane >> 2), dy = (lane >> 1) & 1, dz = lane & 1;
        float* cell = nullptr;
        double w = 0.0;
        if (j < cnt) {
          const SpreadAtom sa = s_at[j];
          w = __dmul_rn(__dmul_rn(sa.w, dy ? sa.yr : __dsub_rn(1.0, sa.yr)), dz ? sa.zr : __dsub_rn(1.0, sa.zr));
          const int y = sa.yi + dy, z = sa.zi + dz;
          if (y < N && z < N) cell = &Pf[((y >> 1) * (N + 1) + z) * 2 + (y & 1)];
        }
        for (int o = 0; o < min(8, cnt - j0); ++o) {
          if ((lane >> 2) == o && cell) *cell = (float)__dadd_rn((double)*cell, w);
          __syncwarp();
        }
      }
    }
    __syncthreads();
  }
  plane_forward<N>(P, O, npairs, tw);
  // write the plane's half spectrum (16-byte stores)
  float4* dst = reinterpret_cast<float4*>(a.A + (((size_t)r * a.K + k) * a.Lb + x) * NCOL);
  const float4* src = reinterpret_cast<const float4*>(O);
  for (int i = tid; i < NCOL / 2; i += nthr) dst[i] = src[i];
}

// ---------------------------------------------------------------------------------------
// Direct (y,z) spectrum of the spread planes of one (rotation, channel).
// The spread is a sum of separable cloud-in-cell kernels, so the 2-D DFT of plane x is
//   A(x, ky, kz) = sum_{atoms a touching x} s_a wx_a(x) Fy_a(ky) Fz_a(kz),
//   Fy_a(ky) = (1 - ry) w^(yi ky) + ry w^((yi+1) ky),   w = exp(-2 pi i / n)
// (the same numbers the spread + radix FFT produce, without the float rounding of the plane).
// Per-atom factor tables in shared memory, then every touched plane's n*(n/2+1) outputs, written in
// the (ky position, kz) order of the FFT path. Atoms are visited in ascending order for every plane:
// deterministic.
// What the plane kernel writes: FP32 planes (A), or the tensor-core x pass's ligand rows (lop)
constexpr int kRowsNone = 0, kRowsF16 = 1, kRowsBf16 = 2;

// One column's 8-plane chunk jc as ligand rows, h: the rows' 16-byte words -- split-FP16: [re, im]
// of the planes times 2^sigma_k (already in the atoms' x weights; k_prep has checked that the
// scaled planes stay inside the FP16 range); split-BF16: [hi re, hi im, lo re, lo im]. Untiled: per
// (rotation, channel) 8 or 16 rows [hi, lo][chunk][re, im] of ncol x 16 B, the tensor-core x
// pass's K order, in 512 B blocks of (8 rotations x 4 columns) x 16 B.
template <int N, int ROWS>
__device__ __forceinline__ void plane_rows_write(const WaveArgs& a, int r, int k, int jc, int c, const uint4* h) {
  constexpr int NCOL = N * (N / 2 + 1);
  constexpr int PER = ROWS == kRowsF16 ? 8 : 16;
  if (a.lop_tiled) {
    if constexpr (ROWS == kRowsF16) tiled_row_store(a, r, k, jc, c, h[0], h[1]);
    else tiled_row_store64(a, r, k, jc, c, h);
    return;
  }
  uint4* dst = reinterpret_cast<uint4*>(a.lop) +
               (((size_t)(r >> 3) * a.K + k) * PER * (NCOL / 4) + (c >> 2)) * 32 + (r & 7) * 4 + (c & 3);
  constexpr size_t RS = (size_t)(NCOL / 4) * 32;  // one row
#pragma unroll
  for (int i = 0; i < PER / 4; ++i) dst[(((i >> 1) * 4 + jc) * 2 + (i & 1)) * RS] = h[i];
}

// Tiled rows: zeros for a chunk of the tile's stage plan that this rotation's channel does not
// touch (the x pass's tensor copies load the rows of all 128 rotations of a row set)
__device__ __forceinline__ void tiled_zero_chunk(const WaveArgs& a, int r, int k, int jc, int c) {
  const uint4 z = make_uint4(0u, 0u, 0u, 0u);
  if (a.f16) {
    tiled_row_store(a, r, k, jc, c, z, z);
  } else {
    const uint4 zz[4] = {z, z, z, z};
    tiled_row_store64(a, r, k, jc, c, zz);
  }
}

// The K-step range [lo, hi] of channel k in the stage plan of rotation r's tile (k_tile_plan);
// lo > hi when no rotation of the tile touches the channel
__device__ __forceinline__ void tile_plan_range(const WaveArgs& a, int r, int k, int& lo, int& hi) {
  const unsigned long long* tp = a.rec[r - r % kTileRot].tplan;
  const unsigned long long pk = tp[0], pl = tp[1], ph = tp[2];
  const int nact = (int)(tp[3] & 0xFFFFu);
  lo = 15;
  hi = -1;
  for (int ai = 0; ai < nact; ++ai)
    if ((int)((pk >> (4 * ai)) & 15) == k) {
      lo = (int)((pl >> (4 * ai)) & 15);
      hi = (int)((ph >> (4 * ai)) & 15);
    }
}

// Largest ligand of the direct plane kernel (larger ones keep FillLigandGrid's 64-bit weights, in the FFT
// planes)
constexpr int kDirectMaxAtoms = 96;

// Shape of the direct plane kernel: threads per CTA and CTAs per SM asked for (registers), shared
// memory for ligands of at most cap atoms
template <int N, int ROWS>
struct DirectShape {
  static constexpr int NZH = N / 2 + 1, NCOL = N * NZH;
  static constexpr int Q = NCOL / 4;  // column quads: c, c + Q, c + 2 Q, c + 3 Q share kz
  static_assert(NCOL % 4 == 0 && Q % NZH == 0, "a quad's columns share kz");
  // measured (ms), ligands of 40 atoms (32^3 24, 96^3 80, 128^3 60); shared memory grows with the atoms, and above
  // about 80 fewer CTAs are resident than asked for. Planes at 64^3, 5,000 rotations: 384 x 2 1.52, 256 x 3 1.65; at 32^3 256 x 3 is the
  // faster; FP16 rows at 64^3, 1e5 rotations: 256 x 3 27.1, 384 x 2 27.7, 192 x 4 27.4; at 128^3, 4,000:
  // 384 x 2 5.6, 256 x 3 6.2 (shared memory holds two CTAs); BF16 rows, 64 result words per thread: at
  // 64^3, 2e4: 192 x 3 9.7, 256 x 2 10.0; at 96^3, 2,000: 2.35 and 2.30; at 128^3, 1,000: 384 x 1 2.5,
  // 192 x 3 3.0
  static constexpr bool WIDE = ROWS == kRowsNone ? N >= 64 : ROWS == kRowsF16 ? N >= 96 : N >= 128;
  static constexpr int T = WIDE ? 384 : ROWS == kRowsBf16 && N <= 64 ? 192 : 256;
  static constexpr int CTAS = ROWS == kRowsBf16 ? (N == 128 ? 1 : N == 96 ? 2 : 3) : WIDE ? 2 : 3;
  static size_t smem(int cap) {
    return sizeof(float2) * (N + (size_t)cap * (N + NZH)) + (4 + 1 + 1) * sizeof(int4) * cap + sizeof(float2) * cap;
  }
};

// Bound: DRAM writes and issue slots together. CTA = a rotation (and a part of its items): cells,
// weights and the separable factors of every atom once, for the atom's vdW channel and the
// electrostatic one. An item is a chunk of 8 planes of one channel; a warp evaluates 32 column quads
// of it, plane by plane: the atoms of a plane come from a list in ascending order (an atom is in the
// lists of its planes xi and xi + 1), so a visit is a fixed sequence of 4 shared loads, 16 scalar
// FMAs (the four columns' Fy Fz) and 4 packed ones (weight times product into the plane's sums).
// Before, a CTA per (rotation, channel) walked a chunk's atoms with a switch on each one's plane
// offset, two columns per thread: 264 k warp instructions per rotation at 64^3, K = 9, 40 atoms,
// 10 % of them floating point. ms before -> now: FP16 rows 64^3, 1e5 rotations 36 -> 27 (the writes'
// floor 23), 96^3, 2,107: 3.5 -> 1.9, 128^3, 4,000: 9.0 -> 5.6; BF16 rows 64^3, 2e4: 10.2 -> 9.7 (floor
// 9.4); planes 64^3, 5,000: 1.77 -> 1.52 (floor 1.35), 128^3, 1,000: 2.25 -> 1.75. Bit-identical.
template <int N, int ROWS>
__global__ void __launch_bounds__(DirectShape<N, ROWS>::T, DirectShape<N, ROWS>::CTAS)
    k_spread_yz_direct(const __grid_constant__ WaveArgs a, const int* __restrict__ kyof, int cap) {
  using S = DirectShape<N, ROWS>;
  constexpr int NZH = S::NZH, NCOL = S::NCOL, Q = S::Q, NY = N / 4, T = S::T, NW = T / 32;
  constexpr bool LOP = ROWS != kRowsNone;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  int4* s_cell = reinterpret_cast<int4*>(smem_raw);                // [cap] x, y, z cells, slot
  float4* s_w = reinterpret_cast<float4*>(s_cell + cap);           // [cap] vdW w(xi), w(xi+1), elec w(xi), w(xi+1)
  int4* s_list = reinterpret_cast<int4*>(s_w + cap);               // [4 cap] (w, w, Fy offset, Fz offset)
  float4* Fy = reinterpret_cast<float4*>(s_list + 4 * cap);        // [cap][NY][2]: re, re, im, im of positions
                                                                   // (p, p + NY) and (p + 2 NY, p + 3 NY)
  float2* Fz = reinterpret_cast<float2*>(Fy + (size_t)cap * NY * 2);  // [cap][NZH]
  float2* tw = Fz + (size_t)cap * NZH;                             // [N]
  float2* s_rr = tw + N;                                           // [cap] y and z ratios
  constexpr int kDirectWords = kDirectMaxAtoms / 32;
  __shared__ uint32_t s_plane[N][kDirectWords];   // atoms with a cell on the plane (bit j)
  __shared__ uint32_t s_chan[KMAX][kDirectWords];  // atoms of the channel
  __shared__ uint32_t s_run[KMAX][N];             // list entries of (channel, plane): first | count << 16
  __shared__ uint16_t s_item[KMAX * (N / 8)];     // channel | chunk << 4 | untouched << 8
  __shared__ int s_nitems;
  const int r = blockIdx.y;
  const RotRec* rec = a.rec + r;
  if (!rec->valid) return;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int K = a.K, elec = K - 1;
  const int na = min(rec->nA, cap);
  const AtomParam* prm = a.params + rec->param_off;
  const float mn0 = rec->mn[0], mn1 = rec->mn[1], mn2 = rec->mn[2];
  const float h = a.spacing;
  for (int i = tid; i < N; i += T) tw[i] = a.tw[i];
  // per atom: cells, ratios and x weights (FillLigandGrid's double arithmetic, once per atom);
  // split-FP16 rows carry 2^sigma_k: a power of two, folded exactly into the x weights (every
  // product and sum below then scales exactly, outside under- and overflow)
  for (int j = tid; j < na; j += T) {
    const AtomParam ap = prm[j];
    const float4 p = a.rot_xyz[(size_t)r * a.max_atoms + j];
    const int xi = cell_of(p.x, mn0, h), yi = cell_of(p.y, mn1, h), zi = cell_of(p.z, mn2, h);
    const double xr = ratio_of(p.x, mn0, h, xi);
    const bool vdw = ap.slot >= 0 && ap.slot < elec;
    const float sv = ROWS == kRowsF16 && vdw ? a.lscale[vdw ? ap.slot : 0] : 1.f, se = ROWS == kRowsF16 ? a.lscale[elec] : 1.f;
    const double wv = (double)ap.w_vdw, we = (double)ap.charge;
    const bool next = xi + 1 < N;
    s_cell[j] = make_int4(xi, yi, zi, vdw ? ap.slot : -1);
    s_w[j] = make_float4(__fmul_rn((float)(wv * (1.0 - xr)), sv), next ? __fmul_rn((float)(wv * xr), sv) : 0.f,
                         __fmul_rn((float)(we * (1.0 - xr)), se), next ? __fmul_rn((float)(we * xr), se) : 0.f);
    s_rr[j] = make_float2((float)ratio_of(p.y, mn1, h, yi), (float)ratio_of(p.z, mn2, h, zi));
  }
  // items: the touched chunks of every channel and, for tiled rows, the chunks of the tile's stage
  // plan that this rotation does not touch (zeros)
  const int chunks = (rec->xhi[elec] >> 3) + 1;  // elec: every atom; planes < n, so <= n / 8
  if (warp == 0) {
    int lo = 1, hi = 0, own_lo = 1, own_hi = 0;
    if (lane < K) {
      const int xlo = rec->xlo[lane], xhi = rec->xhi[lane];
      if (xlo <= xhi) own_lo = lo = xlo >> 3, own_hi = hi = xhi >> 3;
      if (LOP && a.lop_tiled) tile_plan_range(a, r, lane, lo, hi);
    }
    const int cnt = max(0, hi - lo + 1);
    int end = cnt;
    for (int o = 1; o < 32; o <<= 1) {
      const int v = __shfl_up_sync(0xffffffffu, end, o);
      if (lane >= o) end += v;
    }
    for (int q = lo; q <= hi; ++q)
      s_item[end - cnt + q - lo] = (uint16_t)(lane | q << 4 | (q < own_lo || q > own_hi ? 256 : 0));
    if (lane == 31) s_nitems = end;
  }
  __syncthreads();
  // factor tables
  for (int i = tid; i < na * (N + NZH); i += T) {
    const int j = i / (N + NZH), f = i - j * (N + NZH);
    if (f < N) {
      const int yi = s_cell[j].y;
      const float ry = s_rr[j].x;
      const int ky = kyof[f];  // natural frequency of position f
      const float2 w0 = tw[(yi * ky) % N], w1 = tw[((yi + 1) * ky) % N];
      float* d = reinterpret_cast<float*>(Fy + ((size_t)j * NY + f % NY) * 2 + f / (2 * NY)) + f / NY % 2;
      d[0] = (1.f - ry) * w0.x + ry * w1.x;
      d[2] = (1.f - ry) * w0.y + ry * w1.y;
    } else {
      const int kz = f - N;
      const int zi = s_cell[j].z;
      const float rz = s_rr[j].y;
      const float2 w0 = tw[(zi * kz) % N], w1 = tw[((zi + 1) * kz) % N];
      Fz[(size_t)j * NZH + kz] = make_float2((1.f - rz) * w0.x + rz * w1.x, (1.f - rz) * w0.y + rz * w1.y);
    }
  }
  // atoms per plane and per channel (ballots), then the lists: channels in order, planes ascending
  // within a channel, atoms ascending within a plane
  for (int x = warp; x < 8 * chunks + K; x += NW) {
#pragma unroll
    for (int wd = 0; wd < kDirectWords; ++wd) {
      const int j = 32 * wd + lane;
      const int4 c = j < na ? s_cell[j] : make_int4(-2, 0, 0, -2);
      const int k = x - 8 * chunks;
      const unsigned int m =
          __ballot_sync(0xffffffffu, k < 0 ? (c.x == x || c.x + 1 == x) : j < na && (k == elec || c.w == k));
      if (lane == 0) (k < 0 ? s_plane[x] : s_chan[k])[wd] = m;
    }
  }
  __syncthreads();
  for (int i = tid; i < K * 8 * chunks; i += T) {
    const int k = i / (8 * chunks), x = i - k * (8 * chunks);
    uint32_t ch[kDirectWords];
    int first = 0, total = 0;
    for (int kk = 0; kk < k; ++kk)  // an atom has at most two entries per channel
#pragma unroll
      for (int wd = 0; wd < kDirectWords; ++wd) first += 2 * __popc(s_chan[kk][wd]);
#pragma unroll
    for (int wd = 0; wd < kDirectWords; ++wd) {
      ch[wd] = s_chan[k][wd];
      total += __popc(ch[wd]);
    }
    if (total) {
      for (int y = 0; y < x; ++y)
#pragma unroll
        for (int wd = 0; wd < kDirectWords; ++wd) first += __popc(s_plane[y][wd] & ch[wd]);
    }
    int at = first;
#pragma unroll
    for (int wd = 0; wd < kDirectWords; ++wd)
      for (unsigned int m = s_plane[x][wd] & ch[wd]; m; m &= m - 1) {
        const int j = 32 * wd + __ffs(m) - 1;
        const float4 w = s_w[j];
        const bool own = s_cell[j].x == x;
        const int wb = __float_as_int(k == elec ? (own ? w.z : w.w) : (own ? w.x : w.y));
        s_list[at++] = make_int4(wb, wb, j * (NY * 2 * 16), j * (NZH * 8));
      }
    s_run[k][x] = (uint32_t)first | (uint32_t)(at - first) << 16;
  }
  __syncthreads();
  constexpr int BLOCKS = (Q + 31) / 32;
  const int work = s_nitems * BLOCKS;
  for (int b = blockIdx.x * NW + warp; b < work; b += gridDim.x * NW) {
    const int it = s_item[b / BLOCKS], cb = (b % BLOCKS) * 32 + lane;
    const int k = it & 15, q = (it >> 4) & 15;
    if (cb >= Q) continue;
    if (LOP && it >= 256) {
      for (int i = 0; i < 4; ++i) tiled_zero_chunk(a, r, k, q, cb + i * Q);
      continue;
    }
    const int p = cb / NZH, kz = cb - p * NZH;
    const unsigned char* fyb = reinterpret_cast<const unsigned char*>(Fy + p * 2);
    const unsigned char* fzb = reinterpret_cast<const unsigned char*>(Fz + kz);
    uint32_t hw[4][ROWS == kRowsBf16 ? 16 : 8];  // per column the rows' words (ROWS only)
    pair_t px[2], py[2];                         // the even plane's sums
#pragma unroll
    for (int d = 0; d < 8; ++d) {
      pair_t ax[2] = {0ull, 0ull}, ay[2] = {0ull, 0ull};
      const uint32_t run = s_run[k][8 * q + d];
      const int4* e = s_list + (run & 0xffff);
#pragma unroll 1
      for (int cnt = run >> 16; cnt > 0; --cnt, ++e) {
        const int4 en = *e;
        const float4 f0 = *reinterpret_cast<const float4*>(fyb + en.z), f1 = *reinterpret_cast<const float4*>(fyb + en.z + 16);
        const float2 fz = *reinterpret_cast<const float2*>(fzb + en.w);
        const pair_t w = pk(__int_as_float(en.x), __int_as_float(en.y));
        auto gx = [&](float x, float y) { return __fmaf_rn(x, fz.x, -__fmul_rn(y, fz.y)); };
        auto gy = [&](float x, float y) { return __fmaf_rn(y, fz.x, __fmul_rn(x, fz.y)); };
        ax[0] = p_fma(w, pk(gx(f0.x, f0.z), gx(f0.y, f0.w)), ax[0]);
        ay[0] = p_fma(w, pk(gy(f0.x, f0.z), gy(f0.y, f0.w)), ay[0]);
        ax[1] = p_fma(w, pk(gx(f1.x, f1.z), gx(f1.y, f1.w)), ax[1]);
        ay[1] = p_fma(w, pk(gy(f1.x, f1.z), gy(f1.y, f1.w)), ay[1]);
      }
      if constexpr (!LOP) {
        const int x = 8 * q + d;
        if (x >= rec->xlo[k] && x <= rec->xhi[k]) {
          float2* dst = a.A + (((size_t)r * K + k) * a.Lb + x) * NCOL + cb;
#pragma unroll
          for (int i = 0; i < 2; ++i) {
            const float2 vx = unpk(ax[i]), vy = unpk(ay[i]);
            dst[2 * i * Q] = make_float2(vx.x, vy.x);
            dst[(2 * i + 1) * Q] = make_float2(vx.y, vy.y);
          }
        }
      } else if (d % 2 == 0) {
#pragma unroll
        for (int i = 0; i < 2; ++i) {
          px[i] = ax[i];
          py[i] = ay[i];
        }
      } else {
        // planes d - 1 and d (zero outside the channel's planes by construction) into the rows' words
#pragma unroll
        for (int i = 0; i < 2; ++i) {
          const float2 ex = unpk(px[i]), ey = unpk(py[i]), ox = unpk(ax[i]), oy = unpk(ay[i]);
#pragma unroll
          for (int u = 0; u < 2; ++u) {
            uint32_t* w = hw[2 * i + u] + d / 2;
            const float re0 = u ? ex.y : ex.x, re1 = u ? ox.y : ox.x, im0 = u ? ey.y : ey.x, im1 = u ? oy.y : oy.x;
            if constexpr (ROWS == kRowsF16) {
              const __half2 pr = __floats2half2_rn(re0, re1), pi = __floats2half2_rn(im0, im1);
              w[0] = *reinterpret_cast<const uint32_t*>(&pr);
              w[4] = *reinterpret_cast<const uint32_t*>(&pi);
            } else {
              split_bf16x2(re0, re1, w[0], w[8]);
              split_bf16x2(im0, im1, w[4], w[12]);
            }
          }
        }
      }
    }
    if constexpr (LOP) {
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        uint4 rows[ROWS == kRowsBf16 ? 4 : 2];
#pragma unroll
        for (int u = 0; u < (ROWS == kRowsBf16 ? 4 : 2); ++u)
          rows[u] = make_uint4(hw[i][4 * u], hw[i][4 * u + 1], hw[i][4 * u + 2], hw[i][4 * u + 3]);
        plane_rows_write<N, ROWS>(a, r, k, q, cb + i * Q, rows);
      }
    }
  }
}

// ---------------------------------------------------------------------------------------
// Plane x of rotation r read from B in any of its layouts; at(f) is column f of the plane.
// Column-pair groups (cs = 1): float2 (f >> 1) 2G + (f & 1) past the plane's first pair; single-
// column groups (cs = 0): float2 f G past the plane's first column. The plain layout is G = 1.
// BL fixes the layout at compile time (the loads of a butterfly then share one base address):
// kBPlain, kBPairs2 (column pairs, G = 2), kBSingle4 (single columns, G = 4); kBAny reads the
// layout from WaveArgs.
constexpr int kBAny = 0, kBPlain = 1, kBPairs2 = 2, kBSingle4 = 3;
template <int BL>
struct BPlane {
  const float2* p;
  int cs, gs;
  __device__ __forceinline__ BPlane(const WaveArgs& a, int r, int x, int n, int ncol) {
    const int G = BL == kBPlain ? 1 : BL == kBPairs2 ? 2 : BL == kBSingle4 ? 4 : (a.bgroup > 1 ? a.bgroup : 1);
    cs = BL == kBSingle4 ? 0 : BL == kBAny ? (a.bcol ? 0 : 1) : 1;
    gs = G << cs;
    p = a.B + ((size_t)r * n + (x - x % G)) * ncol + ((x % G) << cs);
  }
  __device__ __forceinline__ float2 at(int f) const {
    if constexpr (BL == kBPlain) return p[f];
    else if constexpr (BL == kBPairs2) return p[(f >> 1) * 4 + (f & 1)];
    else if constexpr (BL == kBSingle4) return p[f * 4];
    else return p[(size_t)(f >> cs) * gs + (f & cs)];
  }
};
// the compile-time layout of a wave's B (kBAny for the others)
inline int b_layout(const WaveArgs& a) {
  if (a.bcol) return a.bgroup == 4 ? kBSingle4 : kBAny;
  return a.bgroup <= 1 ? kBPlain : a.bgroup == 2 ? kBPairs2 : kBAny;
}

// inverse (y,z) of one (rotation, x in window) plane + min / first argmin; TOP2: also the
// plane's second-smallest key, for the FP64 near-tie break (WaveArgs.keys2)
template <int N, bool TOP2, int BL>
__global__ void __launch_bounds__(256, (N <= 64 ? 8 : 2)) k_yz_inv_argmin(WaveArgs a) {
  constexpr int NZH = N / 2 + 1;
  constexpr int NCOL = N * NZH;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  float2* tw = reinterpret_cast<float2*>(smem_raw);
  float2* O = tw + N;
  // n <= 64: the packed rows P overwrite O once O has been read (N/2 x (N+1) <= N x (N/2+1)
  // entries), so a CTA holds one plane and the SM more CTAs; larger n keep P apart (the pack
  // would hold too many values in registers)
  constexpr bool ALIAS = N <= 64;
  float2* P = ALIAS ? O : O + N * NZH;
  static_assert((N / 2) * (N + 1) <= N * NZH, "packed rows fit the plane buffer");
  __shared__ unsigned long long s_best[8], s_best2[8];
  const int x = blockIdx.x, r = blockIdx.y;
  const RotRec* rec = a.rec + r;
  if (!rec->valid) return;
  const int Wx = rec->W[0], Wy = rec->W[1], Wz = rec->W[2];
  if (x >= Wx) return;
  const int tid = threadIdx.x, nthr = blockDim.x;
  for (int i = tid; i < N; i += nthr) tw[i] = a.tw[i];
  // plane x: NCOL / 2 column pairs, 16 B each, contiguous (plain layout) or every G-th of the
  // plane group (grouped layout, G planes per 16 B x column-pair block); or, single-column
  // groups, one float2 of every G
  const BPlane<BL> bp(a, r, x, N, NCOL);
  if constexpr (ALIAS) {
    // y: positions -> natural rows, the first (R1-point, twiddle-free) stage reading its rows
    // straight from B: item (column l, block b) takes positions b R1 + j of column l, plane
    // entry f = row * NZH + l, which is half f % 2 of column pair f / 2
    using PL = FFTPlan<N>;
    constexpr int R0 = PL::R0, R1 = PL::R1;
    static_assert(PL::NS == 2 && StageM<N, 2>::value == 1, "two-stage plan");
    for (int w = tid; w < NZH * R0; w += nthr) {
      const int b = w / NZH, l = w - b * NZH;
      float2 v[R1];
#pragma unroll
      for (int j = 0; j < R1; ++j) v[j] = bp.at((b * R1 + j) * NZH + l);
      Radix<R1, +1>::run(v);
      float2* p = O + l + b * R1 * NZH;
#pragma unroll
      for (int j = 0; j < R1; ++j) p[j * NZH] = v[j];
    }
    __syncthreads();
    fft_stage<N, R0, StageM<N, 1>::value, true>(O, NZH, 1, NZH, tw, tid, nthr);
    __syncthreads();
  } else {
    for (int i = tid; i < NCOL; i += nthr) O[i] = bp.at(i);
    __syncthreads();
    fft_lines<N, true>(O, NZH, 1, NZH, tw, tid, nthr);  // y: positions -> natural rows
  }
  const int npairs = (Wy + 1) / 2;
  const float inv = 1.0f / (float)((double)N * N * N);
  unsigned long long best = ~0ull, best2 = ~0ull;
  float thr = INFINITY;
  if constexpr (ALIAS) {
    // Rows (2p, 2p+1) as one complex line Z_p(k) = Y(2p, k) + i Y(2p+1, k) with the Hermitian
    // extension over z, inverse-transformed in two radix stages (N = R0 R1), one work item per
    // thread and stage (line p fastest). The pack is folded into the first stage's loads and
    // the window argmin into the last stage, so neither the packed input nor the energies take
    // a trip through shared memory.
    using PL = FFTPlan<N>;
    constexpr int R0 = PL::R0, R1 = PL::R1;
    static_assert(PL::NS == 2 && R0 * R1 == N && R1 % 2 == 0, "two-stage plan");
    static_assert((N / 2) * R0 <= 256 && (N / 2) * R1 <= 256, "one item per thread of 256");
    // item w -> (line w % npairs, block w / npairs); (w + 0.5) / npairs stays >= 1/64 away from
    // an integer for w < 256, npairs <= 32, far above the float rounding of the product
    const float rinv = npairs > 0 ? __frcp_rn((float)npairs) : 0.f;
    // stage 1 (R1-point, no twiddles): block b reads natural frequencies k = b + R0 j, which sit
    // at digit-reversed positions b R1 + j; k >= N/2 exactly when j >= R1/2
    const bool has1 = tid < npairs * R0;
    int l1 = 0, b1 = 0;
    float2 v1[R1];
    if (has1) {
      b1 = (int)(((float)tid + 0.5f) * rinv);
      l1 = tid - b1 * npairs;
      const float2* A = O + (2 * l1) * NZH;
      const float2* Bv = A + NZH;
#pragma unroll
      for (int j = 0; j < R1; ++j) {
        const int k = b1 + R0 * j;
        if (j < R1 / 2) {
          const float2 ak = A[k], bk = Bv[k];
          v1[j] = make_float2(ak.x - bk.y, ak.y + bk.x);
          if (j == 0 && b1 == 0) v1[j] = make_float2(ak.x, bk.x);  // k = 0
        } else {
          const int m = N - k;
          const float2 am = A[m], bm = Bv[m];
          v1[j] = make_float2(am.x + bm.y, -am.y + bm.x);
          if (j == R1 / 2 && b1 == 0) v1[j] = make_float2(am.x, bm.x);  // k = N/2
        }
      }
    }
    __syncthreads();  // every read of the y-transformed rows is done: the lines overwrite them
    if (has1) {
      Radix<R1, +1>::run(v1);
      float2* dst = P + l1 * (N + 1) + b1 * R1;
#pragma unroll
      for (int j = 0; j < R1; ++j) dst[j] = v1[j];
    }
    __syncthreads();
    // stage 2 (R0-point, twiddles tw[np k]): item np yields z = np + R1 j; line l holds row 2l in
    // its real part and row 2l + 1 in its imaginary part
    if (tid < npairs * R1) {
      const int np = (int)(((float)tid + 0.5f) * rinv);
      const int l = tid - np * npairs;
      const float2* src = P + l * (N + 1) + np;
      float2 v[R0];
#pragma unroll
      for (int j = 0; j < R0; ++j) v[j] = src[j * R1];
#pragma unroll
      for (int k = 1; k < R0; ++k) v[k] = c_mulc(v[k], tw[np * k]);
      Radix<R0, +1>::run(v);
      const int y0 = 2 * l;
      const bool row0 = y0 < Wy, row1 = y0 + 1 < Wy;
      const unsigned int lin0 = (unsigned int)((x * N + y0) * N + np);
#pragma unroll
      for (int j = 0; j < R0; ++j) {
        if (np + R1 * j < Wz) {
          if (row0) keep_min<TOP2>(v[j].x * inv, lin0 + (unsigned int)(R1 * j), best, best2, thr);
          if (row1) keep_min<TOP2>(v[j].y * inv, lin0 + (unsigned int)(N + R1 * j), best, best2, thr);
        }
      }
    }
  } else {
    // pack rows (2p, 2p+1) as one complex line with Hermitian extension over z (into its own
    // buffer), inverse-transform the lines, then take the window minimum from shared memory
    for (int i = tid; i < npairs * N; i += nthr) {
      const int p = i / N, k = i - p * N;
      const float2* A = O + (2 * p) * NZH;
      const float2* Bv = O + (2 * p + 1) * NZH;
      float2 z;
      if (k == 0 || k == N / 2) {
        z = make_float2(A[k].x, Bv[k].x);
      } else if (k < N / 2) {
        z = make_float2(A[k].x - Bv[k].y, A[k].y + Bv[k].x);
      } else {
        const int m = N - k;
        z = make_float2(A[m].x + Bv[m].y, -A[m].y + Bv[m].x);
      }
      P[p * (N + 1) + fft_pos<N>(k)] = z;
    }
    __syncthreads();
    if constexpr (FFTPlan<N>::NS == 2) {
      ifft_lines_slots<N, N / 2>(P, npairs, N + 1, 1, tw, tid, nthr);
    } else {
      fft_lines<N, true>(P, npairs, N + 1, 1, tw, tid, nthr);
    }
    // window rows by warp, columns by lane (the key carries the index: order does not matter)
    for (int y = tid >> 5; y < Wy; y += nthr >> 5) {
      const float2* row = P + (y >> 1) * (N + 1);
      for (int z = tid & 31; z < Wz; z += 32) {
        const float2 v = row[z];
        const float e = ((y & 1) ? v.y : v.x) * inv;
        keep_min<TOP2>(e, (unsigned int)((x * N + y) * N + z), best, best2, thr);
      }
    }
  }
  warp_keep_min<TOP2>(best, best2);
  if ((tid & 31) == 0) {
    s_best[tid >> 5] = best;
    if constexpr (TOP2) s_best2[tid >> 5] = best2;
  }
  __syncthreads();
  if (tid < 32) {
    const int nw = nthr >> 5;
    best = tid < nw ? s_best[tid] : ~0ull;
    if constexpr (TOP2) best2 = tid < nw ? s_best2[tid] : ~0ull;
    warp_keep_min<TOP2>(best, best2);
    if (tid == 0) {
      atomicMin(a.keys + r, best);
      if constexpr (TOP2) {
        a.keys2[((size_t)r * N + x) * 2] = best;
        a.keys2[((size_t)r * N + x) * 2 + 1] = best2;
      }
    }
  }
}

// Inverse (y,z) of one (rotation, x in window) plane + min / first argmin with warp-local line
// transforms, for n = 8 R1 (R1 = 4, 8, 12, 16). An octet of 8 lanes owns one line (a kz column
// for y, a packed row pair for z). The inverse runs the forward plan's two stages backwards:
// stage 1, radix R1 over the 8 contiguous blocks of R1 digit-reversed positions (lane t holds
// block t in registers); stage 2, radix 8 over the R1 groups {np + R1 j} with twiddles
// tw[np k] (lane t takes groups np = t, t + 8, ...), giving natural index np + R1 j. The
// exchange between the two stages goes through the line's own storage in the plane buffer
// (y: its kz column, rows at stride N/2+1; z: the two rows of its row pair, N + 2 slots), with
// __syncwarp only. Stage-1 output m of block t sits at line position t R1 + (m + t) mod R1 --
// block t rotated by t -- so the 8 lanes' stores of one m, and the 8 lanes' loads of one block
// in stage 2, fall in 8 different banks (odd row stride). In the y pass stage 2 gathers both
// of its groups before any lane writes the natural outputs back into the column. Block-wide
// barriers: after the twiddle load, between the y and z passes (the y output is the z input),
// and in the final reduction. Shared memory is the twiddles and the plane only (68 KB at
// 128^3), so three CTAs of 288 threads (72 registers) fit an SM. Same radix stages, twiddles
// and packing as k_yz_inv_argmin.
// 288 threads = 36 octets: the 33 kz columns (and at most 32 row pairs) of a 64^3 plane in one
// round each, 49 / 65 columns at 96^3 / 128^3 in two
constexpr int kOctWarps = 9;
constexpr int kOctets = 4 * kOctWarps;

template <int N>
constexpr size_t octet_smem() {
  return sizeof(float2) * (N + (size_t)N * (N / 2 + 1));
}

template <int N, bool TOP2, int BL>
__global__ void __launch_bounds__(32 * kOctWarps, 3) k_yz_octet(WaveArgs a) {
  constexpr int NZH = N / 2 + 1, NCOL = N * NZH;
  constexpr int R1 = N / 8;           // stage-1 radix; stage 2 is radix 8
  constexpr int NG = (R1 + 7) / 8;    // stage-2 groups per lane
  static_assert(N % 8 == 0 && (R1 == 4 || R1 == 8 || R1 == 12 || R1 == 16), "n = 8 R1");
  static_assert(NZH % 2 == 1, "odd row stride");
  extern __shared__ __align__(16) unsigned char smem_raw[];
  float2* s_tw = reinterpret_cast<float2*>(smem_raw);
  float2* s_y = s_tw + N;  // y-transformed rows Y[y][kz]
  __shared__ unsigned long long s_best[kOctWarps], s_best2[kOctWarps];
  const int x = blockIdx.x, r = blockIdx.y;
  const RotRec* rec = a.rec + r;
  if (!rec->valid) return;
  const int Wx = rec->W[0], Wy = rec->W[1], Wz = rec->W[2];
  if (x >= Wx) return;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int o = lane >> 3, t = lane & 7, g = warp * 4 + o;
  for (int i = tid; i < N; i += 32 * kOctWarps) s_tw[i] = a.tw[i];
  const BPlane<BL> bp(a, r, x, N, NCOL);
  __syncthreads();
  // line position of stage-1 output m of block blk
  auto xpos = [](int blk, int m) { return blk * R1 + (m + blk) % R1; };
  // y: columns l = g, g + 36, ...; a warp stops when none of its octets has a column left
  constexpr int YR = (NZH + kOctets - 1) / kOctets;
#pragma unroll 1
  for (int it = 0; it < YR; ++it) {
    if (warp * 4 + kOctets * it >= NZH) break;  // warp-uniform
    const int l = g + kOctets * it;
    const bool act = l < NZH;
    float2* col = s_y + (act ? l : 0);
    float2 v[R1];
#pragma unroll
    for (int j = 0; j < R1; ++j) v[j] = act ? bp.at((t * R1 + j) * NZH + l) : make_float2(0.f, 0.f);
    Radix<R1, +1>::run(v);
    if (act) {
#pragma unroll
      for (int j = 0; j < R1; ++j) col[xpos(t, j) * NZH] = v[j];
    }
    __syncwarp();
    float2 u[NG][8];
#pragma unroll
    for (int q = 0; q < NG; ++q) {
      const int np = t + 8 * q;
#pragma unroll
      for (int j = 0; j < 8; ++j) u[q][j] = (act && np < R1) ? col[xpos(j, np) * NZH] : make_float2(0.f, 0.f);
    }
    __syncwarp();  // every group of the line gathered before any natural output is written
#pragma unroll
    for (int q = 0; q < NG; ++q) {
      const int np = t + 8 * q;
      if (act && np < R1) {
#pragma unroll
        for (int k = 1; k < 8; ++k) u[q][k] = c_mulc(u[q][k], s_tw[np * k]);
        Radix<8, +1>::run(u[q]);
#pragma unroll
        for (int j = 0; j < 8; ++j) col[(np + R1 * j) * NZH] = u[q][j];
      }
    }
  }
  __syncthreads();
  // z: rows (2p, 2p + 1) packed as one complex line, Hermitian extension over z
  const int npairs = (Wy + 1) / 2;
  const float inv = 1.0f / (float)((double)N * N * N);
  unsigned long long best = ~0ull, best2 = ~0ull;
  float thr = INFINITY;
  constexpr int ZR = (N / 2 + kOctets - 1) / kOctets;
#pragma unroll 1
  for (int it = 0; it < ZR; ++it) {
    if (warp * 4 + kOctets * it >= npairs) break;  // warp-uniform
    const int p = g + kOctets * it;
    const bool act = p < npairs;
    float2* rows = s_y + (size_t)(2 * (act ? p : 0)) * NZH;  // rows 2p, 2p + 1: N + 2 slots
    const float2* A = rows;
    const float2* Bv = rows + NZH;
    float2 v[R1];
#pragma unroll
    for (int j = 0; j < R1; ++j) {
      const int k = t + 8 * j;  // natural frequency at digit-reversed position t R1 + j
      if (!act) {
        v[j] = make_float2(0.f, 0.f);
      } else if (j < R1 / 2) {
        const float2 ak = A[k], bk = Bv[k];
        v[j] = make_float2(ak.x - bk.y, ak.y + bk.x);
        if (j == 0 && t == 0) v[j] = make_float2(ak.x, bk.x);  // k = 0
      } else {
        const int m = N - k;
        const float2 am = A[m], bm = Bv[m];
        v[j] = make_float2(am.x + bm.y, -am.y + bm.x);
        if (j == R1 / 2 && t == 0) v[j] = make_float2(am.x, bm.x);  // k = N/2
      }
    }
    __syncwarp();  // the octet has read its rows: their slots become the exchange
    Radix<R1, +1>::run(v);
    if (act) {
#pragma unroll
      for (int j = 0; j < R1; ++j) rows[xpos(t, j)] = v[j];
    }
    __syncwarp();
    const int y0 = 2 * p;
    const bool row0 = act && y0 < Wy, row1 = act && y0 + 1 < Wy;
#pragma unroll
    for (int q = 0; q < NG; ++q) {
      const int np = t + 8 * q;
      if (act && np < R1) {
        float2 u[8];
#pragma unroll
        for (int j = 0; j < 8; ++j) u[j] = rows[xpos(j, np)];
#pragma unroll
        for (int k = 1; k < 8; ++k) u[k] = c_mulc(u[k], s_tw[np * k]);
        Radix<8, +1>::run(u);
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          const int z = np + R1 * j;
          if (z < Wz) {
            const unsigned int lin0 = (unsigned int)((x * N + y0) * N + z);
            if (row0) keep_min<TOP2>(u[j].x * inv, lin0, best, best2, thr);
            if (row1) keep_min<TOP2>(u[j].y * inv, lin0 + N, best, best2, thr);
          }
        }
      }
    }
  }
  warp_keep_min<TOP2>(best, best2);
  if (lane == 0) {
    s_best[warp] = best;
    if constexpr (TOP2) s_best2[warp] = best2;
  }
  __syncthreads();
  if (warp == 0) {
    best = lane < kOctWarps ? s_best[lane] : ~0ull;
    if constexpr (TOP2) best2 = lane < kOctWarps ? s_best2[lane] : ~0ull;
    warp_keep_min<TOP2>(best, best2);
    if (lane == 0) {
      atomicMin(a.keys + r, best);
      if constexpr (TOP2) {
        a.keys2[((size_t)r * N + x) * 2] = best;
        a.keys2[((size_t)r * N + x) * 2 + 1] = best2;
      }
    }
  }
}

// FP64 energies of rotation r at P translations (linear indices lin[]): the direct trilinear
// grid-energy sum over its rotated atoms (k_prep's rot_xyz and min corner), cells and ratios in
// FillLigandGrid's arithmetic, accumulated in double across the warp's lanes (atoms). A few rotations
// per warp at most, so it is a chain of memory latencies: an atom's 16 P grid values are loaded
// before the first is used, and a tie's two translations go together (64^3, 61 rotations: tie break 15 ->
// 12 us with the caches cold).
template <int P>
__device__ void pose_energies_fp64(const WaveArgs& a, const float* grids, int r, const unsigned int* lin,
                                   int lane, double* e) {
  const RotRec* rec = a.rec + r;
  const AtomParam* prm = a.params + rec->param_off;
  const int n = a.n, K = a.K;
  const size_t Ng = (size_t)n * n * n;
  const float h = a.spacing;
#pragma unroll
  for (int q = 0; q < P; ++q) e[q] = 0.0;
  for (int i = lane; i < rec->nA; i += 32) {
    const float4 p4 = a.rot_xyz[(size_t)r * a.max_atoms + i];
    const AtomParam ap = prm[i];
    const float p[3] = {p4.x, p4.y, p4.z};
    const bool vdw = ap.slot >= 0 && ap.slot < K - 1;
    int ci[3];
#pragma unroll
    for (int d = 0; d < 3; ++d) ci[d] = cell_of(p[d], rec->mn[d], h);
    float gv[P][8], ge[P][8];
    bool in[P][8];
#pragma unroll
    for (int q = 0; q < P; ++q) {
      const int x = ci[0] + (int)(lin[q] / (n * n)), y = ci[1] + (int)((lin[q] / n) % n), z = ci[2] + (int)(lin[q] % n);
#pragma unroll
      for (int c = 0; c < 8; ++c) {
        const int gx = x + ((c >> 2) & 1), gy = y + ((c >> 1) & 1), gz = z + (c & 1);
        in[q][c] = gx < n && gy < n && gz < n;
        const size_t g = ((size_t)gx * n + gy) * n + gz;
        gv[q][c] = in[q][c] && vdw ? grids[(size_t)ap.slot * Ng + g] : 0.f;
        ge[q][c] = in[q][c] ? grids[(size_t)(K - 1) * Ng + g] : 0.f;
      }
    }
    double rr[3];
#pragma unroll
    for (int d = 0; d < 3; ++d) rr[d] = ratio_of(p[d], rec->mn[d], h, ci[d]);
#pragma unroll
    for (int c = 0; c < 8; ++c) {
      const int dx = (c >> 2) & 1, dy = (c >> 1) & 1, dz = c & 1;
      const double w = (dx ? rr[0] : 1.0 - rr[0]) * (dy ? rr[1] : 1.0 - rr[1]) * (dz ? rr[2] : 1.0 - rr[2]);
#pragma unroll
      for (int q = 0; q < P; ++q) {
        if (!in[q][c]) continue;
        if (vdw) e[q] += (double)ap.w_vdw * w * (double)gv[q][c];
        e[q] += (double)ap.charge * w * (double)ge[q][c];
      }
    }
  }
#pragma unroll
  for (int q = 0; q < P; ++q)
    for (int o = 16; o > 0; o >>= 1) e[q] += __shfl_xor_sync(0xffffffffu, e[q], o);
}

// FP64 near-tie break of the argmin (precision forms), warp per rotation: the two smallest keys
// over the rotation's key pairs (one per window plane, or WaveArgs.key_slots); when the second energy lies within tol * max(|E1|, 1) of
// the first, both translations are re-scored in FP64 (pose_energies_fp64) and the lower one is
// kept -- the smaller linear index (x-major first) on an exact FP64 tie. The reported energy
// stays the search's own value at the kept translation. work[4] counts re-scored rotations,
// work[5] the ones whose translation changed.
__global__ void __launch_bounds__(128) k_tiebreak(WaveArgs a, const float* __restrict__ grids, float tol) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int r = blockIdx.x * 4 + warp;
  if (r >= a.nrot) return;
  const RotRec* rec = a.rec + r;
  if (!rec->valid) return;
  const int n = a.n;
  unsigned long long b1 = ~0ull, b2 = ~0ull;
  const int slots = a.key_slots > 0 ? a.key_slots : rec->W[0];
  for (int x = lane; x < slots; x += 32)
    top2_merge(a.keys2[((size_t)r * n + x) * 2], a.keys2[((size_t)r * n + x) * 2 + 1], b1, b2);
  for (int o = 16; o > 0; o >>= 1) {
    const unsigned long long o1 = __shfl_xor_sync(0xffffffffu, b1, o);
    const unsigned long long o2 = __shfl_xor_sync(0xffffffffu, b2, o);
    top2_merge(o1, o2, b1, b2);
  }
  if (b1 == ~0ull || b2 == ~0ull) return;
  const float e1 = key_to_float((unsigned int)(b1 >> 32)), e2 = key_to_float((unsigned int)(b2 >> 32));
  if (!(e2 - e1 <= tol * fmaxf(fabsf(e1), 1.f))) return;
  const unsigned int l1 = (unsigned int)b1, l2 = (unsigned int)b2;
  const unsigned int lin[2] = {l1, l2};
  double f[2];
  pose_energies_fp64<2>(a, grids, r, lin, lane, f);
  const double f1 = f[0], f2 = f[1];
  if (lane == 0) {
    const bool flip = f2 < f1 || (f2 == f1 && l2 < l1);
    if (flip) a.keys[r] = b2;
    if (a.work) {
      atomicAdd(a.work + 4, 1ull);
      if (flip) atomicAdd(a.work + 5, 1ull);
    }
  }
}

// FP64 re-score of the k lowest-energy poses of a wave (precision forms), one CTA of k_finalize: the k
// smallest final keys (energy, then the rotation's place in the wave) by k rounds of a block
// minimum over each thread's own sorted candidates, then one warp per pose for its FP64 direct
// grid-energy sum at its kept translation. out[j]: the rotation's output slot, the search's
// energy, its translation's linear index and the FP64 energy; unused slots get out = -1.
// L: the candidates a thread keeps (k of them are enough). The loads of four rotations are issued
// together: the other blocks are done long before this one.
template <int L>
__device__ void topk_rescore(const WaveArgs& a, const float* __restrict__ grids, int k,
                             TopPose* __restrict__ out) {
  __shared__ unsigned long long s_min[8];
  __shared__ unsigned long long s_pick[L];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  // per thread: its L smallest (energy bits, rotation) keys, ascending
  unsigned long long cand[L];
#pragma unroll
  for (int j = 0; j < L; ++j) cand[j] = ~0ull;
  for (int r0 = tid; r0 < a.nrot; r0 += 4 * blockDim.x) {
    unsigned long long key[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const int r = r0 + u * (int)blockDim.x;
      key[u] = r < a.nrot && a.rec[r].valid ? a.keys[r] : ~0ull;
    }
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      if (key[u] == ~0ull) continue;
      unsigned long long c = (key[u] & 0xffffffff00000000ull) | (unsigned int)(r0 + u * (int)blockDim.x);
      if (c >= cand[L - 1]) continue;
#pragma unroll
      for (int j = 0; j < L; ++j) {
        const unsigned long long lo = c < cand[j] ? c : cand[j];
        c = c < cand[j] ? cand[j] : c;
        cand[j] = lo;
      }
    }
  }
  int head = 0;
  for (int j = 0; j < k; ++j) {
    unsigned long long m = head < L ? cand[0] : ~0ull;
    for (int o = 16; o > 0; o >>= 1) {
      const unsigned long long v = __shfl_xor_sync(0xffffffffu, m, o);
      m = v < m ? v : m;
    }
    if (lane == 0) s_min[warp] = m;
    __syncthreads();
    unsigned long long g = s_min[0];
    for (int w = 1; w < 8; ++w) g = s_min[w] < g ? s_min[w] : g;
    if (tid == 0) s_pick[j] = g;
    // the owner pops its head (keys are unique: one rotation each)
    if (g != ~0ull && cand[0] == g) {
#pragma unroll
      for (int q = 0; q + 1 < L; ++q) cand[q] = cand[q + 1];
      cand[L - 1] = ~0ull;
      ++head;
    }
    __syncthreads();
  }
  for (int j = warp; j < k; j += 8) {
    const unsigned long long g = s_pick[j];
    TopPose tp;
    tp.out = -1;
    tp.lin = -1;
    tp.e = INFINITY;
    tp.e64 = 0.0;
    if (g != ~0ull) {
      const int r = (int)(unsigned int)g;
      const unsigned int lin = (unsigned int)a.keys[r];
      double e64;
      pose_energies_fp64<1>(a, grids, r, &lin, lane, &e64);
      tp.out = a.rots[r].out;
      tp.lin = (int)lin;
      tp.e = key_to_float((unsigned int)(a.keys[r] >> 32));
      tp.e64 = e64;
    }
    if (lane == 0) out[j] = tp;
  }
}

// Results of the final keys. TOP: block 0 re-scores the k lowest-energy poses (it reads the same keys, so
// beside the other blocks and not in a launch before them: 64^3, 61 rotations, 14.5 us and a launch of
// 8 -> 14 together; the whole search 298 -> 278)
template <bool TOP>
__global__ void __launch_bounds__(256) k_finalize(WaveArgs a, const float* __restrict__ grids, int k,
                                                  TopPose* __restrict__ top) {
  if (TOP && blockIdx.x == 0) {
    if (k <= 8) topk_rescore<8>(a, grids, k, top);
    else topk_rescore<kTopMax>(a, grids, k, top);
    return;
  }
  const int r = (blockIdx.x - (TOP ? 1 : 0)) * blockDim.x + threadIdx.x;
  if (r >= a.nrot) return;
  const int out = a.rots[r].out;
  const RotRec* rec = a.rec + r;
  if (rec->err == 1) atomicAdd(a.err_count, 1);  // err 2 is reported through range_err
  if (rec->valid) {
    unsigned long long planes = 0;
    for (int k = 0; k < a.K; ++k)
      if (rec->xlo[k] <= rec->xhi[k]) planes += (unsigned long long)(rec->xhi[k] - rec->xlo[k] + 1);
    atomicAdd(a.work, planes);
    atomicAdd(a.work + 1, (unsigned long long)rec->W[0]);
  }
  const unsigned long long key = a.keys[r];
  if (!rec->valid || key == ~0ull) {
    a.minE[out] = INFINITY;
    a.idx[out * 3 + 0] = a.idx[out * 3 + 1] = a.idx[out * 3 + 2] = -1;
    return;
  }
  const unsigned int lin = (unsigned int)(key & 0xffffffffu);
  const int n = a.n;
  a.minE[out] = key_to_float((unsigned int)(key >> 32));
  a.idx[out * 3 + 0] = lin / (n * n);
  a.idx[out * 3 + 1] = (lin / n) % n;
  a.idx[out * 3 + 2] = lin % n;
}

__global__ void k_finalize_server(WaveArgs a, float* ebase, int* ibase) {
  const int r = blockIdx.x * blockDim.x + threadIdx.x;
  if (r >= a.nrot) return;
  const RotDesc rd = a.rots[r];
  const RotRec* rec = a.rec + r;
  const unsigned long long key = a.keys[r];
  int* idx = ibase + rd.pad0;
  if (rec->err) {
    // a rotation that could not be searched: NaN energy and index -2 (box overflow) or -3
    // (FP16 range), which the server reads back to fail exactly the requests that hold one
    if (rec->err == 1) atomicAdd(a.err_count, 1);
    else atomicOr(a.range_err, 1);
    ebase[rd.out] = __int_as_float(0x7fc00000);
    idx[0] = idx[1] = idx[2] = rec->err == 1 ? -2 : -3;
    return;
  }
  if (!rec->valid || key == ~0ull) {
    ebase[rd.out] = INFINITY;
    idx[0] = idx[1] = idx[2] = -1;
    return;
  }
  const unsigned int lin = (unsigned int)(key & 0xffffffffu);
  const int n = a.n;
  ebase[rd.out] = key_to_float((unsigned int)(key >> 32));
  idx[0] = lin / (n * n);
  idx[1] = (lin / n) % n;
  idx[2] = lin % n;
}

// ---------------------------------------------------------------------------------------
// receptor spectra: dense (y,z) forward of every plane, then x forward per column tile
template <int N>
__global__ void __launch_bounds__(256) k_receptor_yz(const float* grids, float2* out,
                                                      const float2* twg) {
  constexpr int NZH = N / 2 + 1;
  constexpr int NCOL = N * NZH;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  float2* tw = reinterpret_cast<float2*>(smem_raw);
  float2* O = tw + N;
  float2* P = O + N * NZH;
  const int x = blockIdx.x, k = blockIdx.y;
  const int tid = threadIdx.x, nthr = blockDim.x;
  for (int i = tid; i < N; i += nthr) tw[i] = twg[i];
  const float* g = grids + ((size_t)k * N + x) * N * N;
  for (int i = tid; i < N * N; i += nthr) {
    const int y = i / N, z = i - y * N;
    reinterpret_cast<float*>(P)[((y >> 1) * (N + 1) + z) * 2 + (y & 1)] = g[i];
  }
  __syncthreads();
  plane_forward<N>(P, O, N / 2, tw);
  float2* dst = out + ((size_t)k * N + x) * NCOL;
  for (int i = tid; i < NCOL; i += nthr) dst[i] = O[i];
}

template <int N>
__global__ void __launch_bounds__(256) k_receptor_x(const float2* in, float2* phat, int K,
                                                     int ct, const float2* twg) {
  constexpr int NZH = N / 2 + 1;
  constexpr int NCOL = N * NZH;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  float2* tw = reinterpret_cast<float2*>(smem_raw);
  float2* Wb = tw + N;
  const int c0 = blockIdx.x * ct;
  const int k = blockIdx.y;
  const int tid = threadIdx.x, nthr = blockDim.x;
  for (int i = tid; i < N; i += nthr) tw[i] = twg[i];
  for (int i = tid; i < N * ct; i += nthr) {
    const int c = i % ct, x = i / ct;
    Wb[i] = (c0 + c < NCOL) ? in[((size_t)k * N + x) * NCOL + c0 + c] : make_float2(0.f, 0.f);
  }
  __syncthreads();
  fft_lines<N, false>(Wb, ct, 1, ct, tw, tid, nthr);
  for (int i = tid; i < N * ct; i += nthr) {
    const int c = i % ct, xp = i / ct;
    if (c0 + c < NCOL) phat[((size_t)xp * K + k) * NCOL + c0 + c] = Wb[i];
  }
}

template <int N>
constexpr size_t plane_smem() {
  return sizeof(float2) * (N + N * (N / 2 + 1) + (N / 2) * (N + 1));
}

template <int N>
cudaError_t launch_spread_yz_t(const WaveArgs& a, cudaStream_t s) {
  const int cap = a.atom_cap > 0 ? a.atom_cap : a.max_atoms;
  if (a.kyof && cap <= kDirectMaxAtoms) {
    auto launch = [&](auto kern, auto shape) {
      // room for the largest ligand whatever this one's atoms: the attribute is the process's, and another
      // thread's smaller ligand, set between this call and the launch, would refuse it
      const cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                                 (int)shape.smem(kDirectMaxAtoms));
      if (e != cudaSuccess) return e;
      // parts of a rotation's items: enough CTAs for small waves (each part repeats the tables)
      const int parts = std::max(1, std::min(a.K, (148 * 6 + a.nrot - 1) / a.nrot));
      kern<<<dim3(parts, a.nrot), shape.T, shape.smem(cap), s>>>(a, a.kyof, cap);
      return cudaGetLastError();
    };
    if (!a.lop) return launch(k_spread_yz_direct<N, kRowsNone>, DirectShape<N, kRowsNone>{});
    if (a.f16) return launch(k_spread_yz_direct<N, kRowsF16>, DirectShape<N, kRowsF16>{});
    return launch(k_spread_yz_direct<N, kRowsBf16>, DirectShape<N, kRowsBf16>{});
  }
  if (a.lop) return cudaErrorInvalidValue;  // the FFT plane path writes A only
  const size_t sm = plane_smem<N>();
  cudaError_t e = cudaFuncSetAttribute(k_spread_yz<N>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm);
  if (e != cudaSuccess) return e;
  dim3 grid(a.Lb, a.K, a.nrot);
  k_spread_yz<N><<<grid, 256, sm, s>>>(a);
  return cudaGetLastError();
}

template <int N>
cudaError_t launch_yz_inv_t(const WaveArgs& a, cudaStream_t s) {
  // the single-plane kernels: plain and column-pair B (x passes on request), and on request. Octets at
  // n >= 96 (measured 2.1x faster than block stages at 128^3, 1.05x at 96^3); block stages at n <= 64
  // (the packed rows alias the plane there, 8 CTAs per SM: 1.6x faster than the octets at 64^3);
  // yz_block_stages: 1 forces block stages, 2 forces octets
  const bool octet = a.yz_block_stages == 2 || (a.yz_block_stages == 0 && N >= 96);
  // the B layout as a template argument (kBAny reads it at run time)
  const int bl = b_layout(a);
#define CDK_YZ_PICK(KERN)                                                                     \
  (bl == kBPlain    ? (a.keys2 ? KERN<N, true, kBPlain> : KERN<N, false, kBPlain>)           \
   : bl == kBPairs2 ? (a.keys2 ? KERN<N, true, kBPairs2> : KERN<N, false, kBPairs2>)         \
   : bl == kBSingle4 ? (a.keys2 ? KERN<N, true, kBSingle4> : KERN<N, false, kBSingle4>)      \
                     : (a.keys2 ? KERN<N, true, kBAny> : KERN<N, false, kBAny>))
  if (octet) {
    constexpr size_t sm = octet_smem<N>();
    auto kern = CDK_YZ_PICK(k_yz_octet);
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm);
    if (e != cudaSuccess) return e;
    dim3 grid(N, a.nrot);
    kern<<<grid, 32 * kOctWarps, sm, s>>>(a);
    return cudaGetLastError();
  }
  // twiddles + one plane (n <= 64: the packed rows alias it) [+ the packed rows]
  const size_t sm = sizeof(float2) * (N + N * (N / 2 + 1) + (N <= 64 ? 0 : (N / 2) * (N + 1)));
  auto kern = CDK_YZ_PICK(k_yz_inv_argmin);
#undef CDK_YZ_PICK
  cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm);
  if (e != cudaSuccess) return e;
  dim3 grid(N, a.nrot);
  kern<<<grid, 256, sm, s>>>(a);
  return cudaGetLastError();
}

template <int N>
cudaError_t launch_receptor_t(int K, const float* grids, float2* scratch, float2* phat,
                              const float2* tw, int ct, cudaStream_t s) {
  const size_t sm = plane_smem<N>();
  cudaError_t e = cudaFuncSetAttribute(k_receptor_yz<N>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm);
  if (e != cudaSuccess) return e;
  k_receptor_yz<N><<<dim3(N, K), 256, sm, s>>>(grids, scratch, tw);
  if ((e = cudaGetLastError()) != cudaSuccess) return e;
  constexpr int NCOL = N * (N / 2 + 1);
  const size_t sm2 = sizeof(float2) * (N + (size_t)N * ct);
  e = cudaFuncSetAttribute(k_receptor_x<N>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm2);
  if (e != cudaSuccess) return e;
  k_receptor_x<N><<<dim3((NCOL + ct - 1) / ct, K), 256, sm2, s>>>(scratch, phat, K, ct, tw);
  return cudaGetLastError();
}

// ---------------------------------------------------------------------------------------
// Rotation grouping for the tensor-core x pass. A tile of 128 rotations loads and multiplies,
// per channel, the union of the 8-plane chunks its rotations touch. Nearly every rotation
// starts at chunk 0; what varies is whether a channel's atoms reach the box's last chunk. A
// stable counting sort of the rotation list on one bit per channel (folded into kGroupBits)
// puts rotations with the same pattern side by side, so tiles skip more chunks. Results do
// not depend on the order: a chunk a rotation does not touch adds exact zeros to its sums, and
// every output goes to its rotation's RotDesc::out.
constexpr int kGroupBits = 10;
constexpr int kGroupBuckets = 1 << kGroupBits;
constexpr int kGroupSeg = 1024;  // rotations per histogram / scatter CTA

// warp per rotation: the rotated x coordinates and their minimum exactly as k_prep computes
// them, then the channels whose atoms reach chunk jc - 1
__global__ void __launch_bounds__(128) k_group_key(const RotDesc* __restrict__ rots,
                                                   const ConfDesc* __restrict__ confs,
                                                   const float* __restrict__ coords,
                                                   const AtomParam* __restrict__ params, long nrot,
                                                   int max_atoms, int K, float h, int jc,
                                                   unsigned short* __restrict__ key) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const long r = (long)blockIdx.x * 4 + warp;
  if (r >= nrot) return;
  const RotDesc rd = rots[r];
  const ConfDesc cd = confs[rd.conf];
  const int nA = min(cd.n_atoms, max_atoms);
  const float* xyz = coords + (size_t)cd.coord_off * 3;
  const AtomParam* prm = params + cd.param_off;
  float mn = INFINITY;
  for (int i = lane; i < nA; i += 32) {
    float p[3];
    rotate_rn(rd.q, xyz[i * 3 + 0], xyz[i * 3 + 1], xyz[i * 3 + 2], p);
    mn = fminf(mn, p[0]);
  }
  for (int o = 16; o > 0; o >>= 1) mn = fminf(mn, __shfl_xor_sync(0xffffffffu, mn, o));
  const int elec = K - 1;
  unsigned int bits = 0;
  for (int i = lane; i < nA; i += 32) {
    float p[3];
    rotate_rn(rd.q, xyz[i * 3 + 0], xyz[i * 3 + 1], xyz[i * 3 + 2], p);
    if (min((cell_of(p[0], mn, h) + 1) >> 3, jc - 1) == jc - 1) {
      const int sl = prm[i].slot;
      if (sl >= 0 && sl < elec) bits |= 1u << (sl % kGroupBits);
      bits |= 1u << (elec % kGroupBits);
    }
  }
  bits = __reduce_or_sync(0xffffffffu, bits);
  if (lane == 0) key[r] = (unsigned short)bits;
}

// per segment of kGroupSeg rotations, the count of each key: counts[key * nseg + segment]
__global__ void __launch_bounds__(kGroupSeg) k_group_hist(const unsigned short* __restrict__ key,
                                                          long nrot, int nseg, int* __restrict__ counts) {
  __shared__ int hcount[kGroupBuckets];
  for (int b = threadIdx.x; b < kGroupBuckets; b += blockDim.x) hcount[b] = 0;
  __syncthreads();
  const long r = (long)blockIdx.x * kGroupSeg + threadIdx.x;
  if (r < nrot) atomicAdd(&hcount[key[r]], 1);
  __syncthreads();
  for (int b = threadIdx.x; b < kGroupBuckets; b += blockDim.x)
    counts[(size_t)b * nseg + blockIdx.x] = hcount[b];
}

// exclusive scan of counts in place (key-major, so a key's segments follow one another)
__global__ void __launch_bounds__(1024) k_group_scan(int* __restrict__ counts, long total) {
  __shared__ long part[1024];
  const int tid = threadIdx.x, T = blockDim.x;
  const long per = (total + T - 1) / T;
  const long lo = min(total, (long)tid * per), hi = min(total, lo + per);
  long sum = 0;
  for (long i = lo; i < hi; ++i) sum += counts[i];
  part[tid] = sum;
  __syncthreads();
  for (int off = 1; off < T; off <<= 1) {
    const long v = tid >= off ? part[tid - off] : 0;
    __syncthreads();
    part[tid] += v;
    __syncthreads();
  }
  long run = part[tid] - sum;
  for (long i = lo; i < hi; ++i) {
    const int c = counts[i];
    counts[i] = (int)run;
    run += c;
  }
}

// stable scatter: the warps of a segment place their rotations in warp order, lanes with the
// same key by lane order
__global__ void __launch_bounds__(kGroupSeg) k_group_scatter(const RotDesc* __restrict__ rots,
                                                             const unsigned short* __restrict__ key,
                                                             long nrot, int nseg,
                                                             const int* __restrict__ counts,
                                                             RotDesc* __restrict__ out) {
  __shared__ int base[kGroupBuckets];
  for (int b = threadIdx.x; b < kGroupBuckets; b += blockDim.x) base[b] = counts[(size_t)b * nseg + blockIdx.x];
  const long r = (long)blockIdx.x * kGroupSeg + threadIdx.x;
  const bool live = r < nrot;
  const unsigned int kk = live ? key[r] : 0xffffffffu;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const unsigned int same = __match_any_sync(0xffffffffu, kk);
  const int rank = __popc(same & ((1u << lane) - 1));
  __syncthreads();
  for (int w = 0; w < (int)(blockDim.x >> 5); ++w) {
    if (warp == w) {
      const int b0 = live ? base[kk] : 0;
      __syncwarp();
      if (live) {
        out[b0 + rank] = rots[r];
        if (rank == 0) base[kk] = b0 + __popc(same);
      }
    }
    __syncthreads();
  }
}

}  // namespace

int fft_position(int n, int k) {
  switch (n) {
    case 32: return fft_pos<32>(k);
    case 64: return fft_pos<64>(k);
    case 96: return fft_pos<96>(k);
    case 128: return fft_pos<128>(k);
    default: return k;
  }
}

#define CDK_DISPATCH_N(n, fn, ...)                 \
  switch (n) {                                     \
    case 32: return fn<32>(__VA_ARGS__);           \
    case 64: return fn<64>(__VA_ARGS__);           \
    case 96: return fn<96>(__VA_ARGS__);           \
    case 128: return fn<128>(__VA_ARGS__);         \
    default: return cudaErrorInvalidValue;         \
  }

size_t group_rotations_bytes(long nrot) {
  const long nseg = (nrot + kGroupSeg - 1) / kGroupSeg;
  return ((size_t)nrot * sizeof(RotDesc) + 255) / 256 * 256 + ((size_t)nrot * 2 + 255) / 256 * 256 +
         (size_t)kGroupBuckets * nseg * sizeof(int);
}

cudaError_t launch_group_rotations(const RotDesc* rots, const ConfDesc* confs, const float* coords,
                                   const AtomParam* params, long nrot, int max_atoms, int K, float h,
                                   int jc, void* scratch, RotDesc** sorted, cudaStream_t s) {
  if (nrot <= 0 || jc < 1 || K > KMAX) return cudaErrorInvalidValue;
  const long nseg = (nrot + kGroupSeg - 1) / kGroupSeg;
  char* p = static_cast<char*>(scratch);
  RotDesc* out = reinterpret_cast<RotDesc*>(p);
  p += ((size_t)nrot * sizeof(RotDesc) + 255) / 256 * 256;
  unsigned short* key = reinterpret_cast<unsigned short*>(p);
  p += ((size_t)nrot * 2 + 255) / 256 * 256;
  int* counts = reinterpret_cast<int*>(p);
  k_group_key<<<(unsigned)((nrot + 3) / 4), 128, 0, s>>>(rots, confs, coords, params, nrot, max_atoms, K, h, jc, key);
  k_group_hist<<<(unsigned)nseg, kGroupSeg, 0, s>>>(key, nrot, (int)nseg, counts);
  k_group_scan<<<1, 1024, 0, s>>>(counts, (long)kGroupBuckets * nseg);
  k_group_scatter<<<(unsigned)nseg, kGroupSeg, 0, s>>>(rots, key, nrot, (int)nseg, counts, out);
  *sorted = out;
  return cudaGetLastError();
}

cudaError_t launch_prep(const WaveArgs& a, cudaStream_t s) {
  k_prep<<<(a.nrot + 3) / 4, 128, 0, s>>>(a);
  return cudaGetLastError();
}
cudaError_t launch_spread_yz(const WaveArgs& a, cudaStream_t s) {
  if (a.lop_tiled) {
    // the tiled rows zero-fill by the tiles' stage plans: k_tile_plan first
    if (!a.lop || !direct_planes(a) || (reinterpret_cast<uintptr_t>(a.lop) & 127)) return cudaErrorInvalidValue;
    cudaError_t e = launch_tile_plan(a, (a.Lb + 7) / 8, s);
    if (e != cudaSuccess) return e;
  }
  CDK_DISPATCH_N(a.n, launch_spread_yz_t, a, s);
}
bool direct_planes(const WaveArgs& a) {
  const int cap = a.atom_cap > 0 ? a.atom_cap : a.max_atoms;
  return a.kyof != nullptr && cap <= kDirectMaxAtoms;
}
cudaError_t launch_yz_inv_argmin(const WaveArgs& a, cudaStream_t s) {
  if (a.bpairs) return launch_yz_pairs(a, s);
  CDK_DISPATCH_N(a.n, launch_yz_inv_t, a, s);
}
cudaError_t launch_tiebreak(const WaveArgs& a, const float* grids, float tol, cudaStream_t s) {
  if (!a.keys2 || !grids) return cudaErrorInvalidValue;
  k_tiebreak<<<(a.nrot + 3) / 4, 128, 0, s>>>(a, grids, tol);
  return cudaGetLastError();
}
cudaError_t launch_finalize(const WaveArgs& a, cudaStream_t s) {
  k_finalize<false><<<(a.nrot + 255) / 256, 256, 0, s>>>(a, nullptr, 0, nullptr);
  return cudaGetLastError();
}
cudaError_t launch_finalize_topk(const WaveArgs& a, const float* grids, int k, TopPose* top, cudaStream_t s) {
  if (!grids || !top || k < 1 || k > kTopMax) return cudaErrorInvalidValue;
  k_finalize<true><<<(a.nrot + 255) / 256 + 1, 256, 0, s>>>(a, grids, k, top);
  return cudaGetLastError();
}
cudaError_t launch_finalize_server(const WaveArgs& a, float* ebase, int* ibase, cudaStream_t s) {
  k_finalize_server<<<(a.nrot + 255) / 256, 256, 0, s>>>(a, ebase, ibase);
  return cudaGetLastError();
}
cudaError_t launch_receptor_fft(int n, int K, const float* grids, float2* scratch,
                                float2* phat, const float2* tw, int ct, cudaStream_t s) {
  CDK_DISPATCH_N(n, launch_receptor_t, K, grids, scratch, phat, tw, ct, s);
}

}  // namespace cdk
