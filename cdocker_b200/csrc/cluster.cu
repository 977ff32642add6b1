// cluster.cu -- diverse-conformer selection: greedy leader clustering by superposition RMSD.
//
// The reference picks conformer centres in GeneDiverseConformations
// (src/GeneDiverseConformations.cpp:84-111): conformers are ordered by energy with sort_index
// (include/GeneDiverseConformations.h:9-20, std::sort, not stable), the lowest is the first
// centre, and each following conformer becomes a new centre when its RMSD to every centre found
// so far, after optimal superposition (OpenBabel's OBAlign), exceeds the cut-off (1.5 A). The
// loop stops as soon as the number of centres equals maxNumOfConformations, a test made after
// each candidate from the second on (so a limit of 1 stops only if the second conformer is not a
// centre, and a limit <= 0 never stops).
//
// The outcome depends only on the predicate close(i, j) = rmsd(i, j) <= cutoff for j before i in
// energy order, so the GPU evaluates all of it at once and keeps the sequential part (the scan
// over candidates) to one bit-matrix pass:
//   k_center   per conformer (in energy order): centroid, centred coordinates of the selected
//              atoms, laid out [atom][xyz][conformer] so tiles stage with coalesced loads, and
//              G = sum |x|^2.
//   k_pairs    8 candidates x 32 earlier conformers per CTA (warp = candidate, lane = other
//              conformer); atoms streamed through shared memory in chunks of 32; per pair the 3x3
//              correlation S = sum a b^T, Horn's 4x4 quaternion key matrix, its largest
//              eigenvalue by Newton's method on the characteristic polynomial (Theobald's QCP
//              idea; the coefficients come from traces of N^2 and N^3 and det N), and
//              rmsd = sqrt(max(0, (Ga + Gb - 2 lambda) / n)). Cluster mode packs close(i, j) into
//              one 32-bit word per warp with a ballot; matrix mode writes the RMSD itself.
//   k_greedy   one CTA scans the candidates in order, 32 at a time.
// All double arithmetic uses explicit round-to-nearest intrinsics (no contraction), sqrt and
// division are IEEE, and every sum runs in atom order: the RMSDs are bit-identical to a host
// double-precision evaluation of the same recipe without fused multiply-adds.
#include <cudaTypedefs.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <mutex>
#include <string>
#include <vector>

#include "../../include/cdock_b200.h"
#include "cdk_internal.h"

namespace cdk {
namespace {

constexpr int CL_REF = 8;     // candidates per CTA (one per warp)
constexpr int CL_TGT = 32;    // other conformers per CTA (one per lane)
constexpr int CL_CHUNK = 32;  // atoms staged per step
constexpr int CL_MAX_CONF = 32768;      // cluster mode: the centre mask fits one CTA's words
constexpr int CL_MAX_CONF_MATRIX = 16384;

__device__ __forceinline__ double dm(double a, double b) { return __dmul_rn(a, b); }
__device__ __forceinline__ double da(double a, double b) { return __dadd_rn(a, b); }
__device__ __forceinline__ double ds(double a, double b) { return __dsub_rn(a, b); }

// centred coordinates of conformer order[c] (or c) -> X[(a*3 + d) * ld + c], G[c]. CTA = 32
// conformers: a thread per conformer and dimension for the mean and the centring, then one per
// conformer for G. Bound by the latency of one conformer's sums, which run in atom order (bit-
// identical to the host's): 23.7 us per 1,000 conformers of 40 atoms with one thread per conformer
// and its dimensions one after the other, GPU time.
constexpr int CL_CENTER = 32;
__global__ void __launch_bounds__(3 * CL_CENTER) k_center(int nConf, int nAtom, const double* __restrict__ coor,
                                                          const int* __restrict__ sel, int nSel,
                                                          const int* __restrict__ order, int ld, double* X,
                                                          double* __restrict__ G) {
  const int c = blockIdx.x * CL_CENTER + threadIdx.x / 3, d = threadIdx.x % 3;
  if (c < nConf) {
    const double* p = coor + (size_t)(order ? order[c] : c) * nAtom * 3 + d;
    double s = 0.0;
#pragma unroll 8
    for (int i = 0; i < nSel; ++i) s = da(s, p[sel[i] * 3]);
    const double m = __ddiv_rn(s, (double)nSel);
#pragma unroll 8
    for (int i = 0; i < nSel; ++i) X[((size_t)i * 3 + d) * ld + c] = ds(p[sel[i] * 3], m);
  }
  __syncthreads();
  const int g = blockIdx.x * CL_CENTER + threadIdx.x;
  if (threadIdx.x < CL_CENTER && g < nConf) {
    double sum = 0.0;
#pragma unroll 4
    for (int i = 0; i < nSel; ++i) {
      const double* v = X + (size_t)i * 3 * ld + g;
      const double x = v[0], y = v[ld], z = v[2 * (size_t)ld];
      sum = da(sum, da(da(dm(x, x), dm(y, y)), dm(z, z)));
    }
    G[g] = sum;
  }
}

// minimum RMSD over rotations from the correlation S[p*3+q] = sum a_p b_q of centred sets
__device__ double rmsd_from_corr(const double* S, double Ga, double Gb, int n) {
  const double Sxx = S[0], Sxy = S[1], Sxz = S[2], Syx = S[3], Syy = S[4], Syz = S[5],
               Szx = S[6], Szy = S[7], Szz = S[8];
  double N[4][4];
  N[0][0] = da(da(Sxx, Syy), Szz);
  N[0][1] = ds(Syz, Szy);
  N[0][2] = ds(Szx, Sxz);
  N[0][3] = ds(Sxy, Syx);
  N[1][1] = ds(ds(Sxx, Syy), Szz);
  N[1][2] = da(Sxy, Syx);
  N[1][3] = da(Szx, Sxz);
  N[2][2] = ds(ds(Syy, Sxx), Szz);
  N[2][3] = da(Syz, Szy);
  N[3][3] = ds(ds(Szz, Sxx), Syy);
  N[1][0] = N[0][1];
  N[2][0] = N[0][2];
  N[3][0] = N[0][3];
  N[2][1] = N[1][2];
  N[3][1] = N[1][3];
  N[3][2] = N[2][3];
  // char. polynomial of the traceless N: l^4 + c2 l^2 + c1 l + c0,
  // c2 = -tr(N^2)/2, c1 = -tr(N^3)/3, c0 = det N (Newton's identities)
  double p2 = 0.0;
  for (int i = 0; i < 4; ++i)
    for (int j = 0; j < 4; ++j) p2 = da(p2, dm(N[i][j], N[i][j]));
  double p3 = 0.0;
  for (int i = 0; i < 4; ++i)
    for (int j = 0; j < 4; ++j) {
      const double n2 = da(da(da(dm(N[i][0], N[0][j]), dm(N[i][1], N[1][j])), dm(N[i][2], N[2][j])),
                           dm(N[i][3], N[3][j]));
      p3 = da(p3, dm(n2, N[j][i]));
    }
  // det by 2x2 minors of rows (0,1) and (2,3)
  auto mA = [&](int j, int k) { return ds(dm(N[0][j], N[1][k]), dm(N[0][k], N[1][j])); };
  auto mB = [&](int j, int k) { return ds(dm(N[2][j], N[3][k]), dm(N[2][k], N[3][j])); };
  double det = ds(dm(mA(0, 1), mB(2, 3)), dm(mA(0, 2), mB(1, 3)));
  det = da(det, dm(mA(0, 3), mB(1, 2)));
  det = da(det, dm(mA(1, 2), mB(0, 3)));
  det = ds(det, dm(mA(1, 3), mB(0, 2)));
  det = da(det, dm(mA(2, 3), mB(0, 1)));
  const double c2 = -dm(p2, 0.5);
  const double c1 = -__ddiv_rn(p3, 3.0);
  const double c0 = det;
  // Newton from (Ga + Gb) / 2, an upper bound of the largest root: monotone convergence
  double l = dm(da(Ga, Gb), 0.5);
  for (int it = 0; it < 50; ++it) {
    const double l2 = dm(l, l);
    const double P = da(dm(da(dm(da(l2, c2), l), c1), l), c0);
    const double dP = da(dm(da(dm(4.0, l2), dm(2.0, c2)), l), c1);
    if (dP == 0.0) break;
    const double ln = ds(l, __ddiv_rn(P, dP));
    if (fabs(ds(ln, l)) <= dm(1e-11, fabs(ln))) {
      l = ln;
      break;
    }
    l = ln;
  }
  double e = __ddiv_rn(ds(da(Ga, Gb), dm(2.0, l)), (double)n);
  if (!(e > 0.0)) e = 0.0;
  return __dsqrt_rn(e);
}

// rmsd(candidate i = ref, conformer j = target) for the tile i in [8 by, +8), j in [32 bx, +32).
// bits != nullptr: cluster mode (only j < i, packed); else out[i * nConf + j]
__global__ void __launch_bounds__(256) k_pairs(int nConf, int nSel, int ld,
                                               const double* __restrict__ X,
                                               const double* __restrict__ G, double cutoff,
                                               uint32_t* __restrict__ bits, int W,
                                               double* __restrict__ out) {
  __shared__ double sR[CL_CHUNK][3][CL_REF];
  __shared__ double sT[CL_CHUNK][3][CL_TGT];
  const int i0 = blockIdx.y * CL_REF, j0 = blockIdx.x * CL_TGT;
  if (bits && j0 > i0 + CL_REF - 1) return;  // no j < i in this tile (uniform over the CTA)
  const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
  const int i = i0 + w, j = j0 + lane;
  double S[9];
#pragma unroll
  for (int t = 0; t < 9; ++t) S[t] = 0.0;
  for (int a0 = 0; a0 < nSel; a0 += CL_CHUNK) {
    const int na = min(CL_CHUNK, nSel - a0);
    __syncthreads();
    for (int e = tid; e < na * 3 * CL_REF; e += blockDim.x) {
      const int r = e % CL_REF, ad = e / CL_REF;
      sR[ad / 3][ad % 3][r] = (i0 + r < nConf) ? X[((size_t)(a0 * 3) + ad) * ld + i0 + r] : 0.0;
    }
    for (int e = tid; e < na * 3 * CL_TGT; e += blockDim.x) {
      const int r = e % CL_TGT, ad = e / CL_TGT;
      sT[ad / 3][ad % 3][r] = (j0 + r < nConf) ? X[((size_t)(a0 * 3) + ad) * ld + j0 + r] : 0.0;
    }
    __syncthreads();
    for (int a = 0; a < na; ++a) {
      const double ax = sR[a][0][w], ay = sR[a][1][w], az = sR[a][2][w];
      const double bx = sT[a][0][lane], by = sT[a][1][lane], bz = sT[a][2][lane];
      S[0] = da(S[0], dm(ax, bx));
      S[1] = da(S[1], dm(ax, by));
      S[2] = da(S[2], dm(ax, bz));
      S[3] = da(S[3], dm(ay, bx));
      S[4] = da(S[4], dm(ay, by));
      S[5] = da(S[5], dm(ay, bz));
      S[6] = da(S[6], dm(az, bx));
      S[7] = da(S[7], dm(az, by));
      S[8] = da(S[8], dm(az, bz));
    }
  }
  const bool valid = i < nConf && j < nConf;
  double r = 0.0;
  if (valid && (!bits || j < i)) r = rmsd_from_corr(S, G[i], G[j], nSel);
  if (bits) {
    const unsigned word = __ballot_sync(0xffffffffu, valid && j < i && r <= cutoff);
    if (lane == 0 && i < nConf) bits[(size_t)i * W + blockIdx.x] = word;
  } else if (valid) {
    out[(size_t)i * nConf + j] = r;
  }
}

// The reference's greedy pass over candidates in energy order (positions), one CTA, 32 candidates
// at a time: warp w tests candidate w of the block against the centres of the earlier blocks (all
// lanes over the words of its row), then warp 0 settles the block in order, each candidate against
// the block's own centres so far (one word). Two barriers per 32 candidates; one barrier per
// candidate took 171 us for 1,000 conformers.
__global__ void __launch_bounds__(1024) k_greedy(int nConf, int W, const uint32_t* __restrict__ bits,
                                                 const int* __restrict__ order, int maxCenters,
                                                 int* __restrict__ centers, int* __restrict__ count_out) {
  __shared__ uint32_t s_cm[CL_MAX_CONF / 32];  // the centres so far, a bit per position
  __shared__ uint32_t s_word[32];              // the candidates' words of their own block
  __shared__ int s_close[32];
  __shared__ int s_done;
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  if (threadIdx.x == 0) s_done = 0;
  int count = 0;  // warp 0's
  for (int b = 0; b < W; ++b) {
    const int pi = 32 * b + w;
    const uint32_t* row = bits + (size_t)min(pi, nConf - 1) * W;
    uint32_t v = 0;
    for (int t = lane; t < b; t += 32) v |= row[t] & s_cm[t];
    const bool close = __any_sync(0xffffffffu, v != 0);
    if (lane == 0) {
      s_close[w] = close;
      s_word[w] = row[b];
    }
    __syncthreads();
    if (w == 0) {
      const uint32_t word = s_word[lane];
      const unsigned int far = ~__ballot_sync(0xffffffffu, s_close[lane] != 0);
      const int n = min(32, nConf - 32 * b);
      uint32_t cmb = 0;
      bool done = false;
      for (int i = 0; i < n && !done; ++i) {
        const uint32_t wi = __shfl_sync(0xffffffffu, word, i);
        if (b == 0 && i == 0) {  // position 0 is the first centre, before any test of the count
          cmb = 1u;
          if (lane == 0) centers[0] = order[0];
          count = 1;
          continue;
        }
        if (((far >> i) & 1) && !(wi & cmb)) {
          cmb |= 1u << i;
          if (lane == 0) centers[count] = order[32 * b + i];
          ++count;
        }
        done = count == maxCenters;
      }
      if (lane == 0) {
        s_cm[b] = cmb;
        s_done = done;
      }
    }
    __syncthreads();
    if (s_done) break;
  }
  if (threadIdx.x == 0) *count_out = count;
}

bool finite_all(const double* p, size_t n) {
  for (size_t i = 0; i < n; ++i)
    if (!std::isfinite(p[i])) return false;
  return true;
}

// selected atoms (mask != 0, or all)
std::vector<int> selected_atoms(int nAtom, const unsigned char* mask) {
  std::vector<int> sel;
  for (int a = 0; a < nAtom; ++a)
    if (!mask || mask[a]) sel.push_back(a);
  return sel;
}

// Stream and device memory of a call. An allocation, its free and a stream cost 0.8 ms of a
// 1,000-conformer call whose kernels take 0.12 ms (and an allocation up to 12 ms on a machine in use),
// so a few are kept between calls: at most CL_IDLE of at most CL_KEEP bytes each, one call at a time
// on each, given back to the device with its contexts (cdk_ctx_destroy) or on request
// (cdk_cluster_release). The list itself is never destroyed: no CUDA call runs while the process exits.
constexpr size_t CL_KEEP = (size_t)32 << 20;
constexpr size_t CL_IDLE = 2;

// The driver's number of the allocation that holds p: unique in the process, never used again (0: none).
// A device reset takes a kept space's memory and stream away, and a later allocation, the caller's own,
// may get the same address (seen on a B200: the first allocation after a reset did), so a kept space
// is known by this number and not by its address.
unsigned long long buffer_id(const void* p) {
  static const PFN_cuPointerGetAttribute_v4000 attribute = [] {
    void* f = nullptr;
    cudaDriverEntryPointQueryResult q{};
    if (cudaGetDriverEntryPointByVersion("cuPointerGetAttribute", &f, 12000, cudaEnableDefault, &q) != cudaSuccess ||
        q != cudaDriverEntryPointSuccess)
      f = nullptr;
    return reinterpret_cast<PFN_cuPointerGetAttribute_v4000>(f);
  }();
  unsigned long long id = 0;
  if (!attribute || !p ||
      attribute(&id, CU_POINTER_ATTRIBUTE_BUFFER_ID, reinterpret_cast<CUdeviceptr>(p)) != CUDA_SUCCESS)
    return 0;
  return id;
}

struct ClusterSpace {
  int dev = -1;
  void* base = nullptr;
  size_t cap = 0;
  cudaStream_t s = nullptr;
  unsigned long long id = 0;  // of base
  // its memory, and so its context and stream, are still its own
  bool alive() const { return id != 0 && buffer_id(base) == id; }
  void drop() {
    int d = 0;
    const bool moved = dev >= 0 && cudaGetDevice(&d) == cudaSuccess && d != dev;
    if (moved) cudaSetDevice(dev);
    if (base) cudaFree(base);
    if (s) cudaStreamDestroy(s);
    if (moved) cudaSetDevice(d);
    *this = ClusterSpace{};
  }
};
struct ClusterIdle {
  std::mutex mu;
  std::vector<ClusterSpace> spaces;
};
ClusterIdle& cluster_idle() {
  static ClusterIdle* const idle = new ClusterIdle;
  return *idle;
}

// One call's buffers, carved from its space; every return waits for the stream and hands the space
// back (or frees it: too large, or enough are kept)
struct ClusterBuffers {
  double *coor = nullptr, *X = nullptr, *G = nullptr;
  int *sel = nullptr, *order = nullptr;
  void* extra = nullptr;  // the caller's part
  std::vector<int> idx;   // sel, then order: host source of an asynchronous copy
  cudaStream_t s = nullptr;
  ClusterSpace space;
  cudaError_t take(size_t bytes) {
    int d = 0;
    cudaError_t e = cudaGetDevice(&d);
    if (e != cudaSuccess) return e;
    {
      ClusterIdle& idle = cluster_idle();
      std::lock_guard<std::mutex> lk(idle.mu);
      for (size_t i = 0; i < idle.spaces.size() && space.dev < 0; ++i)
        if (idle.spaces[i].dev == d) {
          space = idle.spaces[i];
          idle.spaces.erase(idle.spaces.begin() + i);
        }
    }
    if (space.base && !space.alive()) space = ClusterSpace{};  // the device was reset: nothing to give back
    space.dev = d;
    if (!space.s && (e = cudaStreamCreateWithFlags(&space.s, cudaStreamNonBlocking)) != cudaSuccess) {
      space.s = nullptr;
      return e;
    }
    s = space.s;
    if (bytes > space.cap) {
      if (space.base) cudaFree(space.base);
      space.base = nullptr;
      space.cap = 0;
      space.id = 0;
      if ((e = cudaMalloc(&space.base, bytes)) != cudaSuccess) {
        space.base = nullptr;
        return e;
      }
      space.cap = bytes;
      space.id = buffer_id(space.base);
    }
    return cudaSuccess;
  }
  ~ClusterBuffers() {
    if (!space.s) return;
    if (cudaStreamSynchronize(space.s) == cudaSuccess && space.id != 0 && space.cap <= CL_KEEP) {
      ClusterIdle& idle = cluster_idle();
      std::lock_guard<std::mutex> lk(idle.mu);
      if (idle.spaces.size() < CL_IDLE) {
        idle.spaces.push_back(space);
        return;
      }
    }
    space.drop();
  }
};

#define CL_CUDA(call)                                                     \
  do {                                                                    \
    const cudaError_t e_ = (call);                                        \
    if (e_ != cudaSuccess) {                                              \
      set_error(std::string(#call) + ": " + cudaGetErrorString(e_));      \
      return e_ == cudaErrorMemoryAllocation ? CDK_ERR_NOMEM : CDK_ERR_CUDA; \
    }                                                                     \
  } while (0)

// shared set-up: memory (and `extra` bytes for the caller), copies, centring (in `order` when
// given); returns the leading dimension
int prepare(ClusterBuffers& b, int nConf, int nAtom, const double* coor,
            const std::vector<int>& sel, const std::vector<int>* order, size_t extra, int* ld_out) {
  auto up = [](size_t x) { return (x + 255) & ~(size_t)255; };
  const int ld = (nConf + CL_TGT - 1) / CL_TGT * CL_TGT;
  const int nSel = (int)sel.size();
  const size_t b_coor = up(sizeof(double) * (size_t)nConf * nAtom * 3), b_X = up(sizeof(double) * (size_t)nSel * 3 * ld),
               b_G = up(sizeof(double) * ld);
  std::vector<int>& idx = b.idx;
  idx = sel;
  if (order) idx.insert(idx.end(), order->begin(), order->end());
  const size_t b_idx = up(sizeof(int) * idx.size());
  CL_CUDA(b.take(b_coor + b_X + b_G + b_idx + extra));
  char* p = static_cast<char*>(b.space.base);
  b.coor = reinterpret_cast<double*>(p);
  b.X = reinterpret_cast<double*>(p + b_coor);
  b.G = reinterpret_cast<double*>(p + b_coor + b_X);
  b.sel = reinterpret_cast<int*>(p + b_coor + b_X + b_G);
  b.order = order ? b.sel + nSel : nullptr;
  b.extra = p + b_coor + b_X + b_G + b_idx;
  CL_CUDA(cudaMemcpyAsync(b.coor, coor, sizeof(double) * (size_t)nConf * nAtom * 3,
                          cudaMemcpyHostToDevice, b.s));
  CL_CUDA(cudaMemcpyAsync(b.sel, idx.data(), sizeof(int) * idx.size(), cudaMemcpyHostToDevice, b.s));
  k_center<<<(nConf + CL_CENTER - 1) / CL_CENTER, 3 * CL_CENTER, 0, b.s>>>(nConf, nAtom, b.coor, b.sel, nSel, b.order,
                                                                           ld, b.X, b.G);
  CL_CUDA(cudaGetLastError());
  *ld_out = ld;
  return CDK_OK;
}

int check_inputs(int nConf, int nAtom, const double* coor, const unsigned char* mask, int cap,
                 std::vector<int>* sel) {
  if (nConf <= 0 || nAtom <= 0 || !coor) {
    set_error("nConf and nAtom must be positive and coor non-null");
    return CDK_ERR_INVALID;
  }
  if (nConf > cap) {
    set_error("too many conformers (limit " + std::to_string(cap) + ")");
    return CDK_ERR_INVALID;
  }
  if (!finite_all(coor, (size_t)nConf * nAtom * 3)) {
    set_error("non-finite conformer coordinate");
    return CDK_ERR_INVALID;
  }
  *sel = selected_atoms(nAtom, mask);
  if (sel->empty()) {
    set_error("the atom mask selects no atom");
    return CDK_ERR_INVALID;
  }
  return CDK_OK;
}

}  // namespace

int cluster_release(int dev) {
  std::vector<ClusterSpace> gone;
  {
    ClusterIdle& idle = cluster_idle();
    std::lock_guard<std::mutex> lk(idle.mu);
    for (size_t i = 0; i < idle.spaces.size();) {
      if (dev >= 0 && idle.spaces[i].dev != dev) {
        ++i;
        continue;
      }
      gone.push_back(idle.spaces[i]);
      idle.spaces.erase(idle.spaces.begin() + i);
    }
  }
  int freed = 0;
  for (ClusterSpace& sp : gone)
    if (sp.alive()) {
      sp.drop();
      ++freed;
    }
  return freed;
}

}  // namespace cdk

using namespace cdk;

extern "C" int cdk_cluster_conformers(int nConf, int nAtom, const double* coor,
                                      const double* energy, const unsigned char* atomMask,
                                      double cutoff, int maxCenters, int* centers,
                                      int* nCenters) {
  std::vector<int> sel;
  int rc = check_inputs(nConf, nAtom, coor, atomMask, CL_MAX_CONF, &sel);
  if (rc != CDK_OK) return rc;
  if (!energy || !centers || !nCenters || !(cutoff >= 0.0) || !std::isfinite(cutoff)) {
    set_error("energy, centers and nCenters must be non-null and cutoff finite, >= 0");
    return CDK_ERR_INVALID;
  }
  if (!finite_all(energy, (size_t)nConf)) {
    set_error("non-finite conformer energy");
    return CDK_ERR_INVALID;
  }
  // energy order exactly as sort_index<double> (include/GeneDiverseConformations.h:9-20)
  std::vector<size_t> idx((size_t)nConf);
  for (size_t i = 0; i != idx.size(); ++i) idx[i] = i;
  std::sort(idx.begin(), idx.end(), [energy](size_t i1, size_t i2) { return energy[i1] < energy[i2]; });
  std::vector<int> order(idx.begin(), idx.end());
  ClusterBuffers b;
  int ld = 0;
  const int W = (nConf + 31) / 32;
  // the result: the count, then the centres
  const size_t b_bits = (sizeof(uint32_t) * (size_t)nConf * W + 255) & ~(size_t)255;
  rc = prepare(b, nConf, nAtom, coor, sel, &order, b_bits + sizeof(int) * ((size_t)nConf + 1), &ld);
  if (rc != CDK_OK) return rc;
  uint32_t* bits = static_cast<uint32_t*>(b.extra);
  int* result = reinterpret_cast<int*>(static_cast<char*>(b.extra) + b_bits);
  dim3 grid(W, (nConf + CL_REF - 1) / CL_REF);
  k_pairs<<<grid, 256, 0, b.s>>>(nConf, (int)sel.size(), ld, b.X, b.G, cutoff, bits, W, nullptr);
  CL_CUDA(cudaGetLastError());
  k_greedy<<<1, 1024, 0, b.s>>>(nConf, W, bits, b.order, maxCenters, result + 1, result);
  CL_CUDA(cudaGetLastError());
  std::vector<int> got((size_t)nConf + 1);
  CL_CUDA(cudaMemcpyAsync(got.data(), result, sizeof(int) * got.size(), cudaMemcpyDeviceToHost, b.s));
  CL_CUDA(cudaStreamSynchronize(b.s));
  const int count = got[0];
  if (count < 1 || count > nConf) {
    set_error("clustering returned an invalid centre count");
    return CDK_ERR_CUDA;
  }
  std::copy(got.begin() + 1, got.begin() + 1 + count, centers);
  *nCenters = count;
  return CDK_OK;
}

extern "C" int cdk_cluster_release(void) { return cluster_release(-1); }

extern "C" int cdk_pair_rmsd(int nConf, int nAtom, const double* coor,
                             const unsigned char* atomMask, double* out) {
  std::vector<int> sel;
  int rc = check_inputs(nConf, nAtom, coor, atomMask, CL_MAX_CONF_MATRIX, &sel);
  if (rc != CDK_OK) return rc;
  if (!out) {
    set_error("out must be non-null");
    return CDK_ERR_INVALID;
  }
  ClusterBuffers b;
  int ld = 0;
  rc = prepare(b, nConf, nAtom, coor, sel, nullptr, sizeof(double) * (size_t)nConf * nConf, &ld);
  if (rc != CDK_OK) return rc;
  double* d_out = static_cast<double*>(b.extra);
  dim3 grid((nConf + CL_TGT - 1) / CL_TGT, (nConf + CL_REF - 1) / CL_REF);
  k_pairs<<<grid, 256, 0, b.s>>>(nConf, (int)sel.size(), ld, b.X, b.G, 0.0, nullptr, 0, d_out);
  CL_CUDA(cudaGetLastError());
  CL_CUDA(cudaMemcpyAsync(out, d_out, sizeof(double) * (size_t)nConf * nConf, cudaMemcpyDeviceToHost, b.s));
  CL_CUDA(cudaStreamSynchronize(b.s));
  return CDK_OK;
}
