// Spatial 1- and 2-RDMs of the variational wavefunction.
//
// Restates SHCIrdm::EvaluateRDM (SHCI/SHCIrdm.cpp:863-993) and
// SHCIrdm::EvaluateOneRDM (:996-1100) with cibra = ciket = c, over the
// connection lists of the stored Hamiltonian (every connected pair J < I of
// the variational space, the pairs the reference's build stores with their
// orbital differences, SHCI/SHCImakeHamiltonian.cpp:578-588):
//   diagonal  every occupied pair of every determinant, weight c_I^2;
//   single    J = I with d -> c: the 1-RDM pair (c, d) and, for every other
//             occupied spectator k of I, the 2-RDM elements of
//             populateSpatialRDM (:846-861), sign of the transposition times
//             -1 when k lies between c and d;
//   double    the two 2-RDM elements of the excitation, sign of
//             Determinant::parity(d1, d0, c1, c0) (SHCI/Determinants.cpp:332-357).
// The sums are kept in 64-bit fixed point (units of 2^-58, elements are
// bounded by 4 in magnitude) and added with integer atomics, so the result
// does not depend on the order or grouping of the additions and is bitwise
// reproducible; each term is rounded to the unit (2^-59 error per term).
//
// With an atomic per element the additions in L2 bounded it; now the integer
// instructions do (ALU pipe 79 % in k_rdm_off, L2 30 %). A term (p q; r s) stands for four elements, the images (p q; r s), (q p; s r),
// (r s; p q), (s r; q p), so it is added once and the last kernel sums the
// images: one addition for an alpha-beta double, two for one of a single spin
// ((p q; r s) and, negative, (p q; s r)). A single c <- d with every spectator
// k gives (k c; k d) and, for a k of its spin, -(k c; d k): these go to tables
// indexed [c][d][k], where the spectators of one single are neighbours and are
// added by the lanes of a warp together.
//
//   k_rdm_pack  determinants and coefficients in the matrix's storage order;
//   k_rdm_diag  the diagonal: sum of c_I^2 over the determinants that hold both
//               of two spin orbitals, a pair of orbitals per register;
//   k_rdm_off   warp per row, lanes over the row's connections J < I (rows
//               and columns in the stored Hamiltonian's storage order: each
//               connected pair is visited once, and its terms are symmetric
//               in the two determinants, so the order does not change the
//               sums);
//   k_rdm_fin   images and tables summed, fixed point -> FP64.
// 151,842 determinants, 8e7 pairs (mol24): off-diagonal 8.19 -> 1.20 ms (before,
// every element was added on its own, a spectator loop in one lane), diagonal
// 1.98 -> 0.17 ms (before, atomics in shared memory).
#include "ham.h"

namespace shci {

namespace {

constexpr double kRdmUnit = 288230376151711744.0;  // 2^58
constexpr int kRdmThreads = 256;

inline unsigned grid_for(size_t n, int threads, size_t max_blocks = 152 * 32) {
  size_t b = (n + threads - 1) / threads;
  if (b < 1) b = 1;
  if (b > max_blocks) b = max_blocks;
  return (unsigned)b;
}

__device__ __forceinline__ void add_fix(unsigned long long* p, long long v) {
  atomicAdd(p, (unsigned long long)v);
}

struct RdmDet {
  uint64_t a, b;  // alpha and beta string
  double c;
  double pad;
};
__global__ void k_rdm_pack(const Det2* __restrict__ dets, const double* __restrict__ c,
                           const uint32_t* __restrict__ perm, size_t N, RdmDet* __restrict__ out) {
  for (size_t p = (size_t)blockIdx.x * blockDim.x + threadIdx.x; p < N; p += (size_t)gridDim.x * blockDim.x) {
    const uint32_t u = perm[p];
    const Det2 d = dets[u];
    out[p] = RdmDet{det_alpha(d), det_beta(d), c[u], 0.0};
  }
}

// Pairs (p, q), q <= p, of spin orbitals (p in [0, n) alpha, [n, 2n) beta), 8
// per thread in registers; a block reads its share of the determinants in
// tiles. Pair (p, q) of different orbitals adds to (PQ, PQ) and (QP, QP), and of
// one spin subtracts from (PQ, QP) and (QP, PQ); (p, p) adds to the 1-RDM.
constexpr int kDiagPairs = 8;
__global__ void __launch_bounds__(kRdmThreads) k_rdm_diag(const RdmDet* __restrict__ dets, size_t N, int n,
                                                          unsigned long long* __restrict__ dd,
                                                          unsigned long long* __restrict__ dx,
                                                          unsigned long long* __restrict__ s1) {
  __shared__ ulonglong2 s_d[kRdmThreads];
  __shared__ long long s_v[kRdmThreads];
  const int m = 2 * n, npair = m * (m + 1) / 2;
  unsigned long long acc[kDiagPairs];
  int P[kDiagPairs], Q[kDiagPairs];
#pragma unroll
  for (int t = 0; t < kDiagPairs; ++t) {
    const int q = (int)((blockIdx.y * kDiagPairs + t) * kRdmThreads + threadIdx.x);
    acc[t] = 0ull;
    P[t] = Q[t] = -1;
    if (q < npair) {
      int i = (int)((sqrtf(8.0f * (float)q + 1.0f) - 1.0f) * 0.5f);  // corrected below
      while (i * (i + 1) / 2 > q) --i;
      while ((i + 1) * (i + 2) / 2 <= q) ++i;
      P[t] = i;
      Q[t] = q - i * (i + 1) / 2;
    }
  }
  for (size_t base = (size_t)blockIdx.x * kRdmThreads; base < N; base += (size_t)gridDim.x * kRdmThreads) {
    const size_t i = base + threadIdx.x;
    __syncthreads();
    if (i < N) {
      const RdmDet d = dets[i];
      s_d[threadIdx.x] = make_ulonglong2(d.a, d.b);
      s_v[threadIdx.x] = __double2ll_rn(d.c * d.c * kRdmUnit);
    }
    __syncthreads();
    const int cnt = (int)(N - base < (size_t)kRdmThreads ? N - base : (size_t)kRdmThreads);
    for (int k = 0; k < cnt; ++k) {
      const ulonglong2 d = s_d[k];
      const unsigned long long v = (unsigned long long)s_v[k];
#pragma unroll
      for (int t = 0; t < kDiagPairs; ++t) {
        if (P[t] < 0) continue;
        const uint64_t x = P[t] < n ? d.x >> P[t] : d.y >> (P[t] - n), y = Q[t] < n ? d.x >> Q[t] : d.y >> (Q[t] - n);
        if (x & y & 1ull) acc[t] += v;
      }
    }
  }
#pragma unroll
  for (int t = 0; t < kDiagPairs; ++t) {
    if (P[t] < 0 || acc[t] == 0ull) continue;
    const int I = P[t] < n ? P[t] : P[t] - n, J = Q[t] < n ? Q[t] : Q[t] - n;
    if (P[t] == Q[t]) {
      atomicAdd(s1 + I * n + I, acc[t]);
      continue;
    }
    atomicAdd(dd + I * n + J, acc[t]);
    atomicAdd(dd + J * n + I, acc[t]);
    if ((P[t] < n) == (Q[t] < n)) {
      atomicAdd(dx + I * n + J, 0ull - acc[t]);
      atomicAdd(dx + J * n + I, 0ull - acc[t]);
    }
  }
}

__device__ __forceinline__ size_t elem4(int n, int p, int q, int r, int s) {
  return ((size_t)(p * n + q) * n + r) * n + s;
}

// U: doubles by their first image; any, same: [c][d][k] of the singles over
// all spectators and over those of the moved electron's spin; s1: singles c <- d
// once (the diagonal of k_rdm_diag apart).
__global__ void __launch_bounds__(kRdmThreads) k_rdm_off(const RdmDet* __restrict__ dets, size_t N,
                                                         const int64_t* __restrict__ rowptr,
                                                         const int32_t* __restrict__ col, int n,
                                                         unsigned long long* __restrict__ U,
                                                         unsigned long long* __restrict__ any,
                                                         unsigned long long* __restrict__ same,
                                                         unsigned long long* __restrict__ s1) {
  const int lane = threadIdx.x & 31;
  const size_t warps = ((size_t)gridDim.x * blockDim.x) >> 5;
  for (size_t I = ((size_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5; I < N; I += warps) {
    const uint64_t A = dets[I].a, B = dets[I].b;
    const double cI = dets[I].c;
    const int64_t p0 = rowptr[I];
    int64_t p1 = rowptr[I + 1];
    {  // columns ascend: those below I come first
      int64_t lo = p0;
      while (lo < p1) {
        const int64_t mid = (lo + p1) >> 1;
        if ((size_t)col[mid] < I)
          lo = mid + 1;
        else
          p1 = mid;
      }
    }
    for (int64_t base = p0; base < p1; base += 32) {
      const int64_t p = base + lane;
      bool single = false;
      int cd = 0;  // c | d << 8 | spin << 16 of a single
      long long v = 0;
      if (p < p1) {
        const RdmDet J = dets[col[p]];
        v = __double2ll_rn(J.c * cI * kRdmUnit);
        const uint64_t x = A ^ J.a, y = B ^ J.b;
        if (x != 0 && y != 0) {
          if (bit_count(passed(A, B, x, false) ^ passed(B, J.a, y, true)) & 1) v = -v;
          add_fix(U + elem4(n, bit_index(x & J.a), bit_index(y & J.b), bit_index(x & A), bit_index(y & B)), v);
        } else {
          const bool beta = x == 0;
          const uint64_t z = beta ? y : x, S = beta ? B : A, O = beta ? A : B;
          const uint64_t d = z & S, c = z ^ d, di = low_one(d), ca = low_one(c);
          const int i = bit_index(di), a = bit_index(ca);
          const uint64_t m1 = passed(S, O, di | ca, beta);
          if (d == di) {
            single = true;
            if (bit_count(m1) & 1) v = -v;
            cd = a | (i << 8) | ((int)beta << 16);
          } else {
            const uint64_t dj = d ^ di, cb = c ^ ca;
            const int j = bit_index(dj), b = bit_index(cb);
            if (bit_count(m1 ^ passed(S ^ di ^ ca, O, dj | cb, beta)) & 1) v = -v;
            add_fix(U + elem4(n, b, a, j, i), v);
            add_fix(U + elem4(n, b, a, i, j), -v);
          }
        }
      }
      // the singles of these 32 entries one after another, lanes over orbitals
      for (unsigned ms = __ballot_sync(kFull, single); ms; ms &= ms - 1) {
        const int src = __ffs(ms) - 1;
        const int w = __shfl_sync(kFull, cd, src);
        const long long v0 = __shfl_sync(kFull, v, src);
        const int c0 = w & 255, d0 = (w >> 8) & 255;
        const bool beta = (w >> 16) != 0;
        const uint64_t S = (beta ? B : A) ^ (1ull << d0), O = beta ? A : B;
        if (lane == 0) add_fix(s1 + c0 * n + d0, v0);
        const size_t t = (size_t)(c0 * n + d0) * n;
        for (int k = lane; k < n; k += 32) {
          const long long ks = (long long)((S >> k) & 1ull), ko = (long long)((O >> k) & 1ull);
          if (ks + ko) add_fix(any + t + k, v0 * (ks + ko));
          if (ks) add_fix(same + t + k, v0);
        }
      }
    }
  }
}

__global__ void k_rdm_fin(const unsigned long long* __restrict__ U, const unsigned long long* __restrict__ any,
                          const unsigned long long* __restrict__ same, const unsigned long long* __restrict__ dd,
                          const unsigned long long* __restrict__ dx, const unsigned long long* __restrict__ s1,
                          const unsigned long long* __restrict__ s1d, int n, double* __restrict__ out) {
  const size_t n2 = (size_t)n * n, n4 = n2 * n2;
  for (size_t t = (size_t)blockIdx.x * blockDim.x + threadIdx.x; t < n4 + n2; t += (size_t)gridDim.x * blockDim.x) {
    unsigned long long v;
    if (t < n4) {
      const int s = (int)(t % n), r = (int)(t / n % n), q = (int)(t / n2 % n), p = (int)(t / (n2 * n));
      v = U[t] + U[elem4(n, q, p, s, r)] + U[elem4(n, r, s, p, q)] + U[elem4(n, s, r, q, p)];
      auto tab = [n](const unsigned long long* x, int c, int d, int k) { return x[(size_t)(c * n + d) * n + k]; };
      if (p == r) v += tab(any, q, s, p) + tab(any, s, q, p);
      if (q == s) v += tab(any, p, r, q) + tab(any, r, p, q);
      if (p == s) v -= tab(same, q, r, p) + tab(same, r, q, p);
      if (q == r) v -= tab(same, p, s, q) + tab(same, s, p, q);
      if (p == r && q == s) v += dd[p * n + q];
      if (p == s && q == r) v += dx[p * n + q];
    } else {
      const int q = (int)((t - n4) % n), p = (int)((t - n4) / n);
      v = s1[p * n + q] + s1[q * n + p] + s1d[p * n + q];
    }
    out[t] = (double)(long long)v * (1.0 / kRdmUnit);
  }
}

}  // namespace

void rdm_evaluate(const Det2* dets, const double* c, size_t N, const Csr& H, int n, DevBuf<unsigned long long>& fix,
                  DevBuf<double>& out, cudaStream_t s) {
  const size_t n2 = (size_t)n * n, n3 = n2 * n, n4 = n2 * n2;
  const size_t total = n4 + 2 * n3 + 4 * n2;
  fix.resize(total);
  out.resize(n4 + n2);
  SHCI_CUDA(cudaMemsetAsync(fix.p, 0, total * sizeof(unsigned long long), s));
  unsigned long long *U = fix.p, *any = U + n4, *same = any + n3, *dd = same + n3, *dx = dd + n2, *s1 = dx + n2,
                     *s1d = s1 + n2;
  DevBuf<RdmDet> packed;
  if (N > 0) {
    packed.resize(N);
    k_rdm_pack<<<grid_for(N, 256), 256, 0, s>>>(dets, c, H.perm.p, N, packed.p);
    SHCI_LAUNCH_CHECK();
    const int npair = n * (2 * n + 1);
    const unsigned ny = (unsigned)((npair + kRdmThreads * kDiagPairs - 1) / (kRdmThreads * kDiagPairs));
    const dim3 grid(grid_for(N, kRdmThreads, 152 * 4), ny);
    k_rdm_diag<<<grid, kRdmThreads, 0, s>>>(packed.p, N, n, dd, dx, s1d);
    SHCI_LAUNCH_CHECK();
    // 64 blocks per SM: rows differ, and blocks that end early make room for others
    // (150,000 determinants: 16 per SM 1.30 ms, 64 1.20, 128 1.24)
    k_rdm_off<<<grid_for(N * 32, kRdmThreads, 152 * 64), kRdmThreads, 0, s>>>(packed.p, N, H.rowptr.p, H.col.p, n, U,
                                                                              any, same, s1);
    SHCI_LAUNCH_CHECK();
  }
  k_rdm_fin<<<grid_for(n4 + n2, 256), 256, 0, s>>>(U, any, same, dd, dx, s1, s1d, n, out.p);
  SHCI_LAUNCH_CHECK();
}

}  // namespace shci
