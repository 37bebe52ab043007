// Sigma (y = H x) on the stored Hamiltonian and the tall-skinny vector
// kernels of the block Davidson solver.
//
// Sigma replaces Hmult2::operator() (SHCI/Hmult.h:52-150). The reference
// stores the lower triangle and scatters symmetrically into a private
// temporary; here every row is complete (both triangles), so each row is
// owned by VW lanes of one warp and written once, without atomics:
//   y[I] = diag[I] x[I] (FP64) + sum_J h_IJ x[J]
// Mixed path: h in FP32, x in FP32, FP32 accumulation, the FP64 diagonal term
// added in FP64. Plain path: FP64 throughout. k vectors share one pass over
// the matrix (x is row-interleaved, one 4/8/16-byte gather per column index).
//
// The Davidson kernels (Gram products, Ritz combinations, residuals and the
// diagonal preconditioner of SHCI/Davidson.cpp:85-106) reduce in a fixed
// order, so results do not depend on scheduling.
#include <cstdlib>

#include "ham.h"

namespace shci {

static inline unsigned grid_for(size_t n, int threads, size_t max_blocks = 152 * 32) {
  size_t b = (n + threads - 1) / threads;
  if (b < 1) b = 1;
  if (b > max_blocks) b = max_blocks;
  return (unsigned)b;
}

// Compensated FP32 accumulation: the running sum s carries an FP32 error term
// c that collects the rounding error of every product (FMA residual) and of
// every addition (TwoSum), so s + c equals the exact sum of the FP32 products
// to about 2^-44 relative, whatever the summation order.
//
// Why it matters: the selected space is closed under the alpha <-> beta flip
// and H commutes with it, so a Davidson run seeded with a flip-even vector
// stays flip-even in exact arithmetic -- and in FP64, which is how the
// reference converges to the state of its reference determinant. A row and
// its flipped partner hold the same products in a different order; plain FP32
// accumulation rounds them differently, breaking the symmetry at 1e-7, and a
// lower flip-odd state (present in some spaces) can then take over the solve.
// (Acc, acc_add and acc_merge live in shci_common.cuh.)

template <int KP>
struct VecF;
template <>
struct VecF<1> {
  __device__ static void fma(Acc* acc, float h, const float* x, int j) { acc_add(acc[0], h, __ldg(x + j)); }
};
template <>
struct VecF<2> {
  __device__ static void fma(Acc* acc, float h, const float* x, int j) {
    float2 v = __ldg(reinterpret_cast<const float2*>(x) + j);
    acc_add_rounded(acc[0], h, v.x);
    acc_add_rounded(acc[1], h, v.y);
  }
};
template <>
struct VecF<4> {
  __device__ static void fma(Acc* acc, float h, const float* x, int j) {
    float4 v = __ldg(reinterpret_cast<const float4*>(x) + j);
    acc_add_rounded(acc[0], h, v.x);
    acc_add_rounded(acc[1], h, v.y);
    acc_add_rounded(acc[2], h, v.z);
    acc_add_rounded(acc[3], h, v.w);
  }
};

// Row walk shared by the stored-matrix sigma kernels: 32 / VW rows per warp, VW
// lanes each, every lane of a warp in step, so the width-VW shuffles always run
// on full warps. A kernel's Body sums spans of a row and writes the result.
//
// Single vector (kBalanced): block b owns the contiguous rows whose nonzeros
// fall in the b-th equal share of all nonzeros -- equal work per block
// whatever the row lengths -- and its warps take the next rows of that range
// from a shared-memory counter. Consecutive rows of the determinant order are
// close determinants with largely the same connections, so the rows one block
// runs together gather the same parts of x and hit in L1 (launched as two
// blocks per SM, one wave).
// Several vectors: the grid strides over the rows (x is k times larger and
// the band of rows the whole GPU works on at once is what stays in cache).
//
// A row is summed in pieces of Body::kPiece entries, added in order. The lowest
// determinants' rows hold tens of times the mean (19,739 of 80,730 columns
// against 881), and one warp on such a row outlasts the rest of the launch: in
// the balanced walk their pieces are put aside and shared by the block's warps
// after its other rows (Body::kAside). The sums are the same either way. The FP32
// bodies put nothing aside: the second phase's registers cost their first more
// than the tail (k = 2, 16,068 rows 34 -> 32 us without, compact copy 30 -> 19 us,
// and 2.47 -> 2.41 ms at 1.2 million).
constexpr int kTasks = 96;  // pieces a block can put aside; further long rows stay with their warp

// First index of the ascending a[0, n) with a[i] >= v, found by a warp: 32
// probes a step (a thread's binary search was 2 x 18 dependent loads at the
// start of every launch).
__device__ __forceinline__ size_t warp_lower_bound(const int64_t* __restrict__ a, size_t n, int64_t v) {
  const size_t lane = threadIdx.x & 31;
  size_t lo = 0;
  while (n > 32) {
    const size_t step = (n + 31) / 32, i = step * lane + step - 1;
    const int c = __popc(__ballot_sync(kFull, i < n && a[lo + i] < v));
    lo += step * c;
    n = step * c >= n ? 0 : (n - step * c < step ? n - step * c : step - 1);
  }
  return lo + __popc(__ballot_sync(kFull, lane < n && a[lo + lane] < v));
}

template <int VW, class Body>
__device__ __forceinline__ void reduce_lanes(typename Body::A (&acc)[Body::KP]) {
#pragma unroll
  for (int c = 0; c < Body::KP; ++c) {
#pragma unroll
    for (int o = VW / 2; o; o >>= 1) acc[c] = Body::across(acc[c], o, VW);
  }
}

// The row at position pos (none when !live), by VW lanes of a warp.
template <int VW, class Body>
__device__ __forceinline__ void sum_row(const Body& k, size_t pos, bool live, int64_t p0, int64_t p1) {
  using A = typename Body::A;
  const int sub = threadIdx.x & (VW - 1);
  A tot[Body::KP];
#pragma unroll
  for (int c = 0; c < Body::KP; ++c) tot[c] = A{};
  const bool whole = p1 - p0 <= Body::kPiece;
  int64_t q = whole ? p1 : p0 + Body::kPiece;
  k.template span<VW>(tot, p0, q, sub);
  reduce_lanes<VW, Body>(tot);
  if (VW == 32 ? !whole : __any_sync(kFull, !whole)) {
#pragma unroll 1
    while (VW == 32 ? q < p1 : __any_sync(kFull, q < p1)) {
      const int64_t e = q + Body::kPiece < p1 ? q + Body::kPiece : p1;
      A acc[Body::KP];
#pragma unroll
      for (int c = 0; c < Body::KP; ++c) acc[c] = A{};
      k.template span<VW>(acc, q, e, sub);
      reduce_lanes<VW, Body>(acc);
      if (q < p1)
#pragma unroll
        for (int c = 0; c < Body::KP; ++c) tot[c] = Body::add(tot[c], acc[c]);
      q = e;
    }
  }
  if (sub == 0 && live) k.finish(pos, tot);
}

template <int VW, bool kBalanced, class Body>
__device__ __forceinline__ void walk_rows(const int64_t* __restrict__ rowptr, size_t N, const Body& k) {
  constexpr int kPiece = Body::kPiece;
  const int lane = threadIdx.x & 31;
  if constexpr (kBalanced) {
    using A = typename Body::A;
    struct Task {
      uint32_t row;
      int piece;
    };
    constexpr bool kAside = VW == 32 && Body::kAside;
    __shared__ unsigned s_next, s_end, s_tasks, s_task_next;  // rows are below 2^31
    __shared__ Task s_task[kAside ? kTasks : 1];
    __shared__ A s_acc[kAside ? kTasks : 1][Body::KP];
    const int warp = threadIdx.x >> 5;
    if (warp < 2) {
      const int64_t nnz = rowptr[N];
      const int64_t g = (int64_t)gridDim.x, b = (int64_t)blockIdx.x + warp;
      size_t r = b >= g ? N : warp_lower_bound(rowptr, N + 1, nnz / g * b + nnz % g * b / g);
      if (r > N) r = N;
      if (lane == 0) (warp ? s_end : s_next) = (unsigned)r;
    }
    if (threadIdx.x == 64) s_tasks = s_task_next = 0;
    if (kAside && threadIdx.x >= 128 && threadIdx.x < 128 + kTasks) s_task[threadIdx.x - 128].row = 0xffffffffu;
    __syncthreads();
    const unsigned end = s_end;
    while (true) {
      unsigned wr = 0;
      if (lane == 0) wr = atomicAdd(&s_next, (unsigned)(32 / VW));
      wr = __shfl_sync(kFull, wr, 0);
      if (wr >= end) break;
      const size_t pos = wr + lane / VW;
      const bool live = pos < end;
      const int64_t p0 = live ? __ldg(rowptr + pos) : 0, p1 = live ? __ldg(rowptr + pos + 1) : 0;
      if constexpr (kAside) {
        if (p1 - p0 > kPiece) {
          const int np = (int)((p1 - p0 + kPiece - 1) / kPiece);
          int at = kTasks;
          if (np <= kTasks) {
            if (lane == 0) at = (int)atomicAdd(&s_tasks, (unsigned)np);
            at = __shfl_sync(kFull, at, 0);
          }
          if (at + np <= kTasks) {
            for (int t = lane; t < np; t += 32) s_task[at + t] = Task{(uint32_t)pos, t};
            continue;
          }
        }
      }
      sum_row<VW, Body>(k, live ? pos : 0, live, p0, p1);
    }
    if constexpr (kAside) {
      __syncthreads();
      const int nt = (int)(s_tasks < (unsigned)kTasks ? s_tasks : (unsigned)kTasks);
      if (nt == 0) return;
      while (true) {
        int t = 0;
        if (lane == 0) t = (int)atomicAdd(&s_task_next, 1u);
        t = __shfl_sync(kFull, t, 0);
        if (t >= nt) break;
        const Task w = s_task[t];
        if (w.row == 0xffffffffu) continue;
        const int64_t p0 = rowptr[w.row] + (int64_t)w.piece * kPiece, p1 = rowptr[w.row + 1];
        A acc[Body::KP];
#pragma unroll
        for (int c = 0; c < Body::KP; ++c) acc[c] = A{};
        k.template span<32>(acc, p0, p0 + kPiece < p1 ? p0 + kPiece : p1, lane);
        reduce_lanes<32, Body>(acc);
        if (lane == 0)
#pragma unroll
          for (int c = 0; c < Body::KP; ++c) s_acc[t][c] = acc[c];
      }
      __syncthreads();
      const int t = (int)threadIdx.x;
      if (t < nt && s_task[t].row != 0xffffffffu && s_task[t].piece == 0) {
        A tot[Body::KP];
#pragma unroll
        for (int c = 0; c < Body::KP; ++c) tot[c] = s_acc[t][c];
        for (int u = t + 1; u < nt && s_task[u].row == s_task[t].row; ++u)
#pragma unroll
          for (int c = 0; c < Body::KP; ++c) tot[c] = Body::add(tot[c], s_acc[u][c]);
        k.finish(s_task[t].row, tot);
      }
    }
  } else {
    const size_t rows_per_warp = 32 / VW;
    const size_t stride = ((size_t)gridDim.x * blockDim.x / 32) * rows_per_warp;
    for (size_t wr = (((size_t)blockIdx.x * blockDim.x + threadIdx.x) / 32) * rows_per_warp; wr < N; wr += stride) {
      const size_t r = wr + lane / VW;
      const bool live = r < N;
      sum_row<VW, Body>(k, live ? r : 0, live, live ? __ldg(rowptr + r) : 0, live ? __ldg(rowptr + r + 1) : 0);
    }
  }
}

// Compensated sums: lane halves are merged in lane order, so that both
// partners of a pair compute the same value.
struct AccSum {
  using A = Acc;
  __device__ static __forceinline__ Acc across(Acc a, int o, int width) {
    Acc other{__shfl_xor_sync(kFull, a.s, o, width), __shfl_xor_sync(kFull, a.c, o, width)};
    if ((threadIdx.x & o) == 0) {
      acc_merge(a, other);
      return a;
    }
    acc_merge(other, a);
    return other;
  }
  __device__ static __forceinline__ Acc add(Acc a, const Acc& b) {
    acc_merge(a, b);
    return a;
  }
};
struct DoubleSum {
  using A = double;
  __device__ static __forceinline__ double across(double a, int o, int width) {
    return a + __shfl_xor_sync(kFull, a, o, width);
  }
  __device__ static __forceinline__ double add(double a, double b) { return a + b; }
};

// FP32 sigma on int32 columns. One and two vectors walk balanced row ranges
// (two blocks per SM); four vectors the grid-strided rows, which is
// faster there (mol24, 2.91 M determinants: k = 2 10.8 ms balanced against
// 12.6 ms strided; k = 4 20.6 ms against 16.9 ms).
// Four blocks per SM, 64 registers: the unrolled gathers stay in flight (202,439
// determinants of 36 orbitals, k = 4: 808 us; 852 with the compiler's 71 registers,
// 882 with five blocks, 900 with six, 1105 with eight).
template <int KP_>
struct MixedBody : AccSum {
  static constexpr int KP = KP_;
  static constexpr bool kAside = false;
  static constexpr int kPiece = 4096;
  const int32_t* __restrict__ col;
  const float* __restrict__ val;
  const double* __restrict__ diag;
  const float* __restrict__ x;
  int k;
  double* __restrict__ y;
  size_t ldy;
  const uint32_t* __restrict__ perm;
  const uint32_t* __restrict__ xpos;
  // Consecutive lanes take consecutive nonzeros: the column and value loads
  // are coalesced, and on a column-sorted row the 32 gathers of one
  // instruction land on as few 32-byte sectors of x as the row allows.
  // Four nonzeros per lane per step keep four gathers in flight.
  template <int VW>
  __device__ __forceinline__ void span(Acc (&acc)[KP], int64_t p, int64_t p1, int sub) const {
    p += sub;
    for (; p + 3 * VW < p1; p += 4 * VW) {
      const int j0 = __ldcs(col + p), j1 = __ldcs(col + p + VW);
      const int j2 = __ldcs(col + p + 2 * VW), j3 = __ldcs(col + p + 3 * VW);
      const float h0 = __ldcs(val + p), h1 = __ldcs(val + p + VW);
      const float h2 = __ldcs(val + p + 2 * VW), h3 = __ldcs(val + p + 3 * VW);
      VecF<KP>::fma(acc, h0, x, j0);
      VecF<KP>::fma(acc, h1, x, j1);
      VecF<KP>::fma(acc, h2, x, j2);
      VecF<KP>::fma(acc, h3, x, j3);
    }
    for (; p < p1; p += VW) VecF<KP>::fma(acc, __ldcs(val + p), x, __ldcs(col + p));
  }
  __device__ __forceinline__ void finish(size_t r, const Acc (&acc)[KP]) const {
    const size_t o = __ldg(perm + r);
    const size_t xr = xpos ? (size_t)__ldg(xpos + r) : r;  // the row's own x (row blocks: its storage position)
    const double dg = diag[o];
#pragma unroll
    for (int c = 0; c < KP; ++c)
      if (c < k) y[(size_t)c * ldy + o] = dg * (double)x[xr * KP + c] + ((double)acc[c].s + (double)acc[c].c);
  }
};
template <int VW, int KP, bool kBalWalk = (KP <= 2)>
__global__ void __launch_bounds__(kBalWalk ? 1024 : 256, kBalWalk ? 2 : 4)
    k_sigma_mixed(const int64_t* __restrict__ rowptr, size_t N, const __grid_constant__ MixedBody<KP> k) {
  walk_rows<VW, kBalWalk>(rowptr, N, k);
}

// Single-vector FP32 sigma on the compact copy (Csr::clo, chi, cval): 24-bit
// columns in two planes, 7 bytes per entry streamed instead of 8. A row's
// entries are stored in chunks of 4 x VW, place 4 i + u of a chunk holding
// entry u VW + i: a lane reads its four entries with one load per plane, and
// each of the four gathers takes VW consecutive entries of the row, whose
// columns ascend, so it falls on few 128-byte lines of x. The remainder of a row
// is stored in order. (Before: 16-bit differences of consecutive entries in
// order, 6 bytes, bridged across wide gaps; a lane's four entries were
// neighbours, so each gather spread over four times as many lines, and L1's
// tag rate bound it at 90 %.) 1.2 million determinants, 2.03e9 entries: 2.75 ->
// 2.43 ms, 86 % of the measured copy bandwidth.
struct MixedCompactBody : AccSum {
  static constexpr int KP = 1;
  static constexpr bool kAside = false;
  static constexpr int kPiece = 4096;
  const uint16_t* __restrict__ clo;
  const uint8_t* __restrict__ chi;
  const float* __restrict__ val;
  const double* __restrict__ diag;
  const float* __restrict__ x;
  double* __restrict__ y;
  const uint32_t* __restrict__ perm;
  const uint32_t* __restrict__ xpos;
  // (a padding entry has value 0 and gathers nothing)
  __device__ __forceinline__ float at(float h, unsigned c) const { return h != 0.f ? __ldg(x + c) : 0.f; }
  template <int VW>
  __device__ __forceinline__ void span(Acc (&acc)[1], int64_t q, int64_t p1, int sub) const {
    for (; q + 4 * VW <= p1; q += 4 * VW) {
      const int64_t p = q + 4 * sub;
      const uint2 lo = __ldcs(reinterpret_cast<const uint2*>(clo + p));
      const unsigned hi = __ldcs(reinterpret_cast<const unsigned*>(chi + p));
      const float4 h = __ldcs(reinterpret_cast<const float4*>(val + p));
      const float x0 = at(h.x, __byte_perm(lo.x, hi, 0x5410) & 0xffffffu);
      const float x1 = at(h.y, __byte_perm(lo.x, hi, 0x6532) & 0xffffffu);
      const float x2 = at(h.z, __byte_perm(lo.y, hi, 0x7610) & 0xffffffu);
      const float x3 = at(h.w, __byte_perm(lo.y, hi, 0x0732) & 0xffffffu);
      acc_add(acc[0], h.x, x0);
      acc_add(acc[0], h.y, x1);
      acc_add(acc[0], h.z, x2);
      acc_add(acc[0], h.w, x3);
    }
    for (int64_t p = q + sub; p < p1; p += VW) {
      const float h = __ldcs(val + p);
      acc_add(acc[0], h, at(h, (unsigned)__ldcs(clo + p) | (unsigned)__ldcs(chi + p) << 16));
    }
  }
  __device__ __forceinline__ void finish(size_t r, const Acc (&acc)[1]) const {
    const size_t o = __ldg(perm + r);
    const size_t xr = xpos ? (size_t)__ldg(xpos + r) : r;
    y[o] = diag[o] * (double)x[xr] + ((double)acc[0].s + (double)acc[0].c);
  }
};
template <int VW>
__global__ void __launch_bounds__(1024, 2)
    k_sigma_compact(const int64_t* __restrict__ rowptr, size_t N, const __grid_constant__ MixedCompactBody k) {
  walk_rows<VW, true>(rowptr, N, k);
}

// ---- building the compact copy ----------------------------------------------
// rows padded to a multiple of four entries, for the loads of the next row
__global__ void k_c_len(const int64_t* __restrict__ rowptr, size_t N, int64_t* __restrict__ len) {
  for (size_t r = (size_t)blockIdx.x * blockDim.x + threadIdx.x; r < N; r += (size_t)gridDim.x * blockDim.x)
    len[r] = (rowptr[r + 1] - rowptr[r] + 3) & ~(int64_t)3;
}
template <int VW>
__global__ void __launch_bounds__(256) k_c_fill(const int64_t* __restrict__ rowptr, const int32_t* __restrict__ col,
                                                const float* __restrict__ vhi, size_t N,
                                                const int64_t* __restrict__ crow, uint16_t* __restrict__ clo,
                                                uint8_t* __restrict__ chi, float* __restrict__ cval) {
  const int sub = threadIdx.x & (VW - 1);
  const size_t groups = (size_t)gridDim.x * blockDim.x / VW;
  for (size_t r = ((size_t)blockIdx.x * blockDim.x + threadIdx.x) / VW; r < N; r += groups) {
    const int64_t p0 = rowptr[r], n = rowptr[r + 1] - p0, o0 = crow[r], pad = crow[r + 1] - o0;
    int64_t q = 0;
    for (; q + 4 * VW <= pad; q += 4 * VW) {
      uint32_t c[4];
      float h[4];
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        const int64_t e = q + u * VW + sub;
        c[u] = e < n ? (uint32_t)__ldcs(col + p0 + e) : 0u;
        h[u] = e < n ? __ldcs(vhi + p0 + e) : 0.f;
      }
      const int64_t o = o0 + q + 4 * sub;
      *reinterpret_cast<uint2*>(clo + o) =
          make_uint2(__byte_perm(c[0], c[1], 0x5410), __byte_perm(c[2], c[3], 0x5410));
      *reinterpret_cast<uint32_t*>(chi + o) =
          __byte_perm(__byte_perm(c[0], c[1], 0x0062), __byte_perm(c[2], c[3], 0x0062), 0x5410);
      *reinterpret_cast<float4*>(cval + o) = make_float4(h[0], h[1], h[2], h[3]);
    }
    for (int64_t e = q + sub; e < pad; e += VW) {
      const uint32_t c = e < n ? (uint32_t)col[p0 + e] : 0u;
      clo[o0 + e] = (uint16_t)c;
      chi[o0 + e] = (uint8_t)(c >> 16);
      cval[o0 + e] = e < n ? vhi[p0 + e] : 0.f;
    }
  }
}

static int pick_vw(const Csr& H) {
  double avg = H.N ? (double)H.nnz / (double)H.N : 0.0;
  if (avg >= 96) return 32;
  if (avg >= 40) return 16;
  if (avg >= 14) return 8;
  return 4;
}

// The copy is left out where columns need more than 24 bits and where the
// device has no room for it (SHCI_TRACE says so; shci_sigma_bytes counts what is
// read); the sigma then reads the int32 columns. Past 24 bits those are the better
// form: at 17.5 million columns differences of 16 bits, bridged across wide gaps,
// took 10.8 ms for 34 entries a row where int32 columns take 3.3, and 0.94 ms for
// 400,000 rows of 750 entries against 0.89.
void compress_csr(Csr& H, Prims& pr, cudaStream_t s) {
  H.drop_compressed();
  if (!H.vhi.p || H.N == 0 || H.ncols() > ((size_t)1 << 24)) return;
  const size_t N = H.N;
  try {
    DevBuf<int64_t> len;
    len.resize(N);
    k_c_len<<<grid_for(N, 256), 256, 0, s>>>(H.rowptr.p, N, len.p);
    SHCI_LAUNCH_CHECK();
    H.crow.resize(N + 1);
    int64_t total = 0;
    scan_exclusive_i64(len.p, H.crow.p, N, &total, pr, s);
    SHCI_CUDA(cudaMemcpyAsync(H.crow.p + N, &total, sizeof(int64_t), cudaMemcpyHostToDevice, s));
    const size_t cap = total > 0 ? (size_t)total : 1;
    H.clo.resize(cap);
    H.chi.resize(cap);
    H.cval.resize(cap);
    H.cnnz = total;
  } catch (const Error& e) {
    H.drop_compressed();
    if (e.code != kErrOOM) throw;
    if (trace_level() > 0)
      std::fprintf(stderr, "[ham] no device memory for the compact copy: FP32 sigma on int32 columns\n");
    return;
  }
  const int vw = pick_vw(H);
  const unsigned blocks = grid_for(N * (size_t)vw, 256, 152 * 16);
  switch (vw) {
    case 32: k_c_fill<32><<<blocks, 256, 0, s>>>(H.rowptr.p, H.col.p, H.vhi.p, N, H.crow.p, H.clo.p, H.chi.p, H.cval.p); break;
    case 16: k_c_fill<16><<<blocks, 256, 0, s>>>(H.rowptr.p, H.col.p, H.vhi.p, N, H.crow.p, H.clo.p, H.chi.p, H.cval.p); break;
    case 8: k_c_fill<8><<<blocks, 256, 0, s>>>(H.rowptr.p, H.col.p, H.vhi.p, N, H.crow.p, H.clo.p, H.chi.p, H.cval.p); break;
    default: k_c_fill<4><<<blocks, 256, 0, s>>>(H.rowptr.p, H.col.p, H.vhi.p, N, H.crow.p, H.clo.p, H.chi.p, H.cval.p); break;
  }
  SHCI_LAUNCH_CHECK();
  SHCI_CUDA(cudaStreamSynchronize(s));
  H.cvw = vw;
  H.cvalid = true;
}

template <int KP_>
struct F64Body : DoubleSum {
  static constexpr int KP = KP_;
  static constexpr bool kAside = KP == 1;
  static constexpr int kPiece = 2048;  // 1024: 25.4 ms, 2048: 23.9 ms, 4096: 27.2 ms for 126 sigmas of 81,233 rows
  const int32_t* __restrict__ col;
  const double* __restrict__ v64;
  const double* __restrict__ diag;
  const double* __restrict__ x;
  int k;
  double* __restrict__ y;
  size_t ldy;
  const uint32_t* __restrict__ perm;
  const uint32_t* __restrict__ xpos;
  // consecutive lanes on consecutive nonzeros (see MixedBody)
  template <int VW>
  __device__ __forceinline__ void span(double (&acc)[KP], int64_t p, int64_t p1, int sub) const {
    auto elem = [&](int64_t q, int j) {
      const double h = __ldcs(v64 + q);
#pragma unroll
      for (int c = 0; c < KP; ++c) acc[c] += h * __ldg(x + (size_t)j * KP + c);
    };
    p += sub;
    for (; p + 3 * VW < p1; p += 4 * VW) {
      const int j0 = __ldcs(col + p), j1 = __ldcs(col + p + VW);
      const int j2 = __ldcs(col + p + 2 * VW), j3 = __ldcs(col + p + 3 * VW);
      elem(p, j0);
      elem(p + VW, j1);
      elem(p + 2 * VW, j2);
      elem(p + 3 * VW, j3);
    }
    for (; p < p1; p += VW) elem(p, __ldcs(col + p));
  }
  __device__ __forceinline__ void finish(size_t r, const double (&acc)[KP]) const {
    const size_t o = __ldg(perm + r);
    const size_t xr = xpos ? (size_t)__ldg(xpos + r) : r;
    const double dg = diag[o];
#pragma unroll
    for (int c = 0; c < KP; ++c)
      if (c < k) y[(size_t)c * ldy + o] = dg * x[xr * KP + c] + acc[c];
  }
};
// One FP64 vector runs as two blocks of 768 threads per SM: 42 registers keep a
// row's loads in flight that 1024 threads' 32 do not (16,068 rows 45.7 -> 40.3 us,
// 82,090 rows 194.6 -> 190.1; 512 x 3 and x 4 slower at 250,000). The FP32 and
// float-float bodies are faster with 1024 (refine at 200,836 rows 488 against
// 517 us, compact copy at 1.2 million 2.50 against 2.69 ms).
constexpr int kF64Threads = 768;
template <int VW, int KP>
__global__ void __launch_bounds__(KP == 1 ? kF64Threads : 256, KP == 1 ? 2 : 1)
    k_sigma_f64(const int64_t* __restrict__ rowptr, size_t N, const __grid_constant__ F64Body<KP> k) {
  walk_rows<VW, KP == 1>(rowptr, N, k);
}

// Refinement sigma on the mixed path's head + tail values, in float-float
// arithmetic: x is split as x = xh + xl (two floats) and every product
// (hi + lo)(xh + xl) enters the compensated accumulator as its exactly
// rounded head hi*xh plus the FMA residual and the cross terms hi*xl + lo*xh.
// The result matches the FP64 product sum to ~1e-13 relative while keeping
// every operation of the inner loop on the FP32 pipe (the FP64 pipe of this
// GPU issues about two FMAs per clock per SM, so an FP64 head + tail sum,
// with its two conversions, one add and one FMA per nonzero, runs 3.5x
// slower). The diagonal term is added in FP64 from the unsplit x.
__device__ __forceinline__ void acc_add_ff(Acc& a, float hi, float lo, float xh, float xl) {
  const float p = __fmul_rn(hi, xh);
  const float pe = __fmaf_rn(hi, xh, -p);
  const float small = __fmaf_rn(hi, xl, __fmaf_rn(lo, xh, pe));
  const float t = __fadd_rn(a.s, p);
  const float bp = __fsub_rn(t, a.s);
  const float e = __fadd_rn(__fsub_rn(a.s, __fsub_rn(t, bp)), __fsub_rn(p, bp));
  a.s = t;
  a.c = __fadd_rn(a.c, __fadd_rn(e, small));
}

template <int KP>
struct VecFF;
template <>
struct VecFF<1> {
  __device__ static void fma(Acc* acc, float hi, float lo, const float* x, int j) {
    const float2 v = __ldg(reinterpret_cast<const float2*>(x) + j);
    acc_add_ff(acc[0], hi, lo, v.x, v.y);
  }
};
template <>
struct VecFF<2> {
  __device__ static void fma(Acc* acc, float hi, float lo, const float* x, int j) {
    const float4 v = __ldg(reinterpret_cast<const float4*>(x) + j);
    acc_add_ff(acc[0], hi, lo, v.x, v.y);
    acc_add_ff(acc[1], hi, lo, v.z, v.w);
  }
};
template <>
struct VecFF<4> {
  __device__ static void fma(Acc* acc, float hi, float lo, const float* x, int j) {
    const float4 v0 = __ldg(reinterpret_cast<const float4*>(x) + 2 * (size_t)j);
    const float4 v1 = __ldg(reinterpret_cast<const float4*>(x) + 2 * (size_t)j + 1);
    acc_add_ff(acc[0], hi, lo, v0.x, v0.y);
    acc_add_ff(acc[1], hi, lo, v0.z, v0.w);
    acc_add_ff(acc[2], hi, lo, v1.x, v1.y);
    acc_add_ff(acc[3], hi, lo, v1.z, v1.w);
  }
};

template <int KP_>
struct FFBody : AccSum {
  static constexpr int KP = KP_;
  static constexpr bool kAside = KP == 1;
  static constexpr int kPiece = 4096;
  const int32_t* __restrict__ col;
  const float* __restrict__ vhi;
  const float* __restrict__ vlo;
  const double* __restrict__ diag;
  const float* __restrict__ xff;
  const double* __restrict__ xd;
  size_t ldx;
  int c0, k;
  double* __restrict__ y;
  size_t ldy;
  const uint32_t* __restrict__ perm;
  template <int VW>
  __device__ __forceinline__ void span(Acc (&acc)[KP], int64_t p, int64_t p1, int sub) const {
    p += sub;
    for (; p + 3 * VW < p1; p += 4 * VW) {
      const int j0 = __ldcs(col + p), j1 = __ldcs(col + p + VW);
      const int j2 = __ldcs(col + p + 2 * VW), j3 = __ldcs(col + p + 3 * VW);
      const float h0 = __ldcs(vhi + p), h1 = __ldcs(vhi + p + VW);
      const float h2 = __ldcs(vhi + p + 2 * VW), h3 = __ldcs(vhi + p + 3 * VW);
      const float l0 = __ldcs(vlo + p), l1 = __ldcs(vlo + p + VW);
      const float l2 = __ldcs(vlo + p + 2 * VW), l3 = __ldcs(vlo + p + 3 * VW);
      VecFF<KP>::fma(acc, h0, l0, xff, j0);
      VecFF<KP>::fma(acc, h1, l1, xff, j1);
      VecFF<KP>::fma(acc, h2, l2, xff, j2);
      VecFF<KP>::fma(acc, h3, l3, xff, j3);
    }
    for (; p < p1; p += VW) VecFF<KP>::fma(acc, __ldcs(vhi + p), __ldcs(vlo + p), xff, __ldcs(col + p));
  }
  __device__ __forceinline__ void finish(size_t r, const Acc (&acc)[KP]) const {
    const size_t o = __ldg(perm + r);
    const double dg = diag[o];
#pragma unroll
    for (int c = 0; c < KP; ++c)
      if (c < k)
        y[(size_t)c * ldy + o] = dg * xd[(size_t)(c0 + c) * ldx + o] + ((double)acc[c].s + (double)acc[c].c);
  }
};
template <int VW, int KP>
__global__ void __launch_bounds__(KP == 1 ? 1024 : 256, KP == 1 ? 2 : 1)
    k_sigma_ff(const int64_t* __restrict__ rowptr, size_t N, const __grid_constant__ FFBody<KP> k) {
  walk_rows<VW, KP == 1>(rowptr, N, k);
}

// Launch shape of the stored-matrix sigma kernels (see walk_rows): one vector
// runs as two blocks of `threads1` per SM over nonzero-balanced row ranges;
// several vectors as a grid-strided launch of 256-thread blocks.
struct SigmaLaunch {
  unsigned blocks;
  int threads;
};
static int sm_count() {
  static int n = [] {
    int dev = 0, v = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || cudaDeviceGetAttribute(&v, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess)
      v = 152;
    return v > 0 ? v : 152;
  }();
  return n;
}
static SigmaLaunch sigma_launch(size_t N, int vw, int kp, int threads1 = 1024) {
  if (kp == 1) return SigmaLaunch{(unsigned)(2 * sm_count()), threads1};
  return SigmaLaunch{grid_for(N * (size_t)vw, 256, (size_t)sm_count() * 16), 256};
}

template <int KP>
static void launch_mixed(int vw, const Csr& H, const double* diag, const float* x, int k, double* y, size_t ldy,
                         cudaStream_t s) {
  const SigmaLaunch L = KP <= 2 ? sigma_launch(H.N, vw, 1) : sigma_launch(H.N, vw, KP);
  const MixedBody<KP> b{{}, H.col.p, H.vhi.p, diag, x, k, y, ldy, H.perm.p, H.block ? H.xpos.p : nullptr};
  switch (vw) {
    case 32: k_sigma_mixed<32, KP><<<L.blocks, L.threads, 0, s>>>(H.rowptr.p, H.N, b); break;
    case 16: k_sigma_mixed<16, KP><<<L.blocks, L.threads, 0, s>>>(H.rowptr.p, H.N, b); break;
    case 8: k_sigma_mixed<8, KP><<<L.blocks, L.threads, 0, s>>>(H.rowptr.p, H.N, b); break;
    default: k_sigma_mixed<4, KP><<<L.blocks, L.threads, 0, s>>>(H.rowptr.p, H.N, b); break;
  }
  SHCI_LAUNCH_CHECK();
}

void sigma_csr_mixed(const Csr& H, const double* diag, const float* x32, int kp, int k, double* y, size_t ldy,
                     cudaStream_t s) {
  if (!H.vhi.p) throw Error(kErrState, "Hamiltonian has no FP32 values (built for the FP64 path)");
  if (H.N == 0) return;
  const int vw = pick_vw(H);
  if (kp == 1 && H.cvalid) {
    const SigmaLaunch L = sigma_launch(H.N, H.cvw, 1);
    const MixedCompactBody b{{}, H.clo.p, H.chi.p, H.cval.p, diag, x32, y, H.perm.p, H.block ? H.xpos.p : nullptr};
    switch (H.cvw) {  // the width the copy is laid out for
      case 32: k_sigma_compact<32><<<L.blocks, L.threads, 0, s>>>(H.crow.p, H.N, b); break;
      case 16: k_sigma_compact<16><<<L.blocks, L.threads, 0, s>>>(H.crow.p, H.N, b); break;
      case 8: k_sigma_compact<8><<<L.blocks, L.threads, 0, s>>>(H.crow.p, H.N, b); break;
      default: k_sigma_compact<4><<<L.blocks, L.threads, 0, s>>>(H.crow.p, H.N, b); break;
    }
    SHCI_LAUNCH_CHECK();
    return;
  }
  switch (kp) {
    case 1: launch_mixed<1>(vw, H, diag, x32, k, y, ldy, s); break;
    case 2: launch_mixed<2>(vw, H, diag, x32, k, y, ldy, s); break;
    case 4: launch_mixed<4>(vw, H, diag, x32, k, y, ldy, s); break;
    default: throw Error(kErrInvalid, "sigma block width must be 1, 2 or 4");
  }
}

template <int KP>
static void launch_f64(int vw, const Csr& H, const double* diag, const double* x, int k, double* y, size_t ldy,
                       cudaStream_t s) {
  const SigmaLaunch L = sigma_launch(H.N, vw, KP, kF64Threads);
  const F64Body<KP> b{{}, H.col.p, H.v64.p, diag, x, k, y, ldy, H.perm.p, H.block ? H.xpos.p : nullptr};
  switch (vw) {
    case 32: k_sigma_f64<32, KP><<<L.blocks, L.threads, 0, s>>>(H.rowptr.p, H.N, b); break;
    case 16: k_sigma_f64<16, KP><<<L.blocks, L.threads, 0, s>>>(H.rowptr.p, H.N, b); break;
    case 8: k_sigma_f64<8, KP><<<L.blocks, L.threads, 0, s>>>(H.rowptr.p, H.N, b); break;
    default: k_sigma_f64<4, KP><<<L.blocks, L.threads, 0, s>>>(H.rowptr.p, H.N, b); break;
  }
  SHCI_LAUNCH_CHECK();
}

void sigma_csr_f64(const Csr& H, const double* diag, const double* x64, int kp, int k, double* y, size_t ldy,
                   cudaStream_t s) {
  if (H.N == 0) return;
  if (!H.v64.p) throw Error(kErrState, "Hamiltonian has no FP64 values");
  const int vw = pick_vw(H);
  switch (kp) {
    case 1: launch_f64<1>(vw, H, diag, x64, k, y, ldy, s); break;
    case 2: launch_f64<2>(vw, H, diag, x64, k, y, ldy, s); break;
    case 4: launch_f64<4>(vw, H, diag, x64, k, y, ldy, s); break;
    default: throw Error(kErrInvalid, "sigma block width must be 1, 2 or 4");
  }
}

template <int KP>
static void launch_ff(int vw, const Csr& H, const double* diag, const float* xff, const double* xd, size_t ldx, int c0,
                      int k, double* y, size_t ldy, cudaStream_t s) {
  const SigmaLaunch L = sigma_launch(H.N, vw, KP);
  const FFBody<KP> b{{}, H.col.p, H.vhi.p, H.vlo.p, diag, xff, xd, ldx, c0, k, y, ldy, H.perm.p};
  switch (vw) {
    case 32: k_sigma_ff<32, KP><<<L.blocks, L.threads, 0, s>>>(H.rowptr.p, H.N, b); break;
    case 16: k_sigma_ff<16, KP><<<L.blocks, L.threads, 0, s>>>(H.rowptr.p, H.N, b); break;
    case 8: k_sigma_ff<8, KP><<<L.blocks, L.threads, 0, s>>>(H.rowptr.p, H.N, b); break;
    default: k_sigma_ff<4, KP><<<L.blocks, L.threads, 0, s>>>(H.rowptr.p, H.N, b); break;
  }
  SHCI_LAUNCH_CHECK();
}

void sigma_csr_ff(const Csr& H, const double* diag, const float* xff, int kp, const double* xd, size_t ldx, int c0,
                  int k, double* y, size_t ldy, cudaStream_t s) {
  if (H.N == 0) return;
  if (!(H.vhi.p && H.vlo.p)) throw Error(kErrState, "Hamiltonian has no FP32 head/tail values");
  const int vw = pick_vw(H);
  switch (kp) {
    case 1: launch_ff<1>(vw, H, diag, xff, xd, ldx, c0, k, y, ldy, s); break;
    case 2: launch_ff<2>(vw, H, diag, xff, xd, ldx, c0, k, y, ldy, s); break;
    case 4: launch_ff<4>(vw, H, diag, xff, xd, ldx, c0, k, y, ldy, s); break;
    default: throw Error(kErrInvalid, "sigma block width must be 1, 2 or 4");
  }
}

// ---------------------------------------------------------------------------
// Packing between column-major FP64 blocks and row-interleaved vectors
// ---------------------------------------------------------------------------
__global__ void k_pack_f32(const double* __restrict__ A, size_t lda, int c0, int k, int kp, size_t N,
                           float* __restrict__ out, const uint32_t* __restrict__ perm) {
  for (size_t r = (size_t)blockIdx.x * blockDim.x + threadIdx.x; r < N; r += (size_t)gridDim.x * blockDim.x) {
    const size_t src = perm ? (size_t)perm[r] : r;
    for (int c = 0; c < kp; ++c) out[r * kp + c] = c < k ? (float)A[(size_t)(c0 + c) * lda + src] : 0.f;
  }
}
__global__ void k_pack_f64(const double* __restrict__ A, size_t lda, int c0, int k, int kp, size_t N,
                           double* __restrict__ out, const uint32_t* __restrict__ perm) {
  for (size_t r = (size_t)blockIdx.x * blockDim.x + threadIdx.x; r < N; r += (size_t)gridDim.x * blockDim.x) {
    const size_t src = perm ? (size_t)perm[r] : r;
    for (int c = 0; c < kp; ++c) out[r * kp + c] = c < k ? A[(size_t)(c0 + c) * lda + src] : 0.0;
  }
}
__global__ void k_pack_ff(const double* __restrict__ A, size_t lda, int c0, int k, int kp, size_t N,
                          float2* __restrict__ out, const uint32_t* __restrict__ perm) {
  for (size_t r = (size_t)blockIdx.x * blockDim.x + threadIdx.x; r < N; r += (size_t)gridDim.x * blockDim.x)
    for (int c = 0; c < kp; ++c) {
      float2 v = make_float2(0.f, 0.f);
      if (c < k) {
        const double x = A[(size_t)(c0 + c) * lda + (perm ? (size_t)perm[r] : r)];
        v.x = __double2float_rn(x);
        v.y = __double2float_rn(x - (double)v.x);
      }
      out[r * kp + c] = v;
    }
}
void pack_ff(const double* A, size_t lda, int c0, int k, int kp, size_t N, float* out, cudaStream_t s,
             const uint32_t* perm) {
  k_pack_ff<<<grid_for(N, 256), 256, 0, s>>>(A, lda, c0, k, kp, N, reinterpret_cast<float2*>(out), perm);
  SHCI_LAUNCH_CHECK();
}
void pack_f32(const double* A, size_t lda, int c0, int k, int kp, size_t N, float* out, cudaStream_t s,
              const uint32_t* perm) {
  k_pack_f32<<<grid_for(N, 256), 256, 0, s>>>(A, lda, c0, k, kp, N, out, perm);
  SHCI_LAUNCH_CHECK();
}
void pack_f64(const double* A, size_t lda, int c0, int k, int kp, size_t N, double* out, cudaStream_t s,
              const uint32_t* perm) {
  k_pack_f64<<<grid_for(N, 256), 256, 0, s>>>(A, lda, c0, k, kp, N, out, perm);
  SHCI_LAUNCH_CHECK();
}
struct Row32 {
  double2 a, b;
};
template <class T>
__global__ void k_gather_rows(const T* __restrict__ in, const uint32_t* __restrict__ perm, size_t N,
                              T* __restrict__ out) {
  for (size_t r = (size_t)blockIdx.x * blockDim.x + threadIdx.x; r < N; r += (size_t)gridDim.x * blockDim.x)
    out[r] = in[perm[r]];
}
void gather_rows(const void* in, size_t bytes_per_row, const uint32_t* perm, size_t N, void* out, cudaStream_t s) {
  if (N == 0) return;
  const unsigned g = grid_for(N, 256);
  switch (bytes_per_row) {
    case 4: k_gather_rows<float><<<g, 256, 0, s>>>(static_cast<const float*>(in), perm, N, static_cast<float*>(out)); break;
    case 8: k_gather_rows<double><<<g, 256, 0, s>>>(static_cast<const double*>(in), perm, N, static_cast<double*>(out)); break;
    case 16: k_gather_rows<double2><<<g, 256, 0, s>>>(static_cast<const double2*>(in), perm, N, static_cast<double2*>(out)); break;
    case 32: k_gather_rows<Row32><<<g, 256, 0, s>>>(static_cast<const Row32*>(in), perm, N, static_cast<Row32*>(out)); break;
    default: throw Error(kErrInvalid, "gather_rows: row size must be 4, 8, 16 or 32 bytes");
  }
  SHCI_LAUNCH_CHECK();
}
// ---------------------------------------------------------------------------
// Tall-skinny Gram: G = A^T B. Blocks own contiguous row ranges and write
// one partial per block; a second kernel adds the partials in block order, so
// the result does not depend on scheduling.
// Narrow products (ma * mb <= 16: norms, dots, residual norms) keep every
// pair's sum in registers and stream the rows with independent loads; wider
// ones (the Rayleigh matrix) stage 64-row tiles in shared memory with all
// threads of the block splitting the rows of a tile between them.
// ---------------------------------------------------------------------------
constexpr int kGramMax = 16;
constexpr int kGramRows = 64;
constexpr unsigned kGramBlocks = 152 * 2;
constexpr int kGramRegPairs = 16;

__device__ inline void block_sum_pairs(double* acc, int P, double* __restrict__ out) {
  __shared__ double red[8][kGramRegPairs];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
#pragma unroll
  for (int p = 0; p < kGramRegPairs; ++p) {
    if (p >= P) break;
    double v = acc[p];
#pragma unroll
    for (int o = 16; o; o >>= 1) v += __shfl_xor_sync(kFull, v, o);
    if (lane == 0) red[w][p] = v;
  }
  __syncthreads();
  if ((int)threadIdx.x < P) {
    double v = 0.0;
    for (int ww = 0; ww < (int)(blockDim.x >> 5); ++ww) v += red[ww][threadIdx.x];
    out[threadIdx.x] = v;
  }
}

__global__ void __launch_bounds__(256) k_gram_reg(const double* __restrict__ A, size_t lda, int ma,
                                                  const double* __restrict__ B, size_t ldb, int mb, size_t N,
                                                  double* __restrict__ part) {
  double acc[kGramRegPairs];
#pragma unroll
  for (int p = 0; p < kGramRegPairs; ++p) acc[p] = 0.0;
  const int P = ma * mb;
  const size_t per = (N + gridDim.x - 1) / gridDim.x;
  const size_t r0 = (size_t)blockIdx.x * per;
  const size_t r1 = r0 + per < N ? r0 + per : N;
  // repeated loads of one row's entries hit L1; only distinct ones reach L2
  for (size_t r = r0 + threadIdx.x; r < r1; r += blockDim.x) {
#pragma unroll
    for (int p = 0; p < kGramRegPairs; ++p)
      if (p < P) acc[p] += A[(size_t)(p % ma) * lda + r] * B[(size_t)(p / ma) * ldb + r];
  }
  block_sum_pairs(acc, P, part + (size_t)blockIdx.x * P);
}

__global__ void __launch_bounds__(256) k_gram_part(const double* __restrict__ A, size_t lda, int ma,
                                                   const double* __restrict__ B, size_t ldb, int mb, size_t N,
                                                   double* __restrict__ part) {
  __shared__ double sA[kGramMax][kGramRows + 1];
  __shared__ double sB[kGramMax][kGramRows + 1];
  __shared__ double red[256];
  const int t = threadIdx.x;
  const int P = ma * mb;
  const int S = 256 / P;  // threads per pair, splitting the rows of a tile
  const int pp = t % P, q = t / P;
  const int pi = pp % ma, pj = pp / ma;
  const bool active = q < S;
  double acc = 0.0;
  const size_t per = (N + gridDim.x - 1) / gridDim.x;
  const size_t r0 = (size_t)blockIdx.x * per;
  const size_t r1 = r0 + per < N ? r0 + per : N;
  for (size_t base = r0; base < r1; base += kGramRows) {
    for (int e = t; e < ma * kGramRows; e += blockDim.x) {
      const int c = e / kGramRows, rr = e % kGramRows;
      const size_t row = base + rr;
      sA[c][rr] = row < r1 ? A[(size_t)c * lda + row] : 0.0;
    }
    for (int e = t; e < mb * kGramRows; e += blockDim.x) {
      const int c = e / kGramRows, rr = e % kGramRows;
      const size_t row = base + rr;
      sB[c][rr] = row < r1 ? B[(size_t)c * ldb + row] : 0.0;
    }
    __syncthreads();
    if (active)
      for (int rr = q; rr < kGramRows; rr += S) acc += sA[pi][rr] * sB[pj][rr];
    __syncthreads();
  }
  red[t] = active ? acc : 0.0;
  __syncthreads();
  if (t < P) {
    double v = 0.0;
    for (int k = 0; k < S; ++k) v += red[t + k * P];
    part[(size_t)blockIdx.x * P + t] = v;
  }
}

// Sum of the blocks' partials of one value by one warp, lanes over the blocks
// and a fixed tree: independent of scheduling, and the loads are in flight
// together (one thread per value adding 304 partials in turn took 18 us).
__device__ __forceinline__ double sum_partials(const double* part, int nblocks, int P, int p) {
  const int lane = threadIdx.x & 31;
  double s = 0.0;
  for (int b = lane; b < nblocks; b += 32) s += __ldcg(part + (size_t)b * P + p);
#pragma unroll
  for (int o = 16; o; o >>= 1) s += __shfl_xor_sync(kFull, s, o);
  return s;
}
// one warp per value, 8 per block: with two FP64 lanes per clock and SM, the
// warps of one block would wait for one another
__global__ void __launch_bounds__(256) k_gram_sum(const double* __restrict__ part, int nblocks, int P,
                                                  double* __restrict__ G) {
  const int p = blockIdx.x * 8 + (threadIdx.x >> 5);
  if (p >= P) return;
  const double s = sum_partials(part, nblocks, P, p);
  if ((threadIdx.x & 31) == 0) G[p] = s;
}

void ts_gram(const double* A, size_t lda, int ma, const double* B, size_t ldb, int mb, size_t N, double* G,
             DevBuf<double>& part, cudaStream_t s) {
  if (ma < 1 || mb < 1 || ma > kGramMax || mb > kGramMax) throw Error(kErrInvalid, "Gram block too wide");
  unsigned nb = kGramBlocks;
  if ((size_t)nb * kGramRows > N) nb = (unsigned)((N + kGramRows - 1) / kGramRows);
  if (nb < 1) nb = 1;
  part.reserve((size_t)nb * ma * mb);
  if (ma * mb <= kGramRegPairs)
    k_gram_reg<<<nb, 256, 0, s>>>(A, lda, ma, B, ldb, mb, N, part.p);
  else
    k_gram_part<<<nb, 256, 0, s>>>(A, lda, ma, B, ldb, mb, N, part.p);
  SHCI_LAUNCH_CHECK();
  k_gram_sum<<<(ma * mb + 7) / 8, 256, 0, s>>>(part.p, (int)nb, ma * mb, G);
  SHCI_LAUNCH_CHECK();
}

// Y = alpha * A Q + beta * Y. Each thread owns one row; the row's m entries
// stay in registers (loops unrolled to the 16-column maximum and predicated).
__global__ void __launch_bounds__(256) k_ts_gemm(const double* __restrict__ A, size_t lda, int m,
                                                 const double* __restrict__ Q, int k, size_t N, double alpha,
                                                 double beta, double* __restrict__ Y, size_t ldy) {
  __shared__ double sQ[kGramMax * kGramMax];
  for (int e = threadIdx.x; e < m * k; e += blockDim.x) sQ[e] = Q[e];
  __syncthreads();
  for (size_t r = (size_t)blockIdx.x * blockDim.x + threadIdx.x; r < N; r += (size_t)gridDim.x * blockDim.x) {
    double a[kGramMax];
#pragma unroll
    for (int i = 0; i < kGramMax; ++i) a[i] = i < m ? A[(size_t)i * lda + r] : 0.0;
    for (int c = 0; c < k; ++c) {
      double s = 0.0;
#pragma unroll
      for (int i = 0; i < kGramMax; ++i)
        if (i < m) s += a[i] * sQ[c * m + i];
      double* yp = Y + (size_t)c * ldy + r;
      *yp = (beta == 0.0) ? alpha * s : alpha * s + beta * (*yp);
    }
  }
}
void ts_gemm(const double* A, size_t lda, int m, const double* Q, int k, size_t N, double alpha, double beta,
             double* Y, size_t ldy, cudaStream_t s) {
  if (m > kGramMax || k > kGramMax) throw Error(kErrInvalid, "tall-skinny product too wide");
  k_ts_gemm<<<grid_for(N, 256), 256, 0, s>>>(A, lda, m, Q, k, N, alpha, beta, Y, ldy);
  SHCI_LAUNCH_CHECK();
}

__global__ void k_residual(const double* __restrict__ X, const double* __restrict__ Y, const double* __restrict__ lam,
                           int k, size_t N, size_t ld, double* __restrict__ R) {
  for (size_t r = (size_t)blockIdx.x * blockDim.x + threadIdx.x; r < N; r += (size_t)gridDim.x * blockDim.x)
    for (int c = 0; c < k; ++c) R[(size_t)c * ld + r] = Y[(size_t)c * ld + r] - lam[c] * X[(size_t)c * ld + r];
}
void residual(const double* X, const double* Y, const double* lam, int k, size_t N, size_t ld, double* R,
              cudaStream_t s) {
  k_residual<<<grid_for(N, 256), 256, 0, s>>>(X, Y, lam, k, N, ld, R);
  SHCI_LAUNCH_CHECK();
}

// precondition (SHCI/Davidson.cpp:85-106)
__global__ void k_precondition(const double* __restrict__ diag, const double* __restrict__ lam, int k, size_t N,
                               double* __restrict__ R, size_t ld) {
  for (size_t r = (size_t)blockIdx.x * blockDim.x + threadIdx.x; r < N; r += (size_t)gridDim.x * blockDim.x)
    for (int c = 0; c < k; ++c) {
      double e = lam[c], d = diag[r];
      double* p = R + (size_t)c * ld + r;
      if (fabs(e - d) > 1e-12)
        *p = *p / (e - d);
      else
        *p = *p / (e - d - 1.e-12);
    }
}
void precondition(const double* diag, const double* lam, int k, size_t N, double* R, size_t ld, cudaStream_t s) {
  k_precondition<<<grid_for(N, 256), 256, 0, s>>>(diag, lam, k, N, R, ld);
  SHCI_LAUNCH_CHECK();
}

// Shifted preconditioner r_i / (lam - diag_i - shift_i). The plain denominator
// is kept wherever the shifted one changes sign or shrinks below a fifth of it
// (a shift that would blow the correction up), so the learned or second-order
// shift can only refine the reference's denominator, never replace it wholesale.
__global__ void k_precondition_shift(const double* __restrict__ diag, const double* __restrict__ shift,
                                     const double* __restrict__ lam, int k, size_t N, double* __restrict__ R,
                                     size_t ld) {
  for (size_t r = (size_t)blockIdx.x * blockDim.x + threadIdx.x; r < N; r += (size_t)gridDim.x * blockDim.x)
    for (int c = 0; c < k; ++c) {
      const double e = lam[c], d = diag[r];
      double den = e - d;
      const double d2 = den - shift[r];
      if ((d2 > 0) == (den > 0) && fabs(d2) > 0.2 * fabs(den)) den = d2;
      double* p = R + (size_t)c * ld + r;
      if (fabs(den) > 1e-12)
        *p = *p / den;
      else
        *p = *p / (den - 1.e-12);
    }
}
void precondition_shift(const double* diag, const double* shift, const double* lam, int k, size_t N, double* R,
                        size_t ld, cudaStream_t s) {
  k_precondition_shift<<<grid_for(N, 256), 256, 0, s>>>(diag, shift, lam, k, N, R, ld);
  SHCI_LAUNCH_CHECK();
}

__global__ void k_scale_inv_norm(double* __restrict__ c, size_t N, const double* __restrict__ g) {
  const double nrm = sqrt(g[0]);
  if (!(nrm > 1e-14)) return;  // linearly dependent: left for the host to drop
  const double sc = 1.0 / nrm;
  for (size_t r = (size_t)blockIdx.x * blockDim.x + threadIdx.x; r < N; r += (size_t)gridDim.x * blockDim.x)
    c[r] *= sc;
}
void scale_inv_norm(double* c, size_t N, const double* g, cudaStream_t s) {
  k_scale_inv_norm<<<grid_for(N, 256), 256, 0, s>>>(c, N, g);
  SHCI_LAUNCH_CHECK();
}

// ---------------------------------------------------------------------------
// The Davidson iteration's passes over the basis. The basis is small beside
// the matrix, so what bounds them at ordinary sizes is the number of launches
// and, in each, the FP64 pipe (two lanes per clock and SM: a warp-wide add
// occupies it for 16 clocks), not memory. So every pass does all that one
// reading of V and W allows, sums are reduced by exchanging halves (M - 1 + 5 -
// log2 M adds per lane for M sums instead of 5 M), and the last block to
// finish adds the blocks' partials, in block order, instead of a second launch.
// 81,233 determinants, basis of at most 5: an iteration's vector work, 25
// launches and 8 copies, took 180 us (gram sums 92, products 36, Gram parts 27);
// now five launches, 55 us, the FP64 pipe 32 to 47 % busy and 13 % of the warp slots
// in use: the rest is the latency of loads, shuffles and barriers.
//
// The small matrices are read from and written to pinned host memory (Q, the
// eigenvalues, the norms, the new column of the Rayleigh matrix): a few hundred
// bytes per pass, without copy nodes between the kernels.
// ---------------------------------------------------------------------------
// Sums over the grid of M values per thread; `part` holds gridDim.x * M
// doubles, *count is 0 before and after. Value p goes to out[p * ostride] and,
// if given, to dev[p] (p < n).
template <int M>
__device__ __forceinline__ void grid_sums(double (&v)[M], int n, double* __restrict__ part,
                                          unsigned* __restrict__ count, double* out, int ostride, double* dev) {
  __shared__ double s_w[32][M];
  __shared__ bool s_last;
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, nw = blockDim.x >> 5;
  int idx = 0, o = 16;
#pragma unroll
  for (int half = M / 2; half >= 1; half >>= 1, o >>= 1) {
    const bool up = (lane & o) != 0;
#pragma unroll
    for (int k = 0; k < half; ++k) {
      const double keep = up ? v[k + half] : v[k], send = up ? v[k] : v[k + half];
      v[k] = keep + __shfl_xor_sync(kFull, send, o);
    }
    idx += up ? half : 0;
  }
  for (int q = o; q; q >>= 1) v[0] += __shfl_xor_sync(kFull, v[0], q);
  if ((lane & (o ? 2 * o - 1 : 0)) == 0) s_w[w][idx] = v[0];  // one lane of the group that holds value idx
  __syncthreads();
  if ((int)threadIdx.x < n) {
    double s = 0.0;
    for (int k = 0; k < nw; ++k) s += s_w[k][threadIdx.x];
    __stcg(part + (size_t)blockIdx.x * n + threadIdx.x, s);
    __threadfence();
  }
  __syncthreads();
  if (threadIdx.x == 0) s_last = atomicAdd(count, 1u) == gridDim.x - 1;
  __syncthreads();
  if (!s_last) return;
  __threadfence();
  for (int p = w; p < n; p += nw) {
    const double s = sum_partials(part, (int)gridDim.x, n, p);
    if (lane == 0) {
      if (out) out[p * ostride] = s;
      if (dev) dev[p] = s;
    }
  }
  if (threadIdx.x == 0) *count = 0u;
}

// Two rows a thread before more blocks: half the warps, so half the reductions
// on an SM's FP64 pipe; large spaces fill the SMs with four blocks each.
constexpr int kDavThreads = 256;
constexpr unsigned kDavBlocks = 152 * 4;
static unsigned dav_blocks(size_t N) {
  const size_t b = (N + 2 * kDavThreads - 1) / (2 * kDavThreads);
  return (unsigned)(b < 1 ? 1 : (b > kDavBlocks ? kDavBlocks : b));
}
size_t dav_scratch() { return (size_t)kDavBlocks * (kGramMax + 1); }

// X = V Q, Y = W Q, R = Y - X diag(lam) (written where asked for), |R_c|^2.
template <int M, int NR>
__global__ void __launch_bounds__(kDavThreads) k_ritz(const double* __restrict__ V, const double* __restrict__ W,
                                                      size_t ld, int m, const double* Q, const double* lam, int nroots,
                                                      size_t N, double* __restrict__ X, double* __restrict__ Y,
                                                      double* __restrict__ R, double* __restrict__ part,
                                                      unsigned* __restrict__ count, double* rr) {
  __shared__ double sQ[kGramMax * kGramMax], sL[kGramMax];
  for (int e = threadIdx.x; e < m * nroots; e += blockDim.x) sQ[e] = Q[e];
  for (int e = threadIdx.x; e < nroots; e += blockDim.x) sL[e] = lam[e];
  __syncthreads();
  double acc[NR];
#pragma unroll
  for (int c = 0; c < NR; ++c) acc[c] = 0.0;
  for (size_t r = (size_t)blockIdx.x * blockDim.x + threadIdx.x; r < N; r += (size_t)gridDim.x * blockDim.x) {
    double v[M], w[M];
#pragma unroll
    for (int i = 0; i < M; ++i) {
      v[i] = i < m ? V[(size_t)i * ld + r] : 0.0;
      w[i] = i < m ? W[(size_t)i * ld + r] : 0.0;
    }
#pragma unroll
    for (int c = 0; c < NR; ++c) {
      if (c >= nroots) break;
      double x = 0.0, y = 0.0;
#pragma unroll
      for (int i = 0; i < M; ++i)
        if (i < m) {
          x += v[i] * sQ[c * m + i];
          y += w[i] * sQ[c * m + i];
        }
      const double t = y - sL[c] * x;
      X[(size_t)c * ld + r] = x;
      Y[(size_t)c * ld + r] = y;
      if (R) R[(size_t)c * ld + r] = t;
      acc[c] += t * t;
    }
  }
  grid_sums<NR>(acc, nroots, part, count, rr, nroots + 1, nullptr);
}
void dav_ritz(const double* V, const double* W, size_t ld, int m, const double* Q, const double* lam, int nroots,
              size_t N, double* X, double* Y, double* R, const DavWork& w, double* rr, cudaStream_t s) {
  if (m > kGramMax || nroots > kGramMax) throw Error(kErrInvalid, "tall-skinny product too wide");
  const unsigned nb = dav_blocks(N);
#define SHCI_RITZ(M, NR) \
  k_ritz<M, NR><<<nb, kDavThreads, 0, s>>>(V, W, ld, m, Q, lam, nroots, N, X, Y, R, w.part, w.count, rr)
  if (m <= 8) {
    if (nroots == 1) SHCI_RITZ(8, 1); else if (nroots <= 4) SHCI_RITZ(8, 4); else SHCI_RITZ(8, 16);
  } else {
    if (nroots == 1) SHCI_RITZ(16, 1); else if (nroots <= 4) SHCI_RITZ(16, 4); else SHCI_RITZ(16, 16);
  }
#undef SHCI_RITZ
  SHCI_LAUNCH_CHECK();
}

// One preconditioned residual entry (k_residual, then k_precondition or
// k_precondition_shift).
__device__ __forceinline__ double corrected(const double* __restrict__ X, const double* __restrict__ Y, double lam,
                                            const double* __restrict__ diag, const double* __restrict__ shift,
                                            size_t r) {
  const double t = Y[r] - lam * X[r];
  double den = lam - diag[r];
  if (shift) {
    const double d2 = den - shift[r];
    if ((d2 > 0) == (den > 0) && fabs(d2) > 0.2 * fabs(den)) den = d2;
  }
  return fabs(den) > 1e-12 ? t / den : t / (den - 1.e-12);
}

// D = the preconditioned residual of one root (projected into the flip sector
// p when flip is given), G = V^T D.
template <int M>
__global__ void __launch_bounds__(kDavThreads) k_dav_correct(const double* __restrict__ V, size_t ld, int m,
                                                             const double* __restrict__ X,
                                                             const double* __restrict__ Y, const double* lam,
                                                             const double* __restrict__ diag,
                                                             const double* __restrict__ shift,
                                                             const int32_t* __restrict__ flip,
                                                             const int8_t* __restrict__ sign, double p, size_t N,
                                                             double* __restrict__ D, double* __restrict__ part,
                                                             unsigned* __restrict__ count, double* __restrict__ G) {
  __shared__ double sl;
  if (threadIdx.x == 0) sl = *lam;
  __syncthreads();
  const double l = sl;
  double acc[M];
#pragma unroll
  for (int i = 0; i < M; ++i) acc[i] = 0.0;
  for (size_t r = (size_t)blockIdx.x * blockDim.x + threadIdx.x; r < N; r += (size_t)gridDim.x * blockDim.x) {
    double d = corrected(X, Y, l, diag, shift, r);
    if (flip) d = 0.5 * (d + p * (double)sign[r] * corrected(X, Y, l, diag, shift, (size_t)flip[r]));
    D[r] = d;
#pragma unroll
    for (int i = 0; i < M; ++i)
      if (i < m) acc[i] += V[(size_t)i * ld + r] * d;
  }
  grid_sums<M>(acc, m, part, count, nullptr, 0, G);
}
// D -= V g, then G = V^T D and G[m] = |D|^2.
template <int M>
__global__ void __launch_bounds__(kDavThreads) k_dav_project(const double* __restrict__ V, size_t ld, int m,
                                                             const double* __restrict__ g, size_t N,
                                                             double* __restrict__ D, double* __restrict__ part,
                                                             unsigned* __restrict__ count, double* __restrict__ G) {
  __shared__ double sg[M];
  if ((int)threadIdx.x < m) sg[threadIdx.x] = g[threadIdx.x];
  __syncthreads();
  double acc[2 * M];  // the reduction takes a power of two
#pragma unroll
  for (int i = 0; i < 2 * M; ++i) acc[i] = 0.0;
  for (size_t r = (size_t)blockIdx.x * blockDim.x + threadIdx.x; r < N; r += (size_t)gridDim.x * blockDim.x) {
    double v[M], t = 0.0;
#pragma unroll
    for (int i = 0; i < M; ++i) v[i] = i < m ? V[(size_t)i * ld + r] : 0.0;
#pragma unroll
    for (int i = 0; i < M; ++i)
      if (i < m) t += v[i] * sg[i];
    const double d = D[r] - t;
    D[r] = d;
#pragma unroll
    for (int i = 0; i <= M; ++i)
      if (i < m)
        acc[i] += v[i] * d;
      else if (i == m)
        acc[i] += d * d;
  }
  if (m < M) {
    double low[M];
#pragma unroll
    for (int i = 0; i < M; ++i) low[i] = acc[i];
    grid_sums<M>(low, m + 1, part, count, nullptr, 0, G);
  } else {
    grid_sums<2 * M>(acc, m + 1, part, count, nullptr, 0, G);
  }
}
// The second Gram-Schmidt projection, the normalisation and the append in one
// pass, with the rotation of V and W when the basis collapses (Q given: keep
// columns; in place, every thread owns its row): V[:, at] = (D - V g) / |D - V g|.
// |D - V g|^2 = |D|^2 - |g|^2, V being orthonormal, while g is small beside D
// (a rounding residue, as a rule; a hundredth of D leaves the difference 15
// digits). Where it is not, the first projection left little but rounding: the
// difference has no digits, so D - V g is appended as it is and the norm given as
// -1, for the host to measure it. A dependent D (norm below 1e-14) is left for the
// host to drop.
template <int M>
__global__ void __launch_bounds__(256) k_dav_append(double* __restrict__ V, double* __restrict__ W, size_t ld, int m,
                                                    const double* __restrict__ g, size_t N,
                                                    const double* __restrict__ D, const double* Q, int keep, int at,
                                                    double* nrm, double* nrm_out) {
  __shared__ double sQ[kGramMax * kGramMax];
  __shared__ double sg[M], s_sc;
  if (Q)
    for (int e = threadIdx.x; e < m * keep; e += blockDim.x) sQ[e] = Q[e];
  if ((int)threadIdx.x < m) sg[threadIdx.x] = g[threadIdx.x];
  __syncthreads();
  if (threadIdx.x == 0) {  // one thread's square root and division, not every thread's
    const double d2 = g[m];
    double n2 = d2;
    for (int i = 0; i < m; ++i) n2 -= sg[i] * sg[i];
    if (!(n2 >= 0.9999 * d2)) n2 = -1.0;
    const double n = sqrt(n2);
    s_sc = n > 1e-14 ? 1.0 / n : 1.0;
    if (blockIdx.x == 0) {
      *nrm = n2;
      *nrm_out = n2;
    }
  }
  __syncthreads();
  const double sc = s_sc;
  for (size_t r = (size_t)blockIdx.x * blockDim.x + threadIdx.x; r < N; r += (size_t)gridDim.x * blockDim.x) {
    double v[M], t = 0.0;
#pragma unroll
    for (int i = 0; i < M; ++i) v[i] = i < m ? V[(size_t)i * ld + r] : 0.0;
#pragma unroll
    for (int i = 0; i < M; ++i)
      if (i < m) t += v[i] * sg[i];
    const double d = (D[r] - t) * sc;
    if (Q) {
      double w[M];
#pragma unroll
      for (int i = 0; i < M; ++i) w[i] = i < m ? W[(size_t)i * ld + r] : 0.0;
      for (int c = 0; c < keep; ++c) {
        double x = 0.0, y = 0.0;
#pragma unroll
        for (int i = 0; i < M; ++i)
          if (i < m) {
            x += v[i] * sQ[c * m + i];
            y += w[i] * sQ[c * m + i];
          }
        V[(size_t)c * ld + r] = x;
        W[(size_t)c * ld + r] = y;
      }
    }
    V[(size_t)at * ld + r] = d;
  }
}
void dav_correction(double* V, double* W, size_t ld, int m, const double* X, const double* Y, const double* lam,
                    const double* diag, const double* shift, const int32_t* flip, const int8_t* sign, double p,
                    size_t N, double* D, const DavWork& w, double* g1, double* g2, const double* Q, int keep, int at,
                    double* nrm, double* nrm_out, cudaStream_t s) {
  if (m > kGramMax || keep > m) throw Error(kErrInvalid, "Gram block too wide");
  const unsigned nb = dav_blocks(N);
#define SHCI_CORR(M)                                                                                                 \
  k_dav_correct<M><<<nb, kDavThreads, 0, s>>>(V, ld, m, X, Y, lam, diag, shift, flip, sign, p, N, D, w.part, w.count, \
                                              g1);                                                                   \
  SHCI_LAUNCH_CHECK();                                                                                               \
  k_dav_project<M><<<nb, kDavThreads, 0, s>>>(V, ld, m, g1, N, D, w.part, w.count, g2);                              \
  SHCI_LAUNCH_CHECK();                                                                                               \
  k_dav_append<M><<<grid_for(N, 256), 256, 0, s>>>(V, W, ld, m, g2, N, D, Q, keep, at, nrm, nrm_out);                \
  SHCI_LAUNCH_CHECK()
  if (m <= 8) {
    SHCI_CORR(8);
  } else {
    SHCI_CORR(16);
  }
#undef SHCI_CORR
}

// out[i] = V_i . w for the m columns of V (pinned host memory)
template <int M>
__global__ void __launch_bounds__(kDavThreads) k_dav_column(const double* __restrict__ V, size_t ld, int m,
                                                            const double* __restrict__ w, size_t N,
                                                            double* __restrict__ part, unsigned* __restrict__ count,
                                                            double* out) {
  double acc[M];
#pragma unroll
  for (int i = 0; i < M; ++i) acc[i] = 0.0;
  for (size_t r = (size_t)blockIdx.x * blockDim.x + threadIdx.x; r < N; r += (size_t)gridDim.x * blockDim.x) {
    const double x = w[r];
#pragma unroll
    for (int i = 0; i < M; ++i)
      if (i < m) acc[i] += V[(size_t)i * ld + r] * x;
  }
  grid_sums<M>(acc, m, part, count, out, 1, nullptr);
}
void dav_column(const double* V, size_t ld, int m, const double* w, size_t N, const DavWork& wk, double* out,
                cudaStream_t s) {
  if (m > kGramMax) throw Error(kErrInvalid, "Gram block too wide");
  const unsigned nb = dav_blocks(N);
  if (m <= 8)
    k_dav_column<8><<<nb, kDavThreads, 0, s>>>(V, ld, m, w, N, wk.part, wk.count, out);
  else
    k_dav_column<16><<<nb, kDavThreads, 0, s>>>(V, ld, m, w, N, wk.part, wk.count, out);
  SHCI_LAUNCH_CHECK();
}

// V <- V Q, W <- W Q in place (m columns to keep <= m): every thread owns its
// row, so no second copy of the basis is needed.
__global__ void __launch_bounds__(256) k_dav_collapse(double* __restrict__ V, double* __restrict__ W, size_t ld, int m,
                                                      const double* Q, int keep, size_t N) {
  __shared__ double sQ[kGramMax * kGramMax];
  for (int e = threadIdx.x; e < m * keep; e += blockDim.x) sQ[e] = Q[e];
  __syncthreads();
  for (size_t t = (size_t)blockIdx.x * blockDim.x + threadIdx.x; t < 2 * N; t += (size_t)gridDim.x * blockDim.x) {
    double* A = t < N ? V : W;
    const size_t r = t < N ? t : t - N;
    double a[kGramMax];
#pragma unroll
    for (int i = 0; i < kGramMax; ++i) a[i] = i < m ? A[(size_t)i * ld + r] : 0.0;
    for (int c = 0; c < keep; ++c) {
      double x = 0.0;
#pragma unroll
      for (int i = 0; i < kGramMax; ++i)
        if (i < m) x += a[i] * sQ[c * m + i];
      A[(size_t)c * ld + r] = x;
    }
  }
}
void dav_collapse(double* V, double* W, size_t ld, int m, const double* Q, int keep, size_t N, cudaStream_t s) {
  if (m > kGramMax || keep > m) throw Error(kErrInvalid, "tall-skinny product too wide");
  k_dav_collapse<<<grid_for(2 * N, 256), 256, 0, s>>>(V, W, ld, m, Q, keep, N);
  SHCI_LAUNCH_CHECK();
}

__global__ void k_scale_cols(double* __restrict__ A, size_t ld, const double* __restrict__ sc, int k, size_t N) {
  for (size_t r = (size_t)blockIdx.x * blockDim.x + threadIdx.x; r < N; r += (size_t)gridDim.x * blockDim.x)
    for (int c = 0; c < k; ++c) A[(size_t)c * ld + r] *= sc[c];
}
void scale_cols(double* A, size_t ld, const double* scale, int k, size_t N, cudaStream_t s) {
  k_scale_cols<<<grid_for(N, 256), 256, 0, s>>>(A, ld, scale, k, N);
  SHCI_LAUNCH_CHECK();
}

// ---------------------------------------------------------------------------
// Allocation-free sigma (shci_sigma_device_noalloc). The row-interleaved copy
// of x that the sigma kernels gather from lives in this fixed device array
// instead of a context buffer, so a call never allocates. Every GPU that loads
// the library holds the array until the process exits. All calls share it and
// each call overwrites the part it uses (including the zero padding), so
// nothing has to be cleared between calls; calls that overlap on the GPU
// (different streams or contexts at the same time) race on it.
// ---------------------------------------------------------------------------
static __device__ __align__(256) unsigned char g_sigma_pack_scratch[kNoAllocPackBytes];

// Device address of the array on the current device. Host code cannot use
// the symbol itself: on the host it names a stand-in, not device memory. The
// context calls this while it builds a stored Hamiltonian (a call that may
// allocate and load this file's kernels), so the allocation-free sigma itself
// only reads the address the context kept.
void* noalloc_scratch_address() {
  void* p = nullptr;
  const cudaError_t e = cudaGetSymbolAddress(&p, g_sigma_pack_scratch);
  if (e != cudaSuccess) {
    cudaGetLastError();
    throw Error(kErrCuda, std::string("cudaGetSymbolAddress(scratch): ") + cudaGetErrorString(e));
  }
  return p;
}

void sigma_noalloc(const Csr& H, const double* diag, int mode_mixed, const double* x, size_t ldx, int k, double* y,
                   size_t ldy, void* scratch, cudaStream_t s) {
  const size_t N = H.N;
  const int kp = k == 3 ? 4 : k;
  const size_t need = N * (size_t)kp * (mode_mixed ? sizeof(float) : sizeof(double));
  if (need > kNoAllocPackBytes)
    throw Error(kErrInvalid, "allocation-free sigma: N x k = " + std::to_string(N) + " x " + std::to_string(kp) +
                                 " needs " + std::to_string(need) + " bytes of scratch, the fixed maximum is " +
                                 std::to_string(kNoAllocPackBytes));
  if (!scratch) throw Error(kErrState, "allocation-free sigma: scratch address not set up (build the Hamiltonian)");
  if (mode_mixed) {
    pack_f32(x, ldx, 0, k, kp, N, static_cast<float*>(scratch), s, H.perm.p);
    sigma_csr_mixed(H, diag, static_cast<const float*>(scratch), kp, k, y, ldy, s);
  } else {
    if (H.v64.p) {
      pack_f64(x, ldx, 0, k, kp, N, static_cast<double*>(scratch), s, H.perm.p);
      sigma_csr_f64(H, diag, static_cast<const double*>(scratch), kp, k, y, ldy, s);
    } else {  // head + tail values: float-float refinement sigma (same 8 bytes per entry)
      pack_ff(x, ldx, 0, k, kp, N, static_cast<float*>(scratch), s, H.perm.p);
      sigma_csr_ff(H, diag, static_cast<const float*>(scratch), kp, x, ldx, 0, k, y, ldy, s);
    }
  }
}

}  // namespace shci
