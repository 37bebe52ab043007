// Hamiltonian-side kernels of the variational loop:
//   * alpha/beta string tables and single-excitation neighbour lists
//     (replaces HamHelpers2::PopulateHelpers, SHCI/SHCImakeHamiltonian.cpp:184-408);
//   * the diagonal energies (Determinant::Energy at SHCI/SHCIbasics.cpp:1145-1154);
//   * the two-pass count/emit build of the sparse Hamiltonian as full-row CSR
//     (replaces MakeHfromSMHelpers2, SHCI/SHCImakeHamiltonian.cpp:486-715);
//   * the matrix-free sigma (replaces HmultDirect::operator(), SHCI/Hmult.h:241-381).
//
// One warp enumerates the connections of one row I = (A, B), in four parts:
//   1. determinants sharing I's alpha string: beta distance 1 or 2 (scan of
//      the alpha group);
//   2. determinants whose alpha string As is a single excitation of A and
//      whose beta string equals B or is one excitation away:
//      2a. groups As of at most a few times |B| determinants are scanned;
//      2b. in the others every such J contains the partial string B - b for
//          some occupied b of B, so it is found by looking up the keys
//          (As, B - b) in the partial-string index (a hash table per alpha
//          group As gives each key's run of entries): |B| probes per group
//          that return (nearly) only connections;
//   3. determinants sharing I's beta string: alpha distance 2 (scan of the
//      beta group).
// This visits the same (I, J) set as the reference's five helper-list classes
// (single alpha, alpha-beta, single beta, double beta, double alpha).
//
// The tables are in storage order, the order of the matrix's rows and columns,
// so a scan's hits are column indices in ascending order: each part is emitted
// as one ascending run and a row is finished by merging four runs, not sorted.
#include <algorithm>
#include <type_traits>

#include "engine.h"
#include "ham.h"

namespace shci {

static inline unsigned grid_for(size_t n, int threads, size_t max_blocks = 152 * 64) {
  size_t b = (n + threads - 1) / threads;
  if (b < 1) b = 1;
  if (b > max_blocks) b = max_blocks;
  return (unsigned)b;
}

// ---------------------------------------------------------------------------
// Strings and groups
// ---------------------------------------------------------------------------
__global__ void k_strings(const Det2* __restrict__ dets, size_t n, uint64_t* __restrict__ a,
                          uint64_t* __restrict__ b, uint32_t* __restrict__ idx) {
  for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) {
    const Det2 d = dets[i];
    a[i] = det_alpha(d);
    b[i] = det_beta(d);
    idx[i] = (uint32_t)i;
  }
}

__global__ void k_group_flags(const uint64_t* __restrict__ key, size_t n, int64_t* __restrict__ flag) {
  for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x)
    flag[i] = (i == 0 || key[i] != key[i - 1]) ? 1 : 0;
}

// Groups of equal keys: excl + flag - 1 is an entry's group; writes the group's
// start and key and the group of every position (entry p is position pos[p],
// or p).
__global__ void k_group_fill(const uint64_t* __restrict__ key, const uint32_t* __restrict__ pos, size_t n,
                             const int64_t* __restrict__ flag, const int64_t* __restrict__ excl,
                             uint64_t* __restrict__ ukey, int64_t* __restrict__ start, uint32_t* __restrict__ grp) {
  for (size_t p = (size_t)blockIdx.x * blockDim.x + threadIdx.x; p < n; p += (size_t)gridDim.x * blockDim.x) {
    const int64_t seg = excl[p] + flag[p] - 1;
    if (flag[p]) {
      if (ukey) ukey[seg] = key[p];
      start[seg] = (int64_t)p;
    }
    grp[pos ? pos[p] : (uint32_t)p] = (uint32_t)seg;
  }
}
template <class S>
__global__ void k_pair_strings(const uint64_t* __restrict__ a, const uint64_t* __restrict__ b,
                               const uint32_t* __restrict__ perm, size_t n, typename StrPair<S>::T* __restrict__ str,
                               S* __restrict__ bstr, uint32_t* __restrict__ spos, uint32_t* __restrict__ bpos) {
  for (size_t p = (size_t)blockIdx.x * blockDim.x + threadIdx.x; p < n; p += (size_t)gridDim.x * blockDim.x) {
    str[p] = {(S)a[p], (S)b[p]};
    bstr[p] = (S)b[p];
    spos[perm[p]] = (uint32_t)p;
    bpos[p] = (uint32_t)p;
  }
}
template <class S>
__global__ void k_gather_alpha(const typename StrPair<S>::T* __restrict__ str, const uint32_t* __restrict__ pos,
                               size_t n, S* __restrict__ out) {
  for (size_t q = (size_t)blockIdx.x * blockDim.x + threadIdx.x; q < n; q += (size_t)gridDim.x * blockDim.x)
    out[q] = str[pos[q]].x;
}

__device__ __forceinline__ int64_t bsearch_u64(const uint64_t* __restrict__ a, int64_t n, uint64_t x) {
  int64_t lo = 0, hi = n;
  while (lo < hi) {
    int64_t mid = (lo + hi) >> 1;
    uint64_t v = a[mid];
    if (v < x)
      lo = mid + 1;
    else
      hi = mid;
  }
  return (lo < n && a[lo] == x) ? lo : -1;
}

// Single-excitation neighbours of every unique alpha string among the present
// alpha strings (SinglesFromAlpha, SHCI/SHCImakeHamiltonian.cpp:237-252).
// Warp per string; lanes over (occupied i, empty a) pairs.
template <bool kEmit>
__global__ void k_alpha_singles(const uint64_t* __restrict__ ua, int64_t na, int norb, int64_t* __restrict__ counts,
                                const int64_t* __restrict__ offs, uint32_t* __restrict__ out) {
  const int lane = threadIdx.x & 31;
  const int64_t warps = (int64_t)gridDim.x * (blockDim.x >> 5);
  for (int64_t s = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5; s < na; s += warps) {
    const uint64_t x = ua[s];
    const int nocc = __popcll(x);
    const int nvir = norb - nocc;
    const int total = nocc * nvir;
    int64_t cnt = 0;
    int64_t pos = kEmit ? offs[s] : 0;
    for (int base = 0; base < total; base += 32) {
      int q = base + lane;
      bool hit = false;
      int64_t idx = -1;
      if (q < total) {
        int oi = q / nvir, va = q % nvir;
        // oi-th set bit and va-th clear bit (below norb)
        uint64_t occ = x, vir = (~x) & (norb == 64 ? ~0ull : ((1ull << norb) - 1ull));
        for (int t = 0; t < oi; ++t) occ &= occ - 1;
        for (int t = 0; t < va; ++t) vir &= vir - 1;
        int i = __ffsll((long long)occ) - 1, a = __ffsll((long long)vir) - 1;
        uint64_t y = (x ^ (1ull << i)) | (1ull << a);
        idx = bsearch_u64(ua, na, y);
        hit = idx >= 0;
      }
      unsigned m = __ballot_sync(kFull, hit);
      if (kEmit && hit) out[pos + __popc(m & ((1u << lane) - 1u))] = (uint32_t)idx;
      pos += __popc(m);
      cnt += __popc(m);
    }
    if (!kEmit && lane == 0) counts[s] = cnt;
  }
}

__global__ void k_iota_last(int64_t* start, int64_t n_groups, int64_t n_total) { start[n_groups] = n_total; }

// Partial-string index entries, sorted by (alpha group, partial beta string):
// the entries of one key are one run and the runs of one alpha group are
// contiguous, and so are the slots of the group's hash table, so the probes
// of rows of the same alpha string touch the same small regions.
constexpr uint32_t kM1GroupBits = 26;

template <class S>
__global__ void k_m1_count(const S* __restrict__ bstr, size_t n, int64_t* __restrict__ cnt) {
  for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x)
    cnt[i] = bit_count(bstr[i]);
}
// (index entries refer to their determinant by storage position)
template <class S>
__global__ void k_m1_fill(const S* __restrict__ bstr, const uint32_t* __restrict__ agrp, size_t n,
                          const int64_t* __restrict__ off, uint64_t* __restrict__ key, uint32_t* __restrict__ perm,
                          uint4* __restrict__ ent) {
  for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) {
    const uint64_t B = bstr[i];
    const uint32_t g = agrp[i];
    int64_t q = off[i];
    for (uint64_t r = B; r; r &= r - 1) {
      const int b = __ffsll((long long)r) - 1;
      const uint64_t bm = B ^ (1ull << b);
      key[q] = bm;
      perm[q] = (uint32_t)q;
      ent[q] = make_uint4((uint32_t)bm, (uint32_t)(bm >> 32), g | ((uint32_t)b << kM1GroupBits), (uint32_t)i);
      ++q;
    }
  }
}
__global__ void k_m1_group_keys(const uint4* __restrict__ ent, const uint32_t* __restrict__ perm, int64_t n,
                                uint64_t* __restrict__ gk) {
  const uint32_t mask = (1u << kM1GroupBits) - 1u;
  for (int64_t k = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; k < n; k += (int64_t)gridDim.x * blockDim.x)
    gk[k] = ent[perm[k]].z & mask;
}
__global__ void k_m1_permute(const uint4* __restrict__ src, const uint32_t* __restrict__ perm, int64_t n,
                             uint4* __restrict__ dst) {
  for (int64_t k = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; k < n; k += (int64_t)gridDim.x * blockDim.x)
    dst[k] = src[perm[k]];
}
// Per-group hash tables over the index's distinct keys. Entry k starts a run
// when its key (alpha group, partial string) differs from entry k-1's.
__device__ __forceinline__ bool m1_same_key(const uint4& a, const uint4& b) {
  constexpr uint32_t gmask = (1u << kM1GroupBits) - 1u;
  return a.x == b.x && a.y == b.y && ((a.z ^ b.z) & gmask) == 0;
}
// Fibonacci hashing: the top lg bits of the partial string times 2^64 / phi
// pick the slot; 26 bits of a second product are the slot's fingerprint
__device__ __forceinline__ uint32_t m1_slot(uint64_t bm, unsigned lg) {
  return (uint32_t)((bm * 0x9e3779b97f4a7c15ull) >> (64u - lg));
}
__device__ __forceinline__ uint32_t m1_slot(uint32_t bm, unsigned lg) { return (bm * 0x9e3779b9u) >> (32u - lg); }
__device__ __forceinline__ uint32_t m1_fingerprint(uint64_t bm) {
  return (uint32_t)((bm * 0xc2b2ae3d27d4eb4full) >> 38);
}
__device__ __forceinline__ uint32_t m1_fingerprint(uint32_t bm) { return (bm * 0xc2b2ae3du) >> 6; }
constexpr uint32_t kM1Empty = 0xffffffffu;
// The entries of one group are contiguous, and the largest group holds a tenth
// of them: a warp's heads of one group are added at once (400,000 determinants:
// 640 us with one atomic per head).
__global__ void k_m1_heads(const uint4* __restrict__ ent, int64_t n, uint32_t* __restrict__ keys_of_group) {
  constexpr uint32_t gmask = (1u << kM1GroupBits) - 1u;
  const int lane = threadIdx.x & 31;
  const int64_t stride = (int64_t)gridDim.x * blockDim.x;
  for (int64_t base = (int64_t)blockIdx.x * blockDim.x + threadIdx.x - lane; base < n; base += stride) {
    const int64_t k = base + lane;
    bool head = false;
    uint32_t g = 0xffffffffu;
    if (k < n) {
      const uint4 e = ent[k];
      g = e.z & gmask;
      head = k == 0 || !m1_same_key(e, ent[k - 1]);
    }
    const unsigned peers = __match_any_sync(kFull, g);
    const unsigned heads = __ballot_sync(kFull, head);
    if (k < n && lane == __ffs(peers) - 1 && (heads & peers)) atomicAdd(keys_of_group + g, (uint32_t)__popc(heads & peers));
  }
}
// slots of group g: the power of two >= 2 x its distinct keys, at least 2
__global__ void k_m1_slots(const uint32_t* __restrict__ keys_of_group, int64_t ng, int64_t* __restrict__ slots) {
  for (int64_t g = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; g < ng; g += (int64_t)gridDim.x * blockDim.x) {
    int64_t t = 2;
    while (t < 2 * (int64_t)keys_of_group[g]) t <<= 1;
    slots[g] = t;
  }
}
__global__ void k_m1_dir(const int64_t* __restrict__ slots, const int64_t* __restrict__ first, int64_t ng,
                         uint64_t* __restrict__ dir) {
  for (int64_t g = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; g < ng; g += (int64_t)gridDim.x * blockDim.x)
    dir[g] = ((uint64_t)first[g] << 6) | (uint64_t)(63 - __clzll((long long)slots[g]));
}
// One thread per run: measure the run and claim a slot of its group's table
// by linear probing; a table more than half empty always has a free slot. A
// run of distinct determinants has at most 64 entries, one per beta orbital
// outside the partial string. *too_long is set where repeated determinants make
// one longer than a slot can say.
template <class S>
__global__ void k_m1_insert(const uint4* __restrict__ ent, int64_t n, const uint64_t* __restrict__ dir,
                            uint2* __restrict__ tab, uint32_t* __restrict__ too_long) {
  constexpr uint32_t gmask = (1u << kM1GroupBits) - 1u;
  for (int64_t k = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; k < n; k += (int64_t)gridDim.x * blockDim.x) {
    const uint4 e = ent[k];
    if (k > 0 && m1_same_key(e, ent[k - 1])) continue;
    int64_t f = k + 1;
    while (f < n && m1_same_key(ent[f], e)) ++f;
    if (f - k > 64) *too_long = 1u;
    const uint64_t d = dir[e.z & gmask];
    const unsigned lg = (unsigned)(d & 63);
    const uint64_t mask = (1ull << lg) - 1;
    uint2* t = tab + (d >> 6);
    const S bm = (S)(((uint64_t)e.y << 32) | e.x);
    uint64_t q = m1_slot(bm, lg);
    for (uint64_t step = 0; step <= mask; ++step) {
      if (atomicCAS(&t[q].x, kM1Empty, (uint32_t)k) == kM1Empty) {
        t[q].y = ((uint32_t)(f - k - 1) << kM1GroupBits) | m1_fingerprint(bm);
        break;
      }
      q = (q + 1) & mask;
    }
  }
}

// Orders each alpha group's single-excitation list: groups A_s of at most
// kScanFactor x n_beta determinants first (cheaper to scan, one coalesced
// load and popcount per determinant, than to probe the index n_beta times),
// then the rest; mid[g] is where the large groups start. Each part is in
// ascending order, so that the hits of a row's scans are too: the merge of a
// row's runs rests on it. One warp per group, by counting (a list has at most
// n_alpha x (norb - n_alpha) entries, some hundred). With factors 2 / 4 / 6 / 8 /
// 12 / 16 / 32, FP64 4-vector matrix-free sigma of 100,762 determinants of 36
// orbitals: 3.35 / 3.23 / 3.22 / 3.23 / 3.33 / 3.43 / 3.89 ms, FP64 build of the
// same 7.37 / 7.25 / 7.11 / 7.09 / 7.19 / 7.31 / 7.81 ms.
constexpr int kScanFactor = 8;
template <class S>
__global__ void k_split_singles(const int64_t* __restrict__ sstart, const uint32_t* __restrict__ in,
                                const int64_t* __restrict__ gstart, const S* __restrict__ bstr, int64_t na,
                                uint32_t* __restrict__ out, int64_t* __restrict__ mid) {
  const int lane = threadIdx.x & 31;
  const int64_t warps = (int64_t)gridDim.x * (blockDim.x >> 5);
  for (int64_t g = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5; g < na; g += warps) {
    const int64_t s0 = sstart[g], s1 = sstart[g + 1];
    const int64_t cap = (int64_t)kScanFactor * bit_count(bstr[gstart[g]]);
    int64_t nsmall = 0;
    for (int64_t q = s0 + lane; q < s1; q += 32) nsmall += gstart[in[q] + 1] - gstart[in[q]] <= cap;
#pragma unroll
    for (int o = 16; o; o >>= 1) nsmall += __shfl_xor_sync(kFull, nsmall, o);
    if (lane == 0) mid[g] = s0 + nsmall;
    for (int64_t q = s0; q < s1; q += 32) {
      const bool mine = q + lane < s1;
      const uint32_t me = mine ? in[q + lane] : 0u;
      const bool small = mine && gstart[me + 1] - gstart[me] <= cap;
      int rank = 0;
      for (int64_t t = s0; t < s1; t += 32) {
        const uint32_t other = t + lane < s1 ? in[t + lane] : 0u;
        const bool osmall = t + lane < s1 && gstart[other + 1] - gstart[other] <= cap;
        const unsigned sm = __ballot_sync(kFull, osmall);
        const int cnt = (int)(s1 - t < 32 ? s1 - t : 32);
        for (int k = 0; k < cnt; ++k) {
          const uint32_t v = __shfl_sync(kFull, other, k);
          rank += (v < me) && (((sm >> k) & 1u) != 0) == small;
        }
      }
      if (mine) out[s0 + (small ? 0 : nsmall) + rank] = me;
    }
  }
}

// Single-excitation lists and partial-string index, from the strings by position.
// bits: those in which partial beta strings may differ.
template <class S>
static void build_singles_and_index(Helpers& hp, int norb, uint64_t bits, Prims& pr, cudaStream_t s) {
  const size_t n = hp.N;
  const S* bstr = reinterpret_cast<const S*>(hp.bstr.p);
  // alpha single-excitation lists
  DevBuf<int64_t> cnt;
  cnt.resize(hp.NA);
  hp.aSingStart.resize(hp.NA + 1);
  k_alpha_singles<false><<<grid_for((size_t)hp.NA * 32, 256), 256, 0, s>>>(hp.ua.p, hp.NA, norb, cnt.p, nullptr, nullptr);
  SHCI_LAUNCH_CHECK();
  int64_t total = 0;
  scan_exclusive_i64(cnt.p, hp.aSingStart.p, hp.NA, &total, pr, s);
  k_iota_last<<<1, 1, 0, s>>>(hp.aSingStart.p, hp.NA, total);
  SHCI_LAUNCH_CHECK();
  hp.aSing.resize(total > 0 ? total : 1);
  k_alpha_singles<true><<<grid_for((size_t)hp.NA * 32, 256), 256, 0, s>>>(hp.ua.p, hp.NA, norb, nullptr, hp.aSingStart.p,
                                                                         hp.aSing.p);
  SHCI_LAUNCH_CHECK();
  hp.nsing = total;
  {
    DevBuf<uint32_t> split;
    split.resize(total > 0 ? total : 1);
    hp.aSingMid.resize(hp.NA);
    k_split_singles<S><<<grid_for((size_t)hp.NA * 32, 256), 256, 0, s>>>(hp.aSingStart.p, hp.aSing.p, hp.aStart.p, bstr, hp.NA,
                                                                   split.p, hp.aSingMid.p);
    SHCI_LAUNCH_CHECK();
    hp.aSing.swap(split);
  }
  // partial-string index (one entry per determinant and occupied beta orbital)
  {
    DevBuf<int64_t> c1, o1;
    c1.resize(n);
    o1.resize(n + 1);
    k_m1_count<S><<<grid_for(n, 256), 256, 0, s>>>(bstr, n, c1.p);
    SHCI_LAUNCH_CHECK();
    int64_t ne = 0;
    scan_exclusive_i64(c1.p, o1.p, n, &ne, pr, s);
    if (ne >= ((int64_t)1 << 32)) throw Error(kErrInvalid, "partial-string index too large");
    if (hp.NA >= ((int64_t)1 << kM1GroupBits)) throw Error(kErrInvalid, "too many alpha strings for the partial-string index");
    hp.nm1 = ne;
    if (ne > 0) {
      DevBuf<uint64_t> key;
      DevBuf<uint32_t> perm;
      DevBuf<uint4> raw;
      key.resize(ne);
      perm.resize(ne);
      raw.resize(ne);
      hp.m1ent.resize(ne);
      const unsigned eb = grid_for((size_t)ne, 256);
      k_m1_fill<S><<<grid_for(n, 256), 256, 0, s>>>(bstr, hp.agrp.p, n, o1.p, key.p, perm.p, raw.p);
      SHCI_LAUNCH_CHECK();
      sort_u64(key.p, perm.p, (size_t)ne, bits, pr, s);  // by partial string
      k_m1_group_keys<<<eb, 256, 0, s>>>(raw.p, perm.p, ne, key.p);
      SHCI_LAUNCH_CHECK();
      uint64_t gbits = 1;
      while (((uint64_t)hp.NA & ~gbits) != 0) gbits = 2 * gbits + 1;
      sort_u64(key.p, perm.p, (size_t)ne, gbits, pr, s);  // then by alpha group (stable)
      k_m1_permute<<<eb, 256, 0, s>>>(raw.p, perm.p, ne, hp.m1ent.p);
      SHCI_LAUNCH_CHECK();
      // the groups' hash tables
      DevBuf<uint32_t> nkey;
      DevBuf<int64_t> slots, first;
      nkey.resize((size_t)hp.NA);
      slots.resize((size_t)hp.NA);
      first.resize((size_t)hp.NA + 1);
      SHCI_CUDA(cudaMemsetAsync(nkey.p, 0, (size_t)hp.NA * sizeof(uint32_t), s));
      k_m1_heads<<<eb, 256, 0, s>>>(hp.m1ent.p, ne, nkey.p);
      SHCI_LAUNCH_CHECK();
      k_m1_slots<<<grid_for((size_t)hp.NA, 256), 256, 0, s>>>(nkey.p, hp.NA, slots.p);
      SHCI_LAUNCH_CHECK();
      int64_t nslot = 0;
      scan_exclusive_i64(slots.p, first.p, hp.NA, &nslot, pr, s);
      hp.m1dir.resize((size_t)hp.NA);
      k_m1_dir<<<grid_for((size_t)hp.NA, 256), 256, 0, s>>>(slots.p, first.p, hp.NA, hp.m1dir.p);
      SHCI_LAUNCH_CHECK();
      hp.m1tab.resize((size_t)nslot);
      SHCI_CUDA(cudaMemsetAsync(hp.m1tab.p, 0xff, (size_t)nslot * sizeof(uint2), s));
      DevBuf<uint32_t> flag;
      flag.resize(1);
      SHCI_CUDA(cudaMemsetAsync(flag.p, 0, sizeof(uint32_t), s));
      k_m1_insert<S><<<eb, 256, 0, s>>>(hp.m1ent.p, ne, hp.m1dir.p, hp.m1tab.p, flag.p);
      SHCI_LAUNCH_CHECK();
      uint32_t too_long = 0;
      SHCI_CUDA(cudaMemcpyAsync(&too_long, flag.p, sizeof(uint32_t), cudaMemcpyDeviceToHost, s));
      SHCI_CUDA(cudaStreamSynchronize(s));
      if (too_long) hp.nm1 = 0;  // the views show no index: every group is scanned
    }
  }
}

void Helpers::build(const Det2* dets, size_t n, int norb, const Det2& ref, const Det2& diff, Prims& pr,
                    cudaStream_t s) {
  N = n;
  const uint64_t abits = det_alpha(diff), bbits = det_beta(diff);
  perm.resize(n);
  spos.resize(n);
  narrow = norb <= 32;
  str.resize(narrow ? n : 2 * n);
  bstr.resize(narrow ? (n + 1) / 2 : n);
  bAlpha.resize(narrow ? (n + 1) / 2 : n);
  agrp.resize(n);
  bgrp.resize(n);
  bPos.resize(n);
  DevBuf<uint64_t> bkey;  // beta strings by position, then in beta order
  {
    DevBuf<uint64_t> a;
    DevBuf<int64_t> flag, excl;
    a.resize(n);
    bkey.resize(n);
    flag.resize(n);
    excl.resize(n);
    const unsigned g = grid_for(n, 256);
    k_strings<<<g, 256, 0, s>>>(dets, n, a.p, bkey.p, perm.p);
    SHCI_LAUNCH_CHECK();
    sort_u128(bkey.p, a.p, perm.p, n, bbits, abits, pr, s);  // by (alpha, beta): the storage order
    if (narrow)
      k_pair_strings<uint32_t><<<g, 256, 0, s>>>(a.p, bkey.p, perm.p, n, reinterpret_cast<uint2*>(str.p),
                                                 reinterpret_cast<uint32_t*>(bstr.p), spos.p, bPos.p);
    else
      k_pair_strings<uint64_t><<<g, 256, 0, s>>>(a.p, bkey.p, perm.p, n, reinterpret_cast<ulonglong2*>(str.p), bstr.p,
                                                 spos.p, bPos.p);
    SHCI_LAUNCH_CHECK();
    k_group_flags<<<g, 256, 0, s>>>(a.p, n, flag.p);
    SHCI_LAUNCH_CHECK();
    scan_exclusive_i64(flag.p, excl.p, n, &NA, pr, s);
    ua.resize((size_t)NA);
    aStart.resize((size_t)NA + 1);
    k_group_fill<<<g, 256, 0, s>>>(a.p, nullptr, n, flag.p, excl.p, ua.p, aStart.p, agrp.p);
    SHCI_LAUNCH_CHECK();
    k_iota_last<<<1, 1, 0, s>>>(aStart.p, NA, (int64_t)n);
    SHCI_LAUNCH_CHECK();
    sort_u64(bkey.p, bPos.p, n, bbits, pr, s);  // by beta string, stable: ascending positions within a group
    k_group_flags<<<g, 256, 0, s>>>(bkey.p, n, flag.p);
    SHCI_LAUNCH_CHECK();
    scan_exclusive_i64(flag.p, excl.p, n, &NB, pr, s);
    bStart.resize((size_t)NB + 1);
    k_group_fill<<<g, 256, 0, s>>>(bkey.p, bPos.p, n, flag.p, excl.p, nullptr, bStart.p, bgrp.p);
    SHCI_LAUNCH_CHECK();
    k_iota_last<<<1, 1, 0, s>>>(bStart.p, NB, (int64_t)n);
    SHCI_LAUNCH_CHECK();
    if (narrow)
      k_gather_alpha<uint32_t><<<g, 256, 0, s>>>(reinterpret_cast<const uint2*>(str.p), bPos.p, n,
                                                 reinterpret_cast<uint32_t*>(bAlpha.p));
    else
      k_gather_alpha<uint64_t><<<g, 256, 0, s>>>(reinterpret_cast<const ulonglong2*>(str.p), bPos.p, n, bAlpha.p);
    SHCI_LAUNCH_CHECK();
  }
  // a partial string lacks one electron, so an orbital that all strings hold varies too
  const uint64_t mbits = bbits | det_beta(ref);
  if (narrow)
    build_singles_and_index<uint32_t>(*this, norb, mbits, pr, s);
  else
    build_singles_and_index<uint64_t>(*this, norb, mbits, pr, s);
}
// ---------------------------------------------------------------------------
// Row traversal shared by count, emit and the matrix-free sigma. The visitor's
// v.step<part>(hit, single, p) is called by all 32 lanes together: p the storage
// position of a connection, single whether it is a single excitation.
// ---------------------------------------------------------------------------
enum : int { kSameAlpha = 1, kAlphaMoved = 2, kSameBeta = 3 };

// One lane's probe of the index: the run of entries of key (group As, bm).
template <class S>
__device__ __forceinline__ void probe_index(const HelperView<S>& h, uint32_t As, S bm, uint32_t& lo, int& len) {
  const uint64_t d = __ldg(h.m1dir + As);
  const unsigned lg = (unsigned)(d & 63);
  const uint32_t mask = (uint32_t)((1ull << lg) - 1);
  const uint2* tab = h.m1tab + (d >> 6);
  const uint32_t fp = m1_fingerprint(bm);
  uint32_t q = m1_slot(bm, lg);
  for (uint32_t step = 0; step <= mask; ++step) {
    const uint2 sl = __ldg(tab + q);
    if (sl.x == kM1Empty) return;
    if ((sl.y & ((1u << kM1GroupBits) - 1u)) == fp) {
      // a fingerprint match is confirmed on the run's first entry
      const uint2 k0 = __ldg(reinterpret_cast<const uint2*>(h.m1ent + sl.x));
      if (k0.x == (uint32_t)bm && (sizeof(S) == 4 || k0.y == (uint32_t)((uint64_t)bm >> 32))) {
        lo = sl.x;
        len = (int)(sl.y >> kM1GroupBits) + 1;
        return;
      }
    }
    q = (q + 1) & mask;
  }
}

// The k-th set bit of B (k < its population count), as a bit.
template <class S>
__device__ __forceinline__ S nth_bit(S B, int k) {
  for (int t = 0; t < k; ++t) B &= B - 1;
  return low_one(B);
}

// Owner of flat entry f among the lanes' ranges (excl: first flat entry of each
// lane): the last lane with excl <= f.
__device__ __forceinline__ int flat_owner(int excl, int f) {
  int lo = 0;
#pragma unroll
  for (int st = 16; st >= 1; st >>= 1) {
    const int e = __shfl_sync(kFull, excl, lo + st);
    if (e <= f) lo += st;
  }
  return lo;
}
__device__ __forceinline__ int warp_incl_sum(int v) {
  const int lane = threadIdx.x & 31;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int y = __shfl_up_sync(kFull, v, o);
    if (lane >= o) v += y;
  }
  return v;
}

// Parts 1, 2a and 3: the scans. Each reports its hits in ascending position.
// The next round is loaded before this one is looked at: a round is a few
// instructions behind an L2 latency. (Four rounds at a time put the visitor's
// code in four places, and the matrix-free sigma waited for instructions.)
template <class S, class V>
__device__ __forceinline__ void scan_same_alpha(const HelperView<S>& h, uint32_t ga, S B, V& v) {
  const uint32_t p1 = (uint32_t)h.aStart[ga + 1];
  uint32_t p = (uint32_t)h.aStart[ga] + (threadIdx.x & 31);
  S b = p < p1 ? h.bstr[p] : B;  // B itself: distance 0, no hit
  for (uint32_t base = p - (threadIdx.x & 31); base < p1; base += 32, p += 32) {
    const S nb = p + 32 < p1 ? h.bstr[p + 32] : B;
    const int d = bit_count((S)(b ^ B));
    v.template step<kSameAlpha>(d == 2 || d == 4, d == 2, p);
    b = nb;
  }
}
template <class S, class V>
__device__ __forceinline__ void scan_small_groups(const HelperView<S>& h, int64_t s0, int64_t smid, S B, V& v) {
  const int lane = threadIdx.x & 31;
  for (int64_t base = s0; base < smid; base += 32) {
    uint32_t g0 = 0;
    int len = 0;
    if (base + lane < smid) {
      const uint32_t As = h.aSing[base + lane];
      g0 = (uint32_t)h.aStart[As];
      len = (int)((uint32_t)h.aStart[As + 1] - g0);
    }
    const int incl = warp_incl_sum(len);
    const int total = __shfl_sync(kFull, incl, 31);
    const int excl = incl - len;
    const uint32_t off = g0 - (uint32_t)excl;  // position of flat entry f: off of its owner + f
    uint32_t p = 0, np = 0;
    S b = (S)~B, nb = (S)~B;  // ~B: no orbital in common, no hit
    for (int f0 = -32; f0 < total; f0 += 32) {
      const int f = f0 + 32 + lane;
      nb = (S)~B;
      if (f0 + 32 < total) {
        np = __shfl_sync(kFull, off, flat_owner(excl, f)) + (uint32_t)f;
        if (f < total) nb = h.bstr[np];
      }
      if (f0 >= 0) {
        const int d = bit_count((S)(b ^ B));
        v.template step<kAlphaMoved>(d <= 2, d == 0, p);
      }
      p = np;
      b = nb;
    }
  }
}
template <class S, class V>
__device__ __forceinline__ void scan_same_beta(const HelperView<S>& h, uint32_t gb, S A, V& v) {
  const uint32_t q1 = (uint32_t)h.bStart[gb + 1];
  uint32_t q = (uint32_t)h.bStart[gb] + (threadIdx.x & 31);
  S a = q < q1 ? h.bAlpha[q] : A;
  uint32_t p = q < q1 ? h.bPos[q] : 0u;
  for (uint32_t base = q - (threadIdx.x & 31); base < q1; base += 32, q += 32) {
    const bool more = q + 32 < q1;
    const S na = more ? h.bAlpha[q + 32] : A;
    const uint32_t np = more ? h.bPos[q + 32] : 0u;
    v.template step<kSameBeta>(bit_count((S)(a ^ A)) == 4, false, p);
    a = na;
    p = np;
  }
}

// Part 2b in no particular order: probes t = (group, occupied beta orbital)
// 32 at a time, each lane stepping its own pair (no division per probe).
template <class S, class V>
__device__ __forceinline__ void probe_large_groups(const HelperView<S>& h, int64_t smid, int64_t s1, S B, V& v) {
  const int lane = threadIdx.x & 31;
  const int nb = bit_count(B);
  const int nprobe = (int)(s1 - smid) * nb;
  if (nprobe == 0) return;
  const int occ_k = lane < nb ? bit_index(nth_bit(B, lane)) : 0;  // orbitals beyond the 32nd are found bit by bit
  const int step_q = 32 / nb, step_r = 32 % nb;
  int sidx = lane / nb, which = lane % nb;
  for (int base = 0; base < nprobe; base += 32) {
    uint32_t lo = 0;
    int len = 0;  // at most 64: one entry per beta orbital outside the key
    int bq = __shfl_sync(kFull, occ_k, which & 31);  // the beta orbital removed by this probe
    if (sizeof(S) == 8 && which >= 32) bq = bit_index(nth_bit(B, which));
    const uint32_t tag = (uint32_t)bq | (which == 0 ? 256u : 0u);
    if (base + lane < nprobe) probe_index(h, h.aSing[smid + sidx], (S)(B ^ ((S)1 << bq)), lo, len);
    which += step_r;
    sidx += step_q;
    if (which >= nb) {
      which -= nb;
      ++sidx;
    }
    // flatten the lanes' matches and verify them 32 at a time
    const int incl = warp_incl_sum(len);
    const int total = __shfl_sync(kFull, incl, 31);
    const int excl = incl - len;
    const uint32_t off = lo - (uint32_t)excl;
    for (int f0 = 0; f0 < total; f0 += 32) {
      const int f = f0 + lane;
      const int src = flat_owner(excl, f);
      const uint32_t e = __shfl_sync(kFull, off, src) + (uint32_t)f;
      const uint32_t tg = __shfl_sync(kFull, tag, src);
      bool hit = false, equal = false;
      uint32_t p = 0;
      if (f < total) {
        // the entry holds J and the orbital b' its beta string has beyond
        // B - b: b' == b means beta equal (found once per occupied b, kept
        // for the first), otherwise a beta single excitation b -> b'
        const uint2 en = __ldg(reinterpret_cast<const uint2*>(h.m1ent + e) + 1);
        p = en.y;
        equal = (en.x >> kM1GroupBits) == (tg & 255u);
        hit = !equal || (tg & 256u);
      }
      v.template step<kAlphaMoved>(hit, equal, p);
    }
  }
}

template <class S, class V>
__device__ __forceinline__ void visit_row(const HelperView<S>& h, uint32_t p, S A, S B, V& v) {
  const uint32_t ga = h.agrp[p];
  scan_same_alpha(h, ga, B, v);
  const int64_t s0 = h.aSingStart[ga], s1 = h.aSingStart[ga + 1];
  const int64_t smid = (h.m1ent != nullptr && B != 0) ? h.aSingMid[ga] : s1;
  scan_small_groups(h, s0, smid, B, v);
  if (smid < s1) probe_large_groups(h, smid, s1, B, v);
  scan_same_beta(h, h.bgrp[p], A, v);
}

struct CountVisitor {
  int c = 0;
  template <int part>
  __device__ __forceinline__ void step(bool hit, bool, uint32_t) {
    c += hit;
  }
};
__device__ __forceinline__ int warp_total(int c) {
#pragma unroll
  for (int o = 16; o; o >>= 1) c += __shfl_xor_sync(kFull, c, o);
  return c;
}

// Connections of row k (position rows[k], or k) by part, and their sum.
// The index is only probed: a key's run holds the determinants one beta
// excitation away, and J with B itself (in every run of its group, to be
// counted once), which the run of the first probe shows. The space may hold a
// determinant more than once; every copy of that J is counted, as k_ham_emit
// writes each. A run ascends in its extra orbital, J's position being its order.
template <class S>
__global__ void __launch_bounds__(256, 8) k_ham_count(HelperView<S> h, const uint32_t* __restrict__ rows, int64_t nr,
                                                   uint4* __restrict__ parts, int64_t* __restrict__ counts) {
  const int lane = threadIdx.x & 31;
  const int64_t warps = (int64_t)gridDim.x * (blockDim.x >> 5);
  for (int64_t k = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5; k < nr; k += warps) {
    const uint32_t p = rows ? rows[k] : (uint32_t)k;
    const auto I = h.str[p];
    const S A = I.x, B = I.y;
    const uint32_t ga = h.agrp[p];
    CountVisitor v1, v2, v3;
    scan_same_alpha(h, ga, B, v1);
    const int64_t s0 = h.aSingStart[ga], s1 = h.aSingStart[ga + 1];
    const int64_t smid = (h.m1ent != nullptr && B != 0) ? h.aSingMid[ga] : s1;
    scan_small_groups(h, s0, smid, B, v2);
    int c4 = 0;
    const int nb = bit_count(B);
    const int nprobe = (int)(s1 - smid) * nb;
    if (nprobe > 0) {
      const int occ_k = lane < nb ? bit_index(nth_bit(B, lane)) : 0;
      const int step_q = 32 / nb, step_r = 32 % nb;
      int sidx = lane / nb, which = lane % nb;
      for (int base = 0; base < nprobe; base += 32) {
        int bq = __shfl_sync(kFull, occ_k, which & 31);
        if (sizeof(S) == 8 && which >= 32) bq = bit_index(nth_bit(B, which));
        if (base + lane < nprobe) {
          uint32_t lo = 0;
          int len = 0;
          probe_index(h, h.aSing[smid + sidx], (S)(B ^ ((S)1 << bq)), lo, len);
          c4 += len;
          if (which == 0)
            for (int e = 0; e < len; ++e) {
              const int b = (int)(__ldg(reinterpret_cast<const uint32_t*>(h.m1ent + lo + e) + 2) >> kM1GroupBits);
              if (b > bq) break;
              c4 -= b == bq ? nb - 1 : 0;
            }
        }
        which += step_r;
        sidx += step_q;
        if (which >= nb) {
          which -= nb;
          ++sidx;
        }
      }
    }
    scan_same_beta(h, h.bgrp[p], A, v3);
    const int n1 = warp_total(v1.c), n2 = warp_total(v2.c), n4 = warp_total(c4), n3 = warp_total(v3.c);
    if (lane == 0) {
      parts[k] = make_uint4((uint32_t)n1, (uint32_t)n2, (uint32_t)n4, (uint32_t)n3);
      counts[k] = (int64_t)n1 + n2 + n4 + n3;
    }
  }
}

// Writes the columns of each row as four ascending runs (the parts in the order
// of k_ham_count). The scans' hits come in ascending order. The index's do
// not: the hits of 32 / |B| groups are collected in shared memory and ranked
// by counting (some 40 per collection); groups that hold more hits than fit
// are scanned instead. Bound by instruction issue (68 %) and the L2 latency of
// the probes.
constexpr int kCollect = 256;
struct AppendVisitor {
  int32_t* col;
  int64_t pos;
  unsigned lt;
  template <int part>
  __device__ __forceinline__ void step(bool hit, bool, uint32_t p) {
    const unsigned m = __ballot_sync(kFull, hit);
    if (hit) col[pos + __popc(m & lt)] = (int32_t)p;
    pos += __popc(m);
  }
};
template <class S>
__global__ void __launch_bounds__(256, 6) k_ham_emit(HelperView<S> h, const uint32_t* __restrict__ rows, int64_t nr,
                                                  const int64_t* __restrict__ rowptr, int32_t* __restrict__ col) {
  __shared__ __align__(16) uint32_t s_buf[8][kCollect];
  const int lane = threadIdx.x & 31;
  const unsigned lt = (1u << lane) - 1u;
  uint32_t* buf = s_buf[threadIdx.x >> 5];
  const int64_t warps = (int64_t)gridDim.x * (blockDim.x >> 5);
  for (int64_t k = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5; k < nr; k += warps) {
    const uint32_t p = rows ? rows[k] : (uint32_t)k;
    const auto I = h.str[p];
    const S A = I.x, B = I.y;
    const uint32_t ga = h.agrp[p];
    AppendVisitor v{col, rowptr[k], lt};
    scan_same_alpha(h, ga, B, v);
    const int64_t s0 = h.aSingStart[ga], s1 = h.aSingStart[ga + 1];
    const int64_t smid = (h.m1ent != nullptr && B != 0) ? h.aSingMid[ga] : s1;
    scan_small_groups(h, s0, smid, B, v);
    if (smid < s1) {
      const int nb = bit_count(B);
      const int per = nb <= 32 ? 32 / nb : 1;  // groups per collection
      const int mine = nb <= 32 ? lane / nb : 0, which0 = nb <= 32 ? lane % nb : lane;
      const int bq0 = which0 < nb ? bit_index(nth_bit(B, which0)) : 0;
      for (int64_t s = smid; s < s1; s += per) {
        int n = 0;
        bool over = false;
        for (int w = 0; w < nb; w += 32) {  // more than one round only past 32 beta electrons
          const int which = which0 + w;
          const int bq = sizeof(S) == 4 || w == 0 ? bq0 : (which < nb ? bit_index(nth_bit(B, which)) : 0);
          uint32_t lo = 0;
          int len = 0;
          if (mine < per && which < nb && s + mine < s1) probe_index(h, h.aSing[s + mine], (S)(B ^ ((S)1 << bq)), lo, len);
          const uint32_t tag = (uint32_t)bq | (which == 0 ? 256u : 0u);
          const int incl = warp_incl_sum(len);
          const int total = __shfl_sync(kFull, incl, 31);
          const int excl = incl - len;
          const uint32_t off = lo - (uint32_t)excl;
          for (int f0 = 0; f0 < total && !over; f0 += 32) {
            const int f = f0 + lane;
            const int src = flat_owner(excl, f);
            const uint32_t e = __shfl_sync(kFull, off, src) + (uint32_t)f;
            const uint32_t tg = __shfl_sync(kFull, tag, src);
            bool hit = false;
            uint32_t q = 0;
            if (f < total) {
              const uint2 en = __ldg(reinterpret_cast<const uint2*>(h.m1ent + e) + 1);
              q = en.y;
              hit = (en.x >> kM1GroupBits) != (tg & 255u) || (tg & 256u);
            }
            const unsigned m = __ballot_sync(kFull, hit);
            over = n + __popc(m) > kCollect;
            if (hit && !over) buf[n + __popc(m & lt)] = q;
            if (!over) n += __popc(m);
          }
        }
        if (over) {
          __syncwarp();
          scan_small_groups(h, s, s + per < s1 ? s + per : s1, B, v);
          continue;
        }
        const int pad = (4 - (n & 3)) & 3;
        if (lane < pad) buf[n + lane] = 0xffffffffu;
        __syncwarp();
        for (int t = 0; t < n; t += 32) {
          const uint32_t key = t + lane < n ? buf[t + lane] : 0u;
          int rank = 0;
          for (int j = 0; j < n; j += 4) {
            const uint4 o = *reinterpret_cast<const uint4*>(buf + j);
            rank += (o.x < key) + (o.y < key) + (o.z < key) + (o.w < key);
          }
          if (t + lane < n) col[v.pos + rank] = (int32_t)key;
        }
        v.pos += n;
        __syncwarp();
      }
    }
    scan_same_beta(h, h.bgrp[p], A, v);
  }
}

// ---------------------------------------------------------------------------
// Elements. The values are those of Hij_1Excite / Hij_2Excite
// (SHCI/Determinants.cpp:406-505): the same integrals and differences, summed
// in the same order, with the parity of the moves taken on the strings. Which
// of the two determinants is the ket makes no difference: a double's integrals
// are symmetric, and a single's sum differs only in where its zero terms
// stand ((ai|ii) - (ai|ii) for the orbital left behind).
// ---------------------------------------------------------------------------
// Integral access in either precision (FP64: __dsub_rn, so never contracted).
__device__ __forceinline__ int pair_of(int lo, int hi) { return hi * (hi + 1) / 2 + lo; }  // lo <= hi
template <bool F32>
struct Elem;
template <>
struct Elem<false> {
  using T = double;
  __device__ static T i2(const IntsView& v, int ij, int kl) {
    const unsigned A = (unsigned)max(ij, kl), B = (unsigned)min(ij, kl);
    return __ldg(v.I2 + (A * (A + 1) / 2 + B));
  }
  __device__ static T sub(T a, T b) { return __dsub_rn(a, b); }
  __device__ static T signed_(T v, unsigned odd) {
    return __hiloint2double(__double2hiint(v) ^ (int)(odd << 31), __double2loint(v));
  }
  __device__ static T single(const IntsView& v, const Det2& d, int a, int i) { return hij_single(v, d, a, i); }
};
template <>
struct Elem<true> {
  using T = float;
  __device__ static T i2(const IntsView& v, int ij, int kl) {
    const unsigned A = (unsigned)max(ij, kl), B = (unsigned)min(ij, kl);
    return __ldg(v.I2f + (A * (A + 1) / 2 + B));
  }
  __device__ static T sub(T a, T b) { return __fsub_rn(a, b); }
  __device__ static T signed_(T v, unsigned odd) { return __uint_as_float(__float_as_uint(v) ^ (odd << 31)); }
  __device__ static T single(const IntsView& v, const Det2& d, int a, int i) { return hij_single_f32(v, d, a, i); }
};
// alpha and beta moved once each
template <bool F32, class S>
__device__ __forceinline__ typename Elem<F32>::T elem_ab(const IntsView& v, S A, S B, S A2, S B2) {
  const S x = A ^ A2, y = B ^ B2;
  const unsigned odd = bit_count((S)(passed(A, B, x, false) ^ passed(B, A2, y, true))) & 1;
  const S xl = low_one(x), yl = low_one(y);  // a pair's index does not depend on which of the two was occupied
  return Elem<F32>::signed_(Elem<F32>::i2(v, pair_of(bit_index(xl), bit_index((S)(x ^ xl))),
                                          pair_of(bit_index(yl), bit_index((S)(y ^ yl)))),
                            odd);
}
// the same as FP32 head and tail (exactly those of the FP64 value: the sign
// changes neither rounding)
template <class S>
__device__ __forceinline__ float2 elem_ab_split(const IntsView& v, S A, S B, S A2, S B2) {
  const S x = A ^ A2, y = B ^ B2;
  const unsigned odd = bit_count((S)(passed(A, B, x, false) ^ passed(B, A2, y, true))) & 1;
  const S xl = low_one(x), yl = low_one(y);
  const int ij = pair_of(bit_index(xl), bit_index((S)(x ^ xl))), kl = pair_of(bit_index(yl), bit_index((S)(y ^ yl)));
  const unsigned P = (unsigned)max(ij, kl), Q = (unsigned)min(ij, kl);
  const float2 t = __ldg(v.I2ff + (P * (P + 1) / 2 + Q));
  return make_float2(__uint_as_float(__float_as_uint(t.x) ^ (odd << 31)),
                     __uint_as_float(__float_as_uint(t.y) ^ (odd << 31)));
}
// two electrons of one spin moved: s -> s2, the other string o
template <bool F32, class S>
__device__ __forceinline__ typename Elem<F32>::T elem_same(const IntsView& v, S s, S o, S s2, bool beta) {
  const S x = s ^ s2, d = x & s, c = x ^ d;
  const S di = low_one(d), dj = d ^ di, ca = low_one(c), cb = c ^ ca;
  const unsigned odd = bit_count((S)(passed(s, o, (S)(di | ca), beta) ^ passed((S)(s ^ di ^ ca), o, (S)(dj | cb), beta))) & 1;
  const int i = bit_index(di), j = bit_index(dj), a = bit_index(ca), b = bit_index(cb);
  return Elem<F32>::signed_(Elem<F32>::sub(Elem<F32>::i2(v, pair_index(a, i), pair_index(b, j)),
                                           Elem<F32>::i2(v, pair_index(a, j), pair_index(b, i))),
                            odd);
}
// one electron moved: s -> s2 of a determinant with strings A and B
template <bool F32, class S>
__device__ __forceinline__ typename Elem<F32>::T elem_single(const IntsView& v, S A, S B, S s, S s2, bool beta) {
  const S x = s ^ s2;
  return Elem<F32>::single(v, det_from_strings((uint64_t)A, (uint64_t)B), 2 * bit_index((S)(x & s2)) + (beta ? 1 : 0),
                           2 * bit_index((S)(x & s)) + (beta ? 1 : 0));
}

// ---------------------------------------------------------------------------
// Finishing the rows: the four ascending runs of a row are merged and the
// elements evaluated, a thread per connection. An entry's place is its place
// in its own run plus the entries of the other runs below it; run 1 (same
// alpha string) is one range of positions that no other run enters, so only
// the other two runs are searched. Evaluating here, and not where a connection
// is found, keeps the walk's registers free of the element code and puts
// every lane on an element. 5.5e8 entries (mol24, mixed: the spaces of 81,233
// and 405,690 determinants): emitting 10.5 ms, finishing 6.9 + 1.3 ms; emitting with
// evaluation and sorting each row by a bitonic network took 58.6 ms for 3.6e8.
// ---------------------------------------------------------------------------
// Entries of a row kept in a small block's shared memory; longer rows go to
// blocks of their own size, with up to kLongShared entries in shared memory and
// the few beyond in a scratch copy. 5.5e8 entries, both kernels: 3,072 and blocks
// of 1,024 that search in the scratch copy 8.31 + 1.53 ms; 3,072 8.31 + 0.94; 2,560
// 6.86 + 1.32 (16 blocks per SM instead of 13); 2,048 6.29 + 2.08; 1,536 5.28 + 3.92.
constexpr int kRunCap = 2560;
constexpr int kLongThreads = 512, kLongShared = 7168;
constexpr int kFinThreads = 128;  // 64: 15.4 ms, 96: 12.9 ms, 128: 11.4 ms for 5.5e8 entries (16 blocks per SM)
// Blocks per SM of the launches that go over rows: many times what is resident
// (5 to 16 blocks per SM), so that blocks that end early make room for others.
// 5.5e8 entries, 16 per SM before (3.2 and 1.3 waves): counting 3.88 -> 3.46 ms and
// emitting 12.84 -> 11.30 (5: 4.45 and 13.07; 40: 3.56 and 11.93), finishing 11.42 ->
// 8.31 (12: 9.98; 96: 9.20; 4,000: 8.38). Counting with 8 resident blocks (32
// registers) 3.46 -> 3.12, emitting with 6 (40) 11.32 -> 10.47.
constexpr size_t kRowBlocks = 160, kFinBlocks = 1536;

__device__ __forceinline__ int run_below(const uint32_t* run, int n, uint32_t c) {  // entries of a run below c
  int lo = 0, hi = n;
  while (lo < hi) {
    const int mid = (lo + hi) >> 1;
    if (run[mid] < c)
      lo = mid + 1;
    else
      hi = mid;
  }
  return lo;
}

// Where a row's entries go. Mixed values are an FP32 head and tail; an
// alpha-beta double's come from a table of split integrals, since the two
// conversions and the subtraction would take the FP64 pipe (two lanes per
// clock and SM) 64 clocks per 32 entries.
struct FinishOut {
  int32_t* __restrict__ col;
  double* __restrict__ v64;
  float* __restrict__ vhi;
  float* __restrict__ vlo;
  __device__ __forceinline__ void put(int64_t q, double v) const {
    if (v64) {
      v64[q] = v;
    } else {
      const float hi = (float)v;
      vhi[q] = hi;
      if (vlo) vlo[q] = (float)(v - (double)hi);
    }
  }
  __device__ __forceinline__ void put(int64_t q, float2 v) const {
    vhi[q] = v.x;
    if (vlo) vlo[q] = v.y;
  }
};

// Single excitations wait per warp, over rows, until 32 are there: their
// elements are sums over every electron in FP64 (two lanes per clock and SM),
// and one among a warp's 32 entries would make the whole warp run the sum.
// Entry: place (64 bits), position of the row, of the column.
template <class S>
struct SingleQueue {
  uint4* q;  // 64 entries
  int n = 0;
  __device__ __forceinline__ void push(bool s, int64_t at, uint32_t p, uint32_t c, const HelperView<S>& h,
                                       const IntsView& ints, const FinishOut& out) {
    const unsigned m = __ballot_sync(kFull, s);
    if (!m) return;
    if (s) q[n + __popc(m & ((1u << (threadIdx.x & 31)) - 1u))] = make_uint4((uint32_t)at, (uint32_t)(at >> 32), p, c);
    n += __popc(m);
    __syncwarp();
    if (n >= 32) drain(32, h, ints, out);
  }
  __device__ __forceinline__ void drain(int cnt, const HelperView<S>& h, const IntsView& ints, const FinishOut& out) {
    const int lane = threadIdx.x & 31;
    if (lane < cnt) {
      const uint4 w = q[lane];
      const auto I = h.str[w.z], J = h.str[w.w];
      const bool beta = I.x == J.x;
      out.put((int64_t)(((uint64_t)w.y << 32) | w.x),
              elem_single<false, S>(ints, I.x, I.y, beta ? I.y : I.x, beta ? J.y : J.x, beta));
    }
    __syncwarp();
    const int rest = n - cnt;
    const uint4 v = lane < rest ? q[cnt + lane] : make_uint4(0u, 0u, 0u, 0u);
    __syncwarp();
    if (lane < rest) q[lane] = v;
    __syncwarp();
    n = rest;
  }
};

template <class S, bool kSplit>
__device__ __forceinline__ void finish_row(const HelperView<S>& h, const IntsView& ints, uint32_t p, const uint4& n,
                                           const uint32_t* run, int64_t p0, const FinishOut& out, SingleQueue<S>& sq) {
  const auto I = h.str[p];
  const S A = I.x, B = I.y;
  const int n1 = (int)n.x, n2 = (int)n.y, n3 = (int)n.z, n4 = (int)n.w;
  const uint32_t *r2 = run + n1, *r3 = r2 + n2, *r4 = r3 + n3;
  const int len = n1 + n2 + n3 + n4;
  // kTwo entries of a thread at a time: their strings and integrals are in
  // flight together. All lanes together: the queue's ballots.
  constexpr int kTwo = 2;
  for (int e0 = 0; e0 < len; e0 += kTwo * blockDim.x) {
    bool single[kTwo];
    uint32_t c[kTwo];
    int64_t q[kTwo];
    typename StrPair<S>::T J[kTwo];
#pragma unroll
    for (int u = 0; u < kTwo; ++u) {
      const int e = e0 + u * (int)blockDim.x + (int)threadIdx.x;
      single[u] = false;
      c[u] = e < len ? run[e] : p;
      J[u] = h.str[c[u]];
    }
#pragma unroll
    for (int u = 0; u < kTwo; ++u) {
      const int e = e0 + u * (int)blockDim.x + (int)threadIdx.x;
      if (e >= len) continue;
      // the two other runs to be searched (run 1: all three)
      const bool in1 = e < n1, in2 = !in1 && e < n1 + n2, in4 = e >= n1 + n2 + n3;
      const bool first = !in2, last = in2 || (!in1 && !in4);  // run 2 is searched first; run 4 last (else run 3)
      int rank = e + run_below(first ? r2 : r3, first ? n2 : n3, c[u]) + run_below(last ? r4 : r3, last ? n4 : n3, c[u]);
      if (in1)
        rank += run_below(r4, n4, c[u]);
      else
        rank -= (n1 > 0 && c[u] > run[0] ? 0 : n1) + (in2 ? 0 : in4 ? n2 + n3 : n2);
      q[u] = p0 + rank;
      out.col[q[u]] = (int32_t)c[u];
      if (in1 || in4) {  // same alpha or same beta string
        const bool beta = in1;
        single[u] = beta && bit_count((S)(B ^ J[u].y)) == 2;
        if (!single[u])
          out.put(q[u], elem_same<false, S>(ints, beta ? B : A, beta ? A : B, beta ? J[u].y : J[u].x, beta));
      } else {
        single[u] = J[u].y == B;
        if (!single[u]) {
          if constexpr (kSplit)
            out.put(q[u], elem_ab_split<S>(ints, A, B, J[u].x, J[u].y));
          else
            out.put(q[u], elem_ab<false, S>(ints, A, B, J[u].x, J[u].y));
        }
      }
    }
#pragma unroll
    for (int u = 0; u < kTwo; ++u) sq.push(single[u], q[u], p, c[u], h, ints, out);
  }
}

template <class S, bool kSplit>
__global__ void __launch_bounds__(kFinThreads) k_ham_finish(HelperView<S> h, IntsView ints,
                                                            const uint32_t* __restrict__ rows, int64_t nr,
                                                            const uint4* __restrict__ parts,
                                                            const int64_t* __restrict__ rowptr,
                                                            int32_t* __restrict__ col, double* __restrict__ v64,
                                                            float* __restrict__ vhi, float* __restrict__ vlo) {
  __shared__ uint32_t run[kRunCap];
  __shared__ uint4 s_q[kFinThreads / 32][64];
  const FinishOut out{col, v64, vhi, vlo};
  SingleQueue<S> sq{s_q[threadIdx.x >> 5]};
  for (int64_t k = blockIdx.x; k < nr; k += gridDim.x) {
    const int64_t p0 = rowptr[k];
    const int len = (int)(rowptr[k + 1] - p0);
    if (len == 0 || len > kRunCap) continue;  // uniform across the block
    for (int e = threadIdx.x; e < len; e += blockDim.x) run[e] = (uint32_t)col[p0 + e];
    __syncthreads();
    finish_row<S, kSplit>(h, ints, rows ? rows[k] : (uint32_t)k, parts[k], run, p0, out, sq);
    __syncthreads();
  }
  if (sq.n) sq.drain(sq.n, h, ints, out);
}

// Rows past kRunCap: listed, and with their places in a scratch copy past kLongShared.
__global__ void k_long_runs(const int64_t* __restrict__ rowptr, int64_t nr, uint2* __restrict__ list, uint32_t cap,
                            unsigned long long* __restrict__ tot) {
  for (int64_t k = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; k < nr; k += (int64_t)gridDim.x * blockDim.x) {
    const int64_t len = rowptr[k + 1] - rowptr[k];
    if (len <= kRunCap) continue;
    const unsigned long long i = atomicAdd(tot, 1ull);
    const unsigned long long off = len > kLongShared ? atomicAdd(tot + 1, (unsigned long long)((len + 31) / 32)) : 0;
    if (i < cap) list[i] = make_uint2((uint32_t)k, (uint32_t)off);
  }
}
template <class S, bool kSplit>
__global__ void __launch_bounds__(kLongThreads) k_ham_finish_long(HelperView<S> h, IntsView ints,
                                                          const uint32_t* __restrict__ rows,
                                                          const uint2* __restrict__ list, uint32_t* scratch,
                                                          const uint4* __restrict__ parts,
                                                          const int64_t* __restrict__ rowptr,
                                                          int32_t* __restrict__ col, double* __restrict__ v64,
                                                          float* __restrict__ vhi, float* __restrict__ vlo) {
  __shared__ uint4 s_q[kLongThreads / 32][64];
  __shared__ uint32_t s_run[kLongShared];
  const FinishOut out{col, v64, vhi, vlo};
  SingleQueue<S> sq{s_q[threadIdx.x >> 5]};
  const uint2 l = list[blockIdx.x];
  const int64_t p0 = rowptr[l.x];
  const int len = (int)(rowptr[l.x + 1] - p0);
  const uint32_t p = rows ? rows[l.x] : l.x;
  if (len <= kLongShared) {
    for (int e = threadIdx.x; e < len; e += blockDim.x) s_run[e] = (uint32_t)col[p0 + e];
    __syncthreads();
    finish_row<S, kSplit>(h, ints, p, parts[l.x], s_run, p0, out, sq);
  } else {
    uint32_t* run = scratch + 32 * (size_t)l.y;
    for (int e = threadIdx.x; e < len; e += blockDim.x) run[e] = (uint32_t)col[p0 + e];
    __syncthreads();
    finish_row<S, kSplit>(h, ints, p, parts[l.x], run, p0, out, sq);
  }
  if (sq.n) sq.drain(sq.n, h, ints, out);
}

__global__ void k_set_last(int64_t* rowptr, int64_t n, int64_t total) { rowptr[n] = total; }

// Sort of one row's new columns (extended builds), one block per row. The
// columns become 64-bit keys (column << 12 | position in the row) sorted by a
// bitonic network in which each of the 256 threads keeps E consecutive keys in
// registers: the compare-exchange steps between keys of one thread run in
// registers, only the longer-distance steps go through shared memory (36 of the
// 66 steps for a 2048-key row). The values are then gathered from their old
// positions (read into registers before any write, the row is sorted in place).
// Rows longer than kRowSortCap are sorted by k_long_row_sort.
constexpr int kRowSortCap = 4096;
constexpr int kSortThreads = 256;

template <int E>
__device__ __forceinline__ void sort_exchange_regs(uint64_t (&v)[E], int g0, int k) {
  // the steps of merge size k with partner distance j < E: partner in the same thread
#pragma unroll
  for (int j = E >> 1; j > 0; j >>= 1) {
    if (j >= k) continue;  // merges smaller than E start at j = k / 2
#pragma unroll
    for (int e = 0; e < E; ++e) {
      const int pe = e ^ j;
      if (pe > e) {
        const bool up = ((g0 + e) & k) == 0;
        const uint64_t x = v[e], y = v[pe];
        if ((x > y) == up) {
          v[e] = y;
          v[pe] = x;
        }
      }
    }
  }
}

template <int E>
__device__ void sort_row_keys(uint64_t* sk, int P) {
  // threads [0, P/E) own keys [t*E, t*E+E); others only join the barriers
  const int T = P / E;
  const int t = threadIdx.x;
  const bool act = t < T;
  const int g0 = t * E;
  uint64_t v[E];
  for (int k = 2; k <= P; k <<= 1) {
    // distances j >= E: pairs in shared memory
    for (int j = k >> 1; j >= E; j >>= 1) {
      for (int q = t; q < P / 2; q += blockDim.x) {
        const int lo = ((q & ~(j - 1)) << 1) | (q & (j - 1));  // lower index of the q-th pair (j a power of two)
        const int hi = lo + j;
        const bool up = (lo & k) == 0;
        const uint64_t x = sk[lo], y = sk[hi];
        if ((x > y) == up) {
          sk[lo] = y;
          sk[hi] = x;
        }
      }
      __syncthreads();
    }
    // distances j < E: in registers
    if (E > 1) {
      if (act) {
#pragma unroll
        for (int e = 0; e < E; ++e) v[e] = sk[g0 + e];
        sort_exchange_regs<E>(v, g0, k);
#pragma unroll
        for (int e = 0; e < E; ++e) sk[g0 + e] = v[e];
      }
      __syncthreads();
    }
  }
}

__global__ void __launch_bounds__(kSortThreads) k_row_sort(const int64_t* __restrict__ rowptr, size_t N,
                                                           int32_t* __restrict__ col, double* __restrict__ v64,
                                                           float* __restrict__ vhi, float* __restrict__ vlo) {
  __shared__ uint64_t sk[kRowSortCap];
  constexpr int kPer = kRowSortCap / kSortThreads;  // values gathered per thread
  for (size_t r = blockIdx.x; r < N; r += gridDim.x) {
    const int64_t p0 = rowptr[r], len = rowptr[r + 1] - p0;
    if (len <= 1 || len > kRowSortCap) continue;  // uniform across the block
    int P = 2;
    while (P < len) P <<= 1;
    for (int i = threadIdx.x; i < P; i += blockDim.x)
      sk[i] = i < len ? ((uint64_t)(uint32_t)col[p0 + i] << 12) | (uint64_t)i : ~0ull;
    __syncthreads();
    if (P >= 16 * kSortThreads)
      sort_row_keys<16>(sk, P);
    else if (P >= 8 * kSortThreads)
      sort_row_keys<8>(sk, P);
    else if (P >= 4 * kSortThreads)
      sort_row_keys<4>(sk, P);
    else if (P >= 2 * kSortThreads)
      sort_row_keys<2>(sk, P);
    else
      sort_row_keys<1>(sk, P);
    // gather the values of this thread's output positions, then write
    uint64_t pay[kPer];
#pragma unroll
    for (int m = 0; m < kPer; ++m) {
      const int i = threadIdx.x + m * kSortThreads;
      pay[m] = 0;
      if (i < len) {
        const int src = (int)(sk[i] & 0xFFFull);
        if (v64) {
          pay[m] = (uint64_t)__double_as_longlong(v64[p0 + src]);
        } else {
          pay[m] = (uint64_t)__float_as_uint(vhi[p0 + src]);
          if (vlo) pay[m] |= (uint64_t)__float_as_uint(vlo[p0 + src]) << 32;
        }
      }
    }
    __syncthreads();
#pragma unroll
    for (int m = 0; m < kPer; ++m) {
      const int i = threadIdx.x + m * kSortThreads;
      if (i < len) {
        col[p0 + i] = (int32_t)(sk[i] >> 12);
        if (v64) {
          v64[p0 + i] = __longlong_as_double((long long)pay[m]);
        } else {
          vhi[p0 + i] = __uint_as_float((uint32_t)pay[m]);
          if (vlo) vlo[p0 + i] = __uint_as_float((uint32_t)(pay[m] >> 32));
        }
      }
    }
    __syncthreads();
  }
}

// Value arrays of a CSR as raw pointers.
struct CsrVals {
  int32_t* col;
  double* v64;
  float* vhi;
  float* vlo;
};

// Rows longer than kRowSortCap: one 1024-thread block per row runs the
// bitonic network on 64-bit keys (column << 32 | position) in a global
// scratch segment (L2-resident), then the values are permuted through a second
// scratch segment. Every row then leaves the build sorted, so the order of a
// row's entries (and of sigma's sums over it) does not depend on the atomic
// order in which the incremental build placed its new columns.
__global__ void k_long_rows(const int64_t* __restrict__ rowptr, size_t N, int cap, uint32_t* __restrict__ list,
                            unsigned long long* __restrict__ count) {
  for (size_t r = (size_t)blockIdx.x * blockDim.x + threadIdx.x; r < N; r += (size_t)gridDim.x * blockDim.x)
    if (rowptr[r + 1] - rowptr[r] > cap) list[atomicAdd(count, 1ull)] = (uint32_t)r;
}
__global__ void __launch_bounds__(1024) k_long_row_sort(const int64_t* __restrict__ rowptr,
                                                        const uint32_t* __restrict__ rows,
                                                        const int64_t* __restrict__ soff, uint64_t* __restrict__ key,
                                                        uint64_t* __restrict__ pay, CsrVals v) {
  const size_t r = rows[blockIdx.x];
  const int64_t p0 = rowptr[r], len = rowptr[r + 1] - p0;
  uint64_t* k = key + soff[blockIdx.x];
  uint64_t* y = pay + soff[blockIdx.x];
  int64_t P = 2;
  while (P < len) P <<= 1;
  for (int64_t i = threadIdx.x; i < P; i += blockDim.x)
    k[i] = i < len ? ((uint64_t)(uint32_t)v.col[p0 + i] << 32) | (uint64_t)i : ~0ull;
  __syncthreads();
  for (int64_t kk = 2; kk <= P; kk <<= 1)
    for (int64_t j = kk >> 1; j > 0; j >>= 1) {
      for (int64_t q = threadIdx.x; q < P / 2; q += blockDim.x) {
        const int64_t lo = ((q & ~(j - 1)) << 1) | (q & (j - 1)), hi = lo + j;  // j a power of two
        const bool up = (lo & kk) == 0;
        const uint64_t a = k[lo], b = k[hi];
        if ((a > b) == up) {
          k[lo] = b;
          k[hi] = a;
        }
      }
      __syncthreads();
    }
  // permute the values through y, then write columns and values back
  for (int64_t i = threadIdx.x; i < len; i += blockDim.x) {
    const int64_t src = (int64_t)(k[i] & 0xFFFFFFFFull);
    uint64_t val;
    if (v.v64) {
      val = (uint64_t)__double_as_longlong(v.v64[p0 + src]);
    } else {
      val = (uint64_t)__float_as_uint(v.vhi[p0 + src]);
      if (v.vlo) val |= (uint64_t)__float_as_uint(v.vlo[p0 + src]) << 32;
    }
    y[i] = val;
  }
  __syncthreads();
  for (int64_t i = threadIdx.x; i < len; i += blockDim.x) {
    v.col[p0 + i] = (int32_t)(k[i] >> 32);
    const uint64_t val = y[i];
    if (v.v64) {
      v.v64[p0 + i] = __longlong_as_double((long long)val);
    } else {
      v.vhi[p0 + i] = __uint_as_float((uint32_t)val);
      if (v.vlo) v.vlo[p0 + i] = __uint_as_float((uint32_t)(val >> 32));
    }
  }
}

__global__ void k_list_lens(const int64_t* __restrict__ rowptr, const uint32_t* __restrict__ rows, size_t n,
                            int64_t* __restrict__ len) {
  for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x)
    len[i] = rowptr[rows[i] + 1] - rowptr[rows[i]];
}

static void sort_rows(const int64_t* rowptr, size_t n, const CsrVals& v, cudaStream_t s) {
  if (n == 0) return;
  const unsigned sblocks = (unsigned)std::min<size_t>(n, 152 * 6);
  k_row_sort<<<sblocks, kSortThreads, 0, s>>>(rowptr, n, v.col, v.v64, v.vhi, v.vlo);
  SHCI_LAUNCH_CHECK();
  // rows past the shared-memory cap
  DevBuf<unsigned long long> cnt;
  cnt.resize(1);
  SHCI_CUDA(cudaMemsetAsync(cnt.p, 0, sizeof(unsigned long long), s));
  DevBuf<uint32_t> list;
  list.resize(n);
  k_long_rows<<<grid_for(n, 256), 256, 0, s>>>(rowptr, n, kRowSortCap, list.p, cnt.p);
  SHCI_LAUNCH_CHECK();
  unsigned long long nl = 0;
  SHCI_CUDA(cudaMemcpyAsync(&nl, cnt.p, sizeof(nl), cudaMemcpyDeviceToHost, s));
  SHCI_CUDA(cudaStreamSynchronize(s));
  if (nl == 0) return;
  DevBuf<int64_t> lens;
  lens.resize(nl);
  k_list_lens<<<grid_for(nl, 256), 256, 0, s>>>(rowptr, list.p, nl, lens.p);
  SHCI_LAUNCH_CHECK();
  std::vector<int64_t> hl(nl);
  SHCI_CUDA(cudaMemcpyAsync(hl.data(), lens.p, nl * sizeof(int64_t), cudaMemcpyDeviceToHost, s));
  SHCI_CUDA(cudaStreamSynchronize(s));
  std::vector<int64_t> off(nl);
  int64_t tot = 0;
  for (unsigned long long i = 0; i < nl; ++i) {
    int64_t P = 2;
    while (P < hl[i]) P <<= 1;
    off[i] = tot;
    tot += P;
  }
  DevBuf<int64_t> doff;
  doff.resize(nl);
  SHCI_CUDA(cudaMemcpyAsync(doff.p, off.data(), nl * sizeof(int64_t), cudaMemcpyHostToDevice, s));
  DevBuf<uint64_t> key, pay;
  key.resize(tot);
  pay.resize(tot);
  k_long_row_sort<<<(unsigned)nl, 1024, 0, s>>>(rowptr, list.p, doff.p, key.p, pay.p, v);
  SHCI_LAUNCH_CHECK();
  SHCI_CUDA(cudaStreamSynchronize(s));  // the scratch is freed on return
}

// Full rows of nr positions (rows[k], or all when null) into out's row pointers
// and values, columns ascending; returns nnz. out holds no rows (N = 0) from where
// its arrays are first touched, so that an allocation that fails half way leaves
// nothing that looks like a matrix; the caller sets N.
template <class S>
static int64_t emit_rows_as(const Helpers& hp, const uint32_t* rows, size_t nr, const IntsView& ints, Csr& out,
                            bool want64, bool want32, bool want_lo, Prims& pr, cudaStream_t s, PhaseTimer& pt) {
  DevBuf<int64_t>& rowptr = out.rowptr;
  DevBuf<int32_t>& col = out.col;
  DevBuf<double>& v64 = out.v64;
  DevBuf<float>&vhi = out.vhi, &vlo = out.vlo;
  HelperView<S> hv = hp.view<S>();
  DevBuf<int64_t> counts;
  DevBuf<uint4> parts;
  counts.resize(nr > 0 ? nr : 1);
  parts.resize(nr > 0 ? nr : 1);
  const unsigned blocks = grid_for(nr * 32, 256, 152 * kRowBlocks);
  if (nr) {
    k_ham_count<S><<<blocks, 256, 0, s>>>(hv, rows, (int64_t)nr, parts.p, counts.p);
    SHCI_LAUNCH_CHECK();
  }
  pt.mark("ham count");
  out.N = 0;
  out.nnz = 0;
  rowptr.resize(nr + 1);
  int64_t total = 0;
  scan_exclusive_i64(counts.p, rowptr.p, nr, &total, pr, s);
  k_set_last<<<1, 1, 0, s>>>(rowptr.p, (int64_t)nr, total);
  SHCI_LAUNCH_CHECK();
  const size_t cap = total > 0 ? (size_t)total : 1;
  col.resize(cap);
  if (want64) v64.resize(cap); else v64.release();
  if (want32) vhi.resize(cap); else vhi.release();
  if (want32 && want_lo) vlo.resize(cap); else vlo.release();
  if (total == 0) return 0;
  k_ham_emit<S><<<blocks, 256, 0, s>>>(hv, rows, (int64_t)nr, rowptr.p, col.p);
  SHCI_LAUNCH_CHECK();
  pt.mark("ham emit");
  double* d64 = want64 ? v64.p : nullptr;
  float* dhi = want32 ? vhi.p : nullptr;
  float* dlo = want32 && want_lo ? vlo.p : nullptr;
  // the long rows are listed first, and read from their untouched runs
  const size_t ncap = (size_t)(total / kRunCap) + 1;
  DevBuf<uint2> list;
  DevBuf<unsigned long long> tot;
  list.resize(ncap);
  tot.resize(2);
  SHCI_CUDA(cudaMemsetAsync(tot.p, 0, 2 * sizeof(unsigned long long), s));
  k_long_runs<<<grid_for(nr, 256), 256, 0, s>>>(rowptr.p, (int64_t)nr, list.p, (uint32_t)ncap, tot.p);
  SHCI_LAUNCH_CHECK();
  const bool split = want32 && ints.I2ff != nullptr;
  const unsigned fb = (unsigned)std::min<size_t>(nr, 152 * kFinBlocks);
  if (split)
    k_ham_finish<S, true><<<fb, kFinThreads, 0, s>>>(hv, ints, rows, (int64_t)nr, parts.p, rowptr.p, col.p, d64, dhi,
                                                     dlo);
  else
    k_ham_finish<S, false><<<fb, kFinThreads, 0, s>>>(hv, ints, rows, (int64_t)nr, parts.p, rowptr.p, col.p, d64, dhi,
                                                      dlo);
  SHCI_LAUNCH_CHECK();
  unsigned long long nl[2] = {0, 0};
  SHCI_CUDA(cudaMemcpyAsync(nl, tot.p, sizeof(nl), cudaMemcpyDeviceToHost, s));
  SHCI_CUDA(cudaStreamSynchronize(s));
  if (nl[0] > 0) {
    DevBuf<uint32_t> scratch;
    scratch.resize(nl[1] ? 32 * (size_t)nl[1] : 1);
    if (split)
      k_ham_finish_long<S, true><<<(unsigned)nl[0], kLongThreads, 0, s>>>(hv, ints, rows, list.p, scratch.p, parts.p, rowptr.p,
                                                                  col.p, d64, dhi, dlo);
    else
      k_ham_finish_long<S, false><<<(unsigned)nl[0], kLongThreads, 0, s>>>(hv, ints, rows, list.p, scratch.p, parts.p,
                                                                   rowptr.p, col.p, d64, dhi, dlo);
    SHCI_LAUNCH_CHECK();
  }
  pt.mark("ham finish");
  return total;
}
static int64_t emit_rows(const Helpers& hp, const uint32_t* rows, size_t nr, const IntsView& ints, Csr& out, bool want64,
                         bool want32, bool want_lo, Prims& pr, cudaStream_t s, PhaseTimer& pt) {
  return hp.narrow ? emit_rows_as<uint32_t>(hp, rows, nr, ints, out, want64, want32, want_lo, pr, s, pt)
                   : emit_rows_as<uint64_t>(hp, rows, nr, ints, out, want64, want32, want_lo, pr, s, pt);
}

// Positions of the determinants [r0, r1), ascending: flags, and after their
// scan the positions themselves (and their determinants).
__global__ void k_range_flags(const uint32_t* __restrict__ perm, size_t n, uint32_t r0, uint32_t r1,
                              int64_t* __restrict__ flag) {
  for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) {
    const uint32_t d = perm[i];
    flag[i] = (d >= r0 && d < r1) ? 1 : 0;
  }
}
__global__ void k_range_fill(const uint32_t* __restrict__ perm, size_t n, uint32_t r0, uint32_t r1,
                             const int64_t* __restrict__ pos, uint32_t* __restrict__ where,
                             uint32_t* __restrict__ which) {
  for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) {
    const uint32_t d = perm[i];
    if (d >= r0 && d < r1) {
      where[pos[i]] = (uint32_t)i;
      if (which) which[pos[i]] = d;
    }
  }
}

// Incremental build helpers. The rows of the new determinants R >= n_old are
// emitted in full (in storage order, columns in the new storage order);
// their entries whose column is an old determinant C < n_old are the new
// columns of old row C: an element is bit for bit the same with either of its
// determinants as the ket.
// Bit x of `old` = storage position x holds an old determinant (index < n_old).
__global__ void k_old_bits(const uint32_t* __restrict__ perm, int64_t N, int64_t n_old, uint32_t* __restrict__ old) {
  const int64_t nw = (N + 31) >> 5;
  for (int64_t w = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; w < nw; w += (int64_t)gridDim.x * blockDim.x) {
    uint32_t m = 0;
    for (int b = 0; b < 32 && (w << 5) + b < N; ++b) m |= ((int64_t)perm[(w << 5) + b] < n_old ? 1u : 0u) << b;
    old[w] = m;
  }
}
__device__ __forceinline__ bool is_old(const uint32_t* __restrict__ old, uint32_t x) {
  return (__ldg(old + (x >> 5)) >> (x & 31)) & 1u;
}
// New columns of the old rows, indexed by the old row's new storage position
// (the new rows' columns are storage positions already).
__global__ void k_delta_count(const int64_t* __restrict__ rp_new, size_t nr, const int32_t* __restrict__ col_new,
                              const uint32_t* __restrict__ old, unsigned long long* __restrict__ dcnt) {
  const int lane = threadIdx.x & 31;
  const int64_t warps = (int64_t)gridDim.x * (blockDim.x >> 5);
  for (int64_t r = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5; r < (int64_t)nr; r += warps)
    for (int64_t p = rp_new[r] + lane; p < rp_new[r + 1]; p += 32) {
      const uint32_t c = (uint32_t)col_new[p];
      if (is_old(old, c)) atomicAdd(&dcnt[c], 1ull);
    }
}
// The old row at storage position c receives column rows[r].
__global__ void k_delta_fill(const int64_t* __restrict__ rp_new, size_t nr, CsrVals nv,
                             const uint32_t* __restrict__ old, const uint32_t* __restrict__ rows,
                             const int64_t* __restrict__ dptr, unsigned long long* __restrict__ dfill, CsrVals dv) {
  const int lane = threadIdx.x & 31;
  const int64_t warps = (int64_t)gridDim.x * (blockDim.x >> 5);
  for (int64_t r = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5; r < (int64_t)nr; r += warps) {
    const int32_t me = (int32_t)rows[r];
    for (int64_t p = rp_new[r] + lane; p < rp_new[r + 1]; p += 32) {
      const uint32_t c = (uint32_t)nv.col[p];
      if (!is_old(old, c)) continue;
      const int64_t q = dptr[c] + (int64_t)atomicAdd(&dfill[c], 1ull);
      dv.col[q] = me;
      if (dv.v64) dv.v64[q] = nv.v64[p];
      if (dv.vhi) dv.vhi[q] = nv.vhi[p];
      if (dv.vlo) dv.vlo[q] = nv.vlo[p];
    }
  }
}
// rel[o] = new storage position of the determinant at old storage position o.
// Both orders sort by the same key, so rel is increasing.
__global__ void k_relabel(const uint32_t* __restrict__ perm_old, const uint32_t* __restrict__ spos, int64_t n_old,
                          uint32_t* __restrict__ rel) {
  for (int64_t o = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; o < n_old; o += (int64_t)gridDim.x * blockDim.x)
    rel[o] = spos[perm_old[o]];
}
__global__ void k_merged_len(const uint32_t* __restrict__ perm, const uint32_t* __restrict__ spos_old,
                             const int64_t* __restrict__ rp_old, const int64_t* __restrict__ dptr, int64_t n_old,
                             const int64_t* __restrict__ rp_new, const int64_t* __restrict__ slot, int64_t N,
                             int64_t* __restrict__ len) {
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < N; i += (int64_t)gridDim.x * blockDim.x) {
    const int64_t u = perm[i];
    if (u < n_old) {
      const int64_t o = spos_old[u];
      len[i] = (rp_old[o + 1] - rp_old[o]) + (dptr[i + 1] - dptr[i]);
    } else {
      len[i] = rp_new[slot[i] + 1] - rp_new[slot[i]];
    }
  }
}

// Number of lanes whose v (ascending across the warp) is below key.
__device__ __forceinline__ int warp_rank(uint32_t key, uint32_t v) {
  int r = 0;
#pragma unroll
  for (int st = 16; st >= 1; st >>= 1) {
    const uint32_t t = __shfl_sync(kFull, v, r + st - 1);
    if (t < key) r += st;
  }
  const uint32_t last = __shfl_sync(kFull, v, 31);
  if (r == 31 && last < key) r = 32;
  return r;
}

// Merged row at storage position i, warp per row. An old determinant's row is
// its old row A with columns relabelled (still sorted: the relabelling is
// increasing) merged with its new columns B (sorted; disjoint from A), 32
// outputs a step: the next 32 entries of A and of B are ranked against each
// other by shuffles, and those among the 32 smallest of the 64 (the next 32
// of the merged row) are written; the rest are taken up again next step. A
// new determinant's row is copied from the new rows.
// VK: 0 = FP64 values, 1 = FP32 head + tail.
template <int VK>
struct MergeVal;
template <>
struct MergeVal<0> {
  double v;
  __device__ void load(const double* v64, const float*, const float*, int64_t p) { v = v64[p]; }
  __device__ void store(double* v64, float*, float*, int64_t q) const { v64[q] = v; }
};
template <>
struct MergeVal<1> {
  float h, l;
  __device__ void load(const double*, const float* hi, const float* lo, int64_t p) {
    h = hi[p];
    l = lo[p];
  }
  __device__ void store(double*, float* hi, float* lo, int64_t q) const {
    hi[q] = h;
    lo[q] = l;
  }
};
template <int VK>
__global__ void __launch_bounds__(256) k_merge_rows(const uint32_t* __restrict__ perm,
                                                    const uint32_t* __restrict__ spos_old,
                                                    const int64_t* __restrict__ rp_old, CsrVals ov,
                                                    const uint32_t* __restrict__ rel,
                                                    const int64_t* __restrict__ dptr, CsrVals dv,
                                                    const int64_t* __restrict__ rp_new, CsrVals nv,
                                                    const int64_t* __restrict__ slot, int64_t n_old, int64_t N, const int64_t* __restrict__ rp, CsrVals out) {
  const int lane = threadIdx.x & 31;
  const int64_t warps = (int64_t)gridDim.x * (blockDim.x >> 5);
  int32_t* __restrict__ ocol = out.col;
  double* __restrict__ o64 = out.v64;
  float* __restrict__ ohi = out.vhi;
  float* __restrict__ olo = out.vlo;
  constexpr uint32_t kNone = 0xffffffffu;  // above every storage position
  for (int64_t i = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5; i < N; i += warps) {
    const int64_t d = rp[i];
    const int64_t u = perm[i];
    if (u >= n_old) {  // a new row: copied
      const int64_t a0 = rp_new[slot[i]], la = rp_new[slot[i] + 1] - a0;
      for (int64_t t = lane; t < la; t += 32) {
        MergeVal<VK> v;
        v.load(nv.v64, nv.vhi, nv.vlo, a0 + t);
        ocol[d + t] = nv.col[a0 + t];
        v.store(o64, ohi, olo, d + t);
      }
      continue;
    }
    const int64_t o = spos_old[u];
    const int64_t a0 = rp_old[o], la = rp_old[o + 1] - a0;
    const int64_t b0 = dptr[i], lb = dptr[i + 1] - b0;
    if (lb == 0) {  // no new columns: the old row relabelled
      for (int64_t t = lane; t < la; t += 32) {
        MergeVal<VK> v;
        v.load(ov.v64, ov.vhi, ov.vlo, a0 + t);
        ocol[d + t] = (int32_t)rel[ov.col[a0 + t]];
        v.store(o64, ohi, olo, d + t);
      }
      continue;
    }
    int64_t ia = 0, ib = 0;
    while (ia < la || ib < lb) {
      const bool va = ia + lane < la, vb = ib + lane < lb;
      const uint32_t ka = va ? rel[ov.col[a0 + ia + lane]] : kNone;
      const uint32_t kb = vb ? (uint32_t)dv.col[b0 + ib + lane] : kNone;
      const int pa = lane + warp_rank(ka, kb);  // position among the 64 of this step
      const int pb = lane + warp_rank(kb, ka);
      const bool ea = va && pa < 32, eb = vb && pb < 32;
      const int64_t base = d + ia + ib;
      if (ea) {
        MergeVal<VK> v;
        v.load(ov.v64, ov.vhi, ov.vlo, a0 + ia + lane);
        ocol[base + pa] = (int32_t)ka;
        v.store(o64, ohi, olo, base + pa);
      }
      if (eb) {
        MergeVal<VK> w;
        w.load(dv.v64, dv.vhi, dv.vlo, b0 + ib + lane);
        ocol[base + pb] = (int32_t)kb;
        w.store(o64, ohi, olo, base + pb);
      }
      ia += __popc(__ballot_sync(kFull, ea));
      ib += __popc(__ballot_sync(kFull, eb));
    }
  }
}

void build_ham_csr(const Helpers& hp, const IntsView& ints, Csr& H, bool want64, bool want32, bool want_lo,
                   size_t n_old, Prims& pr, cudaStream_t s) {
  const size_t N = hp.N;
  PhaseTimer pt(s);
  // A step that at least doubles the space is rebuilt; one that adds nothing is left as it is (below). Extended /
  // rebuilt by new per old determinant, mixed form: to 402,058 determinants 0.25 19.4 / 24.1 ms, 0.5 25.3 / 24.1,
  // 0.95 27.3 / 24.1, 1.2 31.0 / 24.1; to 150,924 of 36 orbitals 0.25 10.3 / 12.0, 0.5 12.4 / 12.0; to 30,666
  // 0.25 2.45 / 1.98. From the line on a rebuild is the faster at every size; below it an extension is up to a fifth
  // faster (large spaces, to 0.4) and costs up to a sixth more (0.5 to 1), or 0.9 ms (small spaces).
  const bool incremental = !H.block && n_old > 0 && n_old < N && N - n_old < n_old && H.N == n_old &&
                           H.perm.n >= n_old && (want64 ? !want32 : (want32 && want_lo)) &&
                           (H.v64.p != nullptr) == want64 && (H.vhi.p != nullptr) == want32 &&
                           (H.vlo.p != nullptr) == (want32 && want_lo);
  if (!incremental) {
    if (n_old == N && H.N == N && !H.block) return;  // nothing new
    const int64_t nnz = emit_rows(hp, nullptr, N, ints, H, want64, want32, want_lo, pr, s, pt);
    H.clear_block();
    H.perm.resize(N > 0 ? N : 1);
    H.spos.resize(N > 0 ? N : 1);
    if (N) {
      SHCI_CUDA(cudaMemcpyAsync(H.perm.p, hp.perm.p, N * sizeof(uint32_t), cudaMemcpyDeviceToDevice, s));
      SHCI_CUDA(cudaMemcpyAsync(H.spos.p, hp.spos.p, N * sizeof(uint32_t), cudaMemcpyDeviceToDevice, s));
    }
    H.nnz = nnz;
    H.N = N;
    SHCI_CUDA(cudaStreamSynchronize(s));
    return;
  }
  const size_t nr = N - n_old;
  const DevBuf<uint32_t>&perm = hp.perm, &spos = hp.spos;
  // the new determinants' storage positions, ascending, and each one's row among them
  DevBuf<int64_t> flag, slot;
  DevBuf<uint32_t> rows;
  flag.resize(N);
  slot.resize(N);
  rows.resize(nr);
  k_range_flags<<<grid_for(N, 256), 256, 0, s>>>(perm.p, N, (uint32_t)n_old, (uint32_t)N, flag.p);
  SHCI_LAUNCH_CHECK();
  scan_exclusive_i64(flag.p, slot.p, N, nullptr, pr, s);
  k_range_fill<<<grid_for(N, 256), 256, 0, s>>>(perm.p, N, (uint32_t)n_old, (uint32_t)N, slot.p, rows.p, nullptr);
  SHCI_LAUNCH_CHECK();
  Csr Hn;  // rows of the determinants n_old .. N-1, in storage order
  Hn.nnz = emit_rows(hp, rows.p, nr, ints, Hn, want64, want32, want_lo, pr, s, pt);
  CsrVals nv{Hn.col.p, Hn.v64.p, Hn.vhi.p, Hn.vlo.p};
  // new columns of the old rows, indexed by the old row's new storage position
  DevBuf<uint32_t> oldbits;
  oldbits.resize((N + 31) / 32);
  k_old_bits<<<grid_for((N + 31) / 32, 256), 256, 0, s>>>(perm.p, (int64_t)N, (int64_t)n_old, oldbits.p);
  SHCI_LAUNCH_CHECK();
  DevBuf<unsigned long long> dcnt, dfill;
  dcnt.resize(N);
  dfill.resize(N);
  SHCI_CUDA(cudaMemsetAsync(dcnt.p, 0, N * sizeof(unsigned long long), s));
  SHCI_CUDA(cudaMemsetAsync(dfill.p, 0, N * sizeof(unsigned long long), s));
  const unsigned wblocks = grid_for(nr * 32, 256, 152 * 16);
  k_delta_count<<<wblocks, 256, 0, s>>>(Hn.rowptr.p, nr, Hn.col.p, oldbits.p, dcnt.p);
  SHCI_LAUNCH_CHECK();
  DevBuf<int64_t> dptr;
  dptr.resize(N + 1);
  int64_t dtotal = 0;
  scan_exclusive_i64(reinterpret_cast<const int64_t*>(dcnt.p), dptr.p, N, &dtotal, pr, s);
  k_set_last<<<1, 1, 0, s>>>(dptr.p, (int64_t)N, dtotal);
  SHCI_LAUNCH_CHECK();
  Csr Hd;
  const size_t dcap = dtotal > 0 ? (size_t)dtotal : 1;
  Hd.col.resize(dcap);
  if (want64) Hd.v64.resize(dcap);
  if (want32) Hd.vhi.resize(dcap);
  if (want32 && want_lo) Hd.vlo.resize(dcap);
  CsrVals dv{Hd.col.p, Hd.v64.p, Hd.vhi.p, Hd.vlo.p};
  k_delta_fill<<<wblocks, 256, 0, s>>>(Hn.rowptr.p, nr, nv, oldbits.p, rows.p, dptr.p, dfill.p, dv);
  SHCI_LAUNCH_CHECK();
  sort_rows(dptr.p, N, dv, s);
  pt.mark("ham new columns");
  // merge in the new storage order
  DevBuf<uint32_t> rel;
  rel.resize(n_old);
  k_relabel<<<grid_for(n_old, 256), 256, 0, s>>>(H.perm.p, spos.p, (int64_t)n_old, rel.p);
  SHCI_LAUNCH_CHECK();
  DevBuf<int64_t> len, rp;
  len.resize(N);
  rp.resize(N + 1);
  k_merged_len<<<grid_for(N, 256), 256, 0, s>>>(perm.p, H.spos.p, H.rowptr.p, dptr.p, (int64_t)n_old, Hn.rowptr.p,
                                                slot.p, (int64_t)N, len.p);
  SHCI_LAUNCH_CHECK();
  int64_t total = 0;
  scan_exclusive_i64(len.p, rp.p, N, &total, pr, s);
  k_set_last<<<1, 1, 0, s>>>(rp.p, (int64_t)N, total);
  SHCI_LAUNCH_CHECK();
  Csr M;
  const size_t cap = total > 0 ? (size_t)total : 1;
  M.col.resize(cap);
  if (want64) M.v64.resize(cap);
  if (want32) M.vhi.resize(cap);
  if (want32 && want_lo) M.vlo.resize(cap);
  CsrVals ov{H.col.p, H.v64.p, H.vhi.p, H.vlo.p}, mv{M.col.p, M.v64.p, M.vhi.p, M.vlo.p};
  if (want64)
    k_merge_rows<0><<<grid_for(N * 32, 256, 152 * 16), 256, 0, s>>>(perm.p, H.spos.p, H.rowptr.p, ov, rel.p,
                                                                    dptr.p, dv, Hn.rowptr.p, nv, slot.p, (int64_t)n_old,
                                                                    (int64_t)N, rp.p, mv);
  else
    k_merge_rows<1><<<grid_for(N * 32, 256, 152 * 16), 256, 0, s>>>(perm.p, H.spos.p, H.rowptr.p, ov, rel.p,
                                                                    dptr.p, dv, Hn.rowptr.p, nv, slot.p, (int64_t)n_old,
                                                                    (int64_t)N, rp.p, mv);
  SHCI_LAUNCH_CHECK();
  DevBuf<uint32_t> nperm, nspos;
  nperm.resize(N);
  nspos.resize(N);
  SHCI_CUDA(cudaMemcpyAsync(nperm.p, perm.p, N * sizeof(uint32_t), cudaMemcpyDeviceToDevice, s));
  SHCI_CUDA(cudaMemcpyAsync(nspos.p, spos.p, N * sizeof(uint32_t), cudaMemcpyDeviceToDevice, s));
  SHCI_CUDA(cudaStreamSynchronize(s));
  H.rowptr.swap(rp);
  H.col.swap(M.col);
  H.v64.swap(M.v64);
  H.vhi.swap(M.vhi);
  H.vlo.swap(M.vlo);
  H.perm.swap(nperm);
  H.spos.swap(nspos);
  H.N = N;
  H.nnz = total;
  pt.mark("ham merge");
}

// ---------------------------------------------------------------------------
// Row block: one rank's share of the Hamiltonian in the sharded path, the full
// rows of the determinants [r0, r1) with every column. Local rows are those
// determinants in storage order (alpha-major, as in the whole matrix);
// H.perm[r] is the determinant of local row r, H.xpos[r] its storage position
// (where its own x sits for the diagonal term) and H.xperm the whole storage
// order (storage position -> determinant), through which x is packed. Columns
// are storage positions of the whole space. A row's entries and their order
// are those of the same row in the whole matrix.
// ---------------------------------------------------------------------------
void build_ham_block(const Helpers& hp, const IntsView& ints, Csr& H, bool want64, bool want32, bool want_lo,
                     size_t r0, size_t r1, Prims& pr, cudaStream_t s) {
  const size_t N = hp.N;
  if (!(r0 < r1 && r1 <= N)) throw Error(kErrInvalid, "row block [r0, r1) must be a non-empty range of the space");
  const size_t nb = r1 - r0;
  PhaseTimer pt(s);
  DevBuf<int64_t> flag, pos;
  flag.resize(N);
  pos.resize(N);
  k_range_flags<<<grid_for(N, 256), 256, 0, s>>>(hp.perm.p, N, (uint32_t)r0, (uint32_t)r1, flag.p);
  SHCI_LAUNCH_CHECK();
  int64_t nflag = 0;
  scan_exclusive_i64(flag.p, pos.p, N, &nflag, pr, s);
  if ((size_t)nflag != nb) throw Error(kErrState, "row block: storage order lost determinants");
  DevBuf<uint32_t> rows, xpos;
  rows.resize(nb);
  xpos.resize(nb);
  k_range_fill<<<grid_for(N, 256), 256, 0, s>>>(hp.perm.p, N, (uint32_t)r0, (uint32_t)r1, pos.p, xpos.p, rows.p);
  SHCI_LAUNCH_CHECK();
  pt.mark("ham block order");
  H.drop_compressed();
  H.nnz = emit_rows(hp, xpos.p, nb, ints, H, want64, want32, want_lo, pr, s, pt);
  H.xperm.resize(N);
  SHCI_CUDA(cudaMemcpyAsync(H.xperm.p, hp.perm.p, N * sizeof(uint32_t), cudaMemcpyDeviceToDevice, s));
  SHCI_CUDA(cudaStreamSynchronize(s));
  H.perm.swap(rows);
  H.xpos.swap(xpos);
  H.spos.release();
  H.N = nb;
  H.nfull = N;
  H.row0 = r0;
  H.block = true;
}

// ---------------------------------------------------------------------------
// Diagonal energies: thread per determinant, Direct/Exchange in shared memory.
// ---------------------------------------------------------------------------
__global__ void k_diag(const Det2* __restrict__ dets, size_t n, IntsView ints, double* __restrict__ diag) {
  extern __shared__ double sm[];
  const int nn = ints.norb * ints.norb;
  double* sD = sm;
  double* sX = sm + nn;
  for (int j = threadIdx.x; j < nn; j += blockDim.x) {
    sD[j] = ints.Direct[j];
    sX[j] = ints.Exchange[j];
  }
  __syncthreads();
  for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x)
    diag[i] = det_energy(ints, dets[i], sD, sX);
}

void compute_diag(const Det2* dets, size_t n, const IntsView& ints, double* diag, cudaStream_t s) {
  if (n == 0) return;
  size_t smem = 2 * sizeof(double) * ints.norb * ints.norb;
  SHCI_CUDA(cudaFuncSetAttribute(k_diag, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  k_diag<<<grid_for(n, 128, 152 * 8), 128, smem, s>>>(dets, n, ints, diag);
  SHCI_LAUNCH_CHECK();
}

// ---------------------------------------------------------------------------
// Matrix-free sigma (HmultDirect, SHCI/Hmult.h:241-381): y[I] = diag[I] x[I] +
// sum_J H_IJ x[J], row I's connections found by visit_row and H_IJ recomputed.
// Hits wait per warp in three queues (singles, alpha-beta doubles, doubles of
// one spin) and are evaluated on full warps, one element formula at a time, on
// strings read by position. x is in storage order: the hits of a scan are
// neighbours there. FP64: the reference's arithmetic. FP32 (the first stage of
// the mixed matrix-free path): FP32 integrals, FP32 elements, compensated FP32
// accumulation of h * x.
// Bound by instruction issue (61 %) and latency at 28 warps per SM. 100,762
// determinants of 36 orbitals, 1.1e8 connections, 4 vectors: 6.65 ms with a
// generic element routine and 64-bit decoding per hit, now 3.21 ms.
// ---------------------------------------------------------------------------
template <class S, int K, bool F32>
struct DirectVisitor {
  using T = typename Elem<F32>::T;
  const HelperView<S>& h;
  const IntsView& ints;
  S A, B;
  const T* x;  // [N][K]
  uint32_t* q;  // three queues of 64: singles, alpha-beta doubles, doubles of one spin
  int ns, nd, nm;
  Acc a32[F32 ? K : 1];
  double a64[F32 ? 1 : K];

  __device__ __forceinline__ void load(T (&v)[K], uint32_t p) const {
    if constexpr (K == 1) {
      v[0] = __ldg(x + p);
    } else if constexpr (F32 && K == 2) {
      const float2 t = __ldg(reinterpret_cast<const float2*>(x) + p);
      v[0] = t.x;
      v[1] = t.y;
    } else if constexpr (F32) {
      const float4 t = __ldg(reinterpret_cast<const float4*>(x) + p);
      v[0] = t.x;
      v[1] = t.y;
      v[2] = t.z;
      v[3] = t.w;
    } else {
#pragma unroll
      for (int r = 0; r < K; r += 2) {
        const double2 t = __ldg(reinterpret_cast<const double2*>(x + (size_t)p * K + r));
        v[r] = t.x;
        v[r + 1] = t.y;
      }
    }
  }
  template <int which>
  __device__ __forceinline__ T element(const typename StrPair<S>::T& J) const {
    if constexpr (which == 0) {
      const bool beta = J.x == A;
      return elem_single<F32, S>(ints, A, B, beta ? B : A, beta ? J.y : J.x, beta);
    } else if constexpr (which == 1) {
      return elem_ab<F32, S>(ints, A, B, J.x, J.y);
    } else {
      const bool beta = J.x == A;
      return elem_same<F32, S>(ints, beta ? B : A, beta ? A : B, beta ? J.y : J.x, beta);
    }
  }
  __device__ __forceinline__ void add(T hv, const T (&xv)[K]) {
#pragma unroll
    for (int r = 0; r < K; ++r) {
      if constexpr (F32)
        acc_add(a32[r], hv, xv[r]);
      else
        a64[r] += hv * xv[r];
    }
  }
  template <int which>
  __device__ __forceinline__ void one(uint32_t p) {
    T xv[K];
    load(xv, p);
    add(element<which>(h.str[p]), xv);
  }
  template <int which>
  __device__ __forceinline__ int drain(uint32_t* w, int n) {  // the first 32 of n entries, 32 <= n < 64
    const int lane = threadIdx.x & 31;
    __syncwarp();
    one<which>(w[lane]);
    const uint32_t v = w[32 + lane];
    __syncwarp();
    if (lane < n - 32) w[lane] = v;
    return n - 32;
  }
  template <int part>
  __device__ __forceinline__ void step(bool hit, bool single, uint32_t p) {
    const unsigned lt = (1u << (threadIdx.x & 31)) - 1u;
    if (part != kSameBeta) {  // no single excitation there
      const unsigned ms = __ballot_sync(kFull, hit && single);
      if (ms) {
        if (hit && single) q[ns + __popc(ms & lt)] = p;
        ns += __popc(ms);
        if (ns >= 32) ns = drain<0>(q, ns);
      }
    }
    const unsigned md = __ballot_sync(kFull, hit && !single);
    if (part == kAlphaMoved) {
      if (hit && !single) q[64 + nd + __popc(md & lt)] = p;
      nd += __popc(md);
      if (nd >= 32) nd = drain<1>(q + 64, nd);
    } else {
      if (hit && !single) q[128 + nm + __popc(md & lt)] = p;
      nm += __popc(md);
      if (nm >= 32) nm = drain<2>(q + 128, nm);
    }
  }
  __device__ __forceinline__ void flush() {
    const int lane = threadIdx.x & 31;
    __syncwarp();
    if (lane < ns) one<0>(q[lane]);
    if (lane < nd) one<1>(q[64 + lane]);
    if (lane < nm) one<2>(q[128 + lane]);
  }
};

// A warp per row, four rows a block and as many blocks as rows need: the
// rows' work differs by two orders of magnitude (the lowest determinant's row
// holds 29,219 of 100,000 columns), and the block scheduler evens it out.
constexpr int kDirThreads = 128;
template <class S, int K, bool F32>
__global__ void __launch_bounds__(kDirThreads, 8)
    k_sigma_direct(HelperView<S> h, IntsView ints, const uint32_t* __restrict__ perm, const double* __restrict__ diag,
                   const typename Elem<F32>::T* __restrict__ x, int kw, double* __restrict__ y, size_t ldy) {
  __shared__ uint32_t s_q[kDirThreads / 32][192];
  const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
  const size_t p = (size_t)blockIdx.x * (kDirThreads / 32) + wib;
  if (p >= h.N) return;
  const auto I = h.str[p];
  DirectVisitor<S, K, F32> v{h, ints, I.x, I.y, x, s_q[wib], 0, 0, 0, {}, {}};
  visit_row<S>(h, (uint32_t)p, I.x, I.y, v);
  v.flush();
  const size_t o = perm[p];
  const double dg = diag[o];
#pragma unroll
  for (int r = 0; r < K; ++r) {
    double t;
    if constexpr (F32) {
      Acc a = v.a32[r];
      // merge in lane order (a fixed tree); FP64 diagonal term
#pragma unroll
      for (int b = 16; b; b >>= 1) {
        Acc other{__shfl_xor_sync(kFull, a.s, b), __shfl_xor_sync(kFull, a.c, b)};
        if ((lane & b) == 0) {
          acc_merge(a, other);
        } else {
          acc_merge(other, a);
          a = other;
        }
      }
      t = (double)a.s + (double)a.c;
    } else {
      t = v.a64[r];
#pragma unroll
      for (int b = 16; b; b >>= 1) t += __shfl_xor_sync(kFull, t, b);
    }
    if (lane == 0 && r < kw) y[(size_t)r * ldy + o] = dg * (double)x[p * K + r] + t;
  }
}

template <class S, bool F32>
static void launch_direct(const Helpers& hp, const IntsView& ints, const double* diag,
                          const typename Elem<F32>::T* x, int k, int kw, double* y, size_t ldy, cudaStream_t s) {
  if (hp.N == 0) return;
  HelperView<S> hv = hp.view<S>();
  const unsigned blocks = (unsigned)((hp.N + kDirThreads / 32 - 1) / (kDirThreads / 32));
  switch (k) {
    case 1: k_sigma_direct<S, 1, F32><<<blocks, kDirThreads, 0, s>>>(hv, ints, hp.perm.p, diag, x, kw, y, ldy); break;
    case 2: k_sigma_direct<S, 2, F32><<<blocks, kDirThreads, 0, s>>>(hv, ints, hp.perm.p, diag, x, kw, y, ldy); break;
    case 4: k_sigma_direct<S, 4, F32><<<blocks, kDirThreads, 0, s>>>(hv, ints, hp.perm.p, diag, x, kw, y, ldy); break;
    default: throw Error(kErrInvalid, "direct sigma supports k in {1,2,4}");
  }
  SHCI_LAUNCH_CHECK();
}
void sigma_direct(const Helpers& hp, const IntsView& ints, const double* diag, const double* x, int k, int kw,
                  double* y, size_t ldy, cudaStream_t s) {
  if (hp.narrow)
    launch_direct<uint32_t, false>(hp, ints, diag, x, k, kw, y, ldy, s);
  else
    launch_direct<uint64_t, false>(hp, ints, diag, x, k, kw, y, ldy, s);
}
void sigma_direct32(const Helpers& hp, const IntsView& ints, const double* diag, const float* x, int k, int kw,
                    double* y, size_t ldy, cudaStream_t s) {
  if (!ints.I1f || !ints.I2f) throw Error(kErrState, "FP32 integrals missing");
  if (hp.narrow)
    launch_direct<uint32_t, true>(hp, ints, diag, x, k, kw, y, ldy, s);
  else
    launch_direct<uint64_t, true>(hp, ints, diag, x, k, kw, y, ldy, s);
}

}  // namespace shci
