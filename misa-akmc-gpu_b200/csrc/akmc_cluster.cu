// akmc_cluster.cu -- Cu cluster statistics of a job's resident lattice.
//
// The isolated-Cu count of MEventHook::onStepFinished (profiles/m_event_hook.cpp:17-55: a Cu
// atom none of whose 8 first neighbours is Cu) and the Cu cluster-size histogram by 1nn
// connectivity, on the device, so that a run can sample them every few rounds without
// copying the lattice out.
//
//   k_cu_bits     one pass over the occupancy bytes (32 sites a thread, two 16-byte loads) into a
//                 bit per site: the only pass over the whole lattice.  33.5 MB in 7.8 us out of L2,
//                 where a sampled lattice mostly lies, in 9.0 from DRAM (4.1 TB/s).
//   k_cu_classify 32 sites a thread from their own bits and those of the seven rows around: the Cu
//                 atoms without a Cu first neighbour are counted, the others are listed and start
//                 as their own roots.  All in L2 (a bit a site).
//   k_cu_union    per listed site, each Cu bond to a higher site id is merged into one set
//                 (lock-free union-find: the larger root is hooked under the smaller with a CAS,
//                 finds halve their paths).
//   k_cu_hist     per listed site, +1 on its root's size, and the root moves on in the histogram:
//                 out of the bin of the size it had, into the bin of the size it has.
// At dilute concentrations nine Cu atoms in ten are isolated, and only the rest is written to the
// scattered list, parent and size entries.  33.5 M sites, 1.34 % Cu: collecting every Cu atom and
// testing its neighbours byte by byte took 56 + 35 us, sizes and histogram 15 + 18 us, the whole
// call 165 us; now 8 + 15 us, 11 us for the union, 8 us for the histogram, and the call 61 us.
// The partition, hence every count, does not depend on the order the threads run in.
#include <algorithm>
#include <cstdint>

#include "akmc_device.h"

namespace akmc {
namespace {

constexpr unsigned kFull = 0xffffffffu;
constexpr int kCuCode = AKMC_CU;
constexpr int kFindLimit = 1 << 24;   // a find walks at most the set's size; the bound only guards
constexpr int kUnionLimit = 1 << 20;  // CAS retries; each failure means another hook succeeded

__device__ __forceinline__ int64_t nn1_site(int64_t s, int b, int sx, int sy, int sz) {
  const int X = static_cast<int>(s % sx);
  const int64_t t = s / sx;
  const int y = static_cast<int>(t % sy), z = static_cast<int>(t / sy);
  const int p = X & 1;
  int gx = X + ((b & 4) ? 1 : -1);
  int gy = y + ((b >> 1) & 1) - 1 + p;
  int gz = z + (b & 1) - 1 + p;
  gx = gx < 0 ? gx + sx : (gx >= sx ? gx - sx : gx);
  gy = gy < 0 ? gy + sy : (gy >= sy ? gy - sy : gy);
  gz = gz < 0 ? gz + sz : (gz >= sz ? gz - sz : gz);
  return gx + static_cast<int64_t>(sx) * (gy + static_cast<int64_t>(sy) * gz);
}

// Mask with bit 7 of every byte of w that equals the Cu code (exact per byte: no borrow
// crosses a byte boundary).
__device__ __forceinline__ uint32_t cu_bytes(uint32_t w) {
  const uint32_t x = w ^ (0x01010101u * kCuCode);
  return ~(((x & 0x7F7F7F7Fu) + 0x7F7F7F7Fu) | x | 0x7F7F7F7Fu);
}

// Bit k of the result: byte k of w holds the Cu code.
__device__ __forceinline__ uint32_t cu_nibble(uint32_t w) { return (((cu_bytes(w) >> 7) & 0x01010101u) * 0x10204080u) >> 28; }
__device__ __forceinline__ uint32_t cu_16(const uint4& v) {
  return cu_nibble(v.x) | cu_nibble(v.y) << 4 | cu_nibble(v.z) << 8 | cu_nibble(v.w) << 12;
}

// Word w of the bits: sites 32 k .. 32 k + 31 of row w / wpr, k = w mod wpr.  The row's last word reaches at most 31
// sites into the halo (kHaloR = 32), whose bits are left out.  Block 0 clears what the later kernels count in.
__global__ void k_cu_bits(const uint8_t* __restrict__ occ, int nwords, int wpr, int sx, int px, uint32_t* __restrict__ bits,
                          unsigned long long* misc, int nmisc) {
  if (blockIdx.x == 0)
    for (int k = threadIdx.x; k < nmisc; k += blockDim.x) misc[k] = 0;
  for (int w = blockIdx.x * blockDim.x + threadIdx.x; w < nwords; w += gridDim.x * blockDim.x) {
    const int row = w / wpr, k = w - row * wpr;
    const uint4* p = reinterpret_cast<const uint4*>(occ + static_cast<int64_t>(row) * px + kHaloL + 32 * k);
    const uint4 v0 = __ldg(p), v1 = __ldg(p + 1);
    const int valid = sx - 32 * k;
    bits[w] = (cu_16(v0) | cu_16(v1) << 16) & (valid < 32 ? (1u << valid) - 1u : kFull);
  }
}

// An even site's first neighbours are x -+ 1 in the rows (y - 1 | y, z - 1 | z), an odd one's in (y | y + 1,
// z | z + 1); x +- 1 is of the other parity.  So the even sites of a word test the union E of four rows' words,
// moved one site either way, and the odd ones the union O of four: only the site below the word (odd) is missing
// from E, only the one above (even) from O.  kWords words a thread and round, one global slot request a block.
constexpr int kClassWords = 2;
__global__ void __launch_bounds__(256) k_cu_classify(const uint32_t* __restrict__ bits, int nwords, int wpr, int sx, int sy,
                                                     int sz, int32_t* list, unsigned int* n_list, int32_t* parent,
                                                     int32_t* size, unsigned long long* iso) {
  __shared__ unsigned int s_cnt, s_base, s_iso;
  unsigned int isolated = 0;
  if (threadIdx.x == 0) s_iso = 0;
  const int chunk = static_cast<int>(blockDim.x) * kClassWords;
  for (int w0 = blockIdx.x * chunk; w0 < nwords; w0 += gridDim.x * chunk) {  // alike in every thread of the block
    if (threadIdx.x == 0) s_cnt = 0;
    __syncthreads();
    uint32_t bonded[kClassWords];
    int cnt = 0;
#pragma unroll
    for (int q = 0; q < kClassWords; ++q) {
      const int w = w0 + q * static_cast<int>(blockDim.x) + static_cast<int>(threadIdx.x);
      const int wc = min(w, nwords - 1);  // every load is issued: the word alone is not waited for
      const uint32_t own = w < nwords ? __ldg(bits + wc) : 0u;
      const int row = wc / wpr, k = wc - row * wpr;
      const int z = row / sy, y = row - z * sy;
      const int ym = y > 0 ? y - 1 : sy - 1, yp = y + 1 < sy ? y + 1 : 0;
      const int zm = z > 0 ? z - 1 : sz - 1, zp = z + 1 < sz ? z + 1 : 0;
      const int last = k == wpr - 1, end = (sx - 1) & 31;  // the row's last site is bit `end` of its last word
      const int kl = k > 0 ? k - 1 : wpr - 1, bl = k > 0 ? 31 : end;
      const int kr = last ? 0 : k + 1;
      const uint32_t* const r[7] = {bits + static_cast<int64_t>(wpr) * (ym + static_cast<int64_t>(sy) * zm),
                                    bits + static_cast<int64_t>(wpr) * (y + static_cast<int64_t>(sy) * zm),
                                    bits + static_cast<int64_t>(wpr) * (ym + static_cast<int64_t>(sy) * z),
                                    bits + static_cast<int64_t>(wpr) * row,
                                    bits + static_cast<int64_t>(wpr) * (yp + static_cast<int64_t>(sy) * z),
                                    bits + static_cast<int64_t>(wpr) * (y + static_cast<int64_t>(sy) * zp),
                                    bits + static_cast<int64_t>(wpr) * (yp + static_cast<int64_t>(sy) * zp)};
      const uint32_t e = __ldg(r[0] + k) | __ldg(r[1] + k) | __ldg(r[2] + k) | __ldg(r[3] + k);
      const uint32_t o = __ldg(r[3] + k) | __ldg(r[4] + k) | __ldg(r[5] + k) | __ldg(r[6] + k);
      const uint32_t below = (__ldg(r[0] + kl) | __ldg(r[1] + kl) | __ldg(r[2] + kl) | __ldg(r[3] + kl)) >> bl & 1u;
      const uint32_t above = (__ldg(r[3] + kr) | __ldg(r[4] + kr) | __ldg(r[5] + kr) | __ldg(r[6] + kr)) & 1u;
      const uint32_t near = ((e << 1 | below | e >> 1) & 0x55555555u) |
                            ((o << 1 | o >> 1 | above << (last ? end : 31)) & 0xaaaaaaaau);
      bonded[q] = own & near;
      isolated += __popc(own & ~near);
      cnt += __popc(bonded[q]);
    }
    unsigned int at = cnt ? atomicAdd(&s_cnt, static_cast<unsigned int>(cnt)) : 0u;
    __syncthreads();
    if (threadIdx.x == 0 && s_cnt) s_base = atomicAdd(n_list, s_cnt);
    __syncthreads();
    at += s_base;
#pragma unroll
    for (int q = 0; q < kClassWords; ++q) {
      if (!bonded[q]) continue;
      const int w = w0 + q * static_cast<int>(blockDim.x) + static_cast<int>(threadIdx.x);
      const int row = w / wpr, k = w - row * wpr;
      const int32_t s0 = static_cast<int32_t>(static_cast<int64_t>(row) * sx + 32 * k);
      for (uint32_t m = bonded[q]; m; m &= m - 1) {
        const int32_t s = s0 + __ffs(static_cast<int>(m)) - 1;
        parent[s] = s;
        size[s] = 0;
        list[at++] = s;
      }
    }
  }
  isolated = __reduce_add_sync(kFull, isolated);
  __syncthreads();
  if ((threadIdx.x & 31) == 0 && isolated) atomicAdd(&s_iso, isolated);
  __syncthreads();
  if (threadIdx.x == 0 && s_iso) atomicAdd(iso, static_cast<unsigned long long>(s_iso));
}

__device__ __forceinline__ int32_t find_root(int32_t* parent, int32_t x, unsigned int* status) {
  for (int it = 0; it < kFindLimit; ++it) {
    const int32_t p = __ldcg(parent + x);
    if (p == x) return x;
    const int32_t gp = __ldcg(parent + p);
    if (gp != p) atomicCAS(parent + x, p, gp);  // path halving; losing the race is harmless
    x = gp;
  }
  atomicOr(status, kErrTimeout);
  return x;
}

__global__ void k_cu_union(const uint8_t* __restrict__ occ, int sx, int sy, int sz, int px, const int32_t* list,
                           const unsigned int* n_list, int32_t* parent, unsigned int* status) {
  const int64_t n = *n_list;
  for (int64_t i = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x; i < n;
       i += static_cast<int64_t>(gridDim.x) * blockDim.x) {
    const int32_t s = list[i];
    unsigned cu = 0;  // bit b: first neighbour b is Cu, of a higher site id
#pragma unroll
    for (int b = 0; b < 8; ++b) {
      const int64_t r = nn1_site(s, b, sx, sy, sz);
      if (r > s && __ldg(occ + lattice_index(static_cast<int32_t>(r), sx, px)) == kCuCode) cu |= 1u << b;
    }
    for (; cu; cu &= cu - 1) {
      int32_t a = s, c = static_cast<int32_t>(nn1_site(s, __ffs(static_cast<int>(cu)) - 1, sx, sy, sz));
      int it = 0;
      for (; it < kUnionLimit; ++it) {
        a = find_root(parent, a, status);
        c = find_root(parent, c, status);
        if (a == c) break;
        if (a < c) {
          const int32_t t = a;
          a = c;
          c = t;
        }
        if (atomicCAS(parent + a, a, c) == a) break;  // root a now hangs under c
      }
      if (it == kUnionLimit) atomicOr(status, kErrTimeout);
    }
  }
}

// The lanes of a warp with the same root add once, through their leader: clusters may span the box.  Each block
// counts how the roots moved through the histogram (signed: a root may come in one block and leave in another); the
// sums are those of the final sizes.  The last block adds the isolated atoms, clusters of one, to their bin and
// writes the counts out.
__global__ void k_cu_hist(const int32_t* list, const unsigned int* n_list, int32_t* parent, int32_t* size,
                          const unsigned long long* iso, unsigned long long* hist, int bins, unsigned int* ticket,
                          unsigned long long* out, unsigned int* status) {
  extern __shared__ int h_s[];
  __shared__ bool s_last;
  for (int k = threadIdx.x; k < bins; k += blockDim.x) h_s[k] = 0;
  __syncthreads();
  const int lane = threadIdx.x & 31;
  const int64_t n = *n_list;
  // warp-uniform trip count
  for (int64_t w0 = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x - lane; w0 < n;
       w0 += static_cast<int64_t>(gridDim.x) * blockDim.x) {
    const int64_t i = w0 + lane;
    const int32_t root = i < n ? find_root(parent, list[i], status) : -1;
    const unsigned same = __match_any_sync(kFull, root);
    if (root >= 0 && lane == __ffs(static_cast<int>(same)) - 1) {
      const int m = __popc(same), had = atomicAdd(size + root, m);
      if (had > 0) atomicSub(h_s + min(had, bins - 1), 1);
      atomicAdd(h_s + min(had + m, bins - 1), 1);
    }
  }
  __syncthreads();
  for (int k = threadIdx.x; k < bins; k += blockDim.x)
    if (h_s[k]) atomicAdd(hist + k, static_cast<unsigned long long>(static_cast<long long>(h_s[k])));
  __threadfence();
  __syncthreads();
  if (threadIdx.x == 0) s_last = atomicAdd(ticket, 1u) == gridDim.x - 1;
  __syncthreads();
  if (!s_last) return;
  __threadfence();
  const unsigned long long isolated = __ldcg(iso);
  if (threadIdx.x == 0) {
    out[0] = *reinterpret_cast<volatile unsigned int*>(status);
    out[1] = isolated;
  }
  for (int k = threadIdx.x; k < bins; k += blockDim.x) out[2 + k] = __ldcg(hist + k) + (k == min(1, bins - 1) ? isolated : 0);
}

}  // namespace

int launch_cluster_stats(const ClusterArgs& c, void* stream) {
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  const int wpr = (c.sx + 31) / 32, nwords = static_cast<int>(cluster_words(c.sx, c.sy, c.sz));
  const int grid = std::min((nwords + 255) / 256, 148 * 8);
  unsigned int* const n_list = reinterpret_cast<unsigned int*>(c.misc);  // and the ticket behind it
  unsigned long long* const iso = c.misc + 1;
  unsigned long long* const hist = c.misc + kClusterHist;
  k_cu_bits<<<grid, 256, 0, st>>>(c.occ, nwords, wpr, c.sx, c.px, c.bits, c.misc, kClusterHist + c.bins);
  k_cu_classify<<<std::min((nwords + 256 * kClassWords - 1) / (256 * kClassWords), 148 * 8), 256, 0, st>>>(
      c.bits, nwords, wpr, c.sx, c.sy, c.sz, c.list, n_list, c.parent, c.size, iso);
  const int g2 = std::min((nwords * 4 + 255) / 256, 148 * 8);  // a thread for one site in 8, more than that in turns
  k_cu_union<<<g2, 256, 0, st>>>(c.occ, c.sx, c.sy, c.sz, c.px, c.list, n_list, c.parent, c.status);
  k_cu_hist<<<std::min(g2, 148 * 2), 256, sizeof(int) * c.bins, st>>>(c.list, n_list, c.parent, c.size, iso, hist, c.bins,
                                                                     n_list + 1, c.out, c.status);
  return static_cast<int>(cudaGetLastError());
}

}  // namespace akmc
