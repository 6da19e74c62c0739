// Length-limited Huffman code lengths for one CTA (core/src/util/huffman.rs:10-86, build_lengths with max_len 16)
// over 257 symbols: the 256 real symbols plus the dummy symbol of frequency 1 that optimal_table adds
// (jpeg/src/encode.rs:241-244). The sort is a parallel rank sort on the unique keys (freq, reverse symbol); the
// two-queue merge and the Kraft fix-up are sequential, as in the reference; the leaf depths, the per-length counts
// and the final assignment are computed one thread per leaf, with the same results.
#pragma once

namespace rcg {

constexpr int kHuffSyms = 257;

struct HuffScratch {
  uint4 key[(kHuffSyms + 3) / 4];  // the counts, an unused symbol's as the largest value
  int order[kHuffSyms];  // sorted position -> symbol
  unsigned long long weight[2 * kHuffSyms];
  int parent[2 * kHuffSyms];
  int count[17];
  int n_used;
};

// The merges of n > 1 leaves with weights W[0..n-1] ascending, by one thread: internal nodes n.. in creation order; ties go
// to the leaf (huffman.rs:38-46). Bound by the latency of a pick, so it has no branches, and weights are of 32 bits where
// they all fit: a rate-table launch 13.5 -> 11.2 us (0.3 of it from the width).
template <class T>
__device__ __forceinline__ void huff_merge(T* W, HuffScratch& s, int n) {
  // The heads of the two queues and the elements behind them; an empty place holds the largest value, which no weight has.
  const T none = ~(T)0;
  int leaf = 0, node = n, next = n;
  T wl = W[0], wl1 = W[1], wn = none, wn1 = none;
  auto pick = [&](T& w) -> int {
    const bool from_leaves = wl <= wn;
    const int at = from_leaves ? leaf : node, behind = at + 2;
    const T load = behind < (from_leaves ? n : next) ? W[behind] : none;
    w = from_leaves ? wl : wn;
    wl = from_leaves ? wl1 : wl;
    wl1 = from_leaves ? load : wl1;
    wn = from_leaves ? wn : wn1;
    wn1 = from_leaves ? wn1 : load;
    leaf += from_leaves;
    node += !from_leaves;
    return at;
  };
  while (next < 2 * n - 1) {
    T wa, wb;
    const int a = pick(wa);
    const int b = pick(wb);
    const T sum = wa + wb;
    W[next] = sum;
    s.parent[a] = next;
    s.parent[b] = next;
    wn = node == next ? sum : wn;
    wn1 = node + 1 == next ? sum : wn1;
    next++;
  }
}


// freq: 257 counts in shared memory (freq[256] = 1); lens: 257 code lengths out (0 = unused), shared memory.
// Every thread of the CTA calls it; the CTA has at least 260 threads (one per count and padding of the last quad).
//
// The two-queue merge is the one sequential step: one thread, with the head of each queue and the element behind it
// held in registers so that a pick does not wait for a shared-memory load. The depth pass, the per-length counts
// and the final assignment run one thread per leaf / sorted position.
__device__ inline void huff_lengths(const unsigned* freq, unsigned char* lens, HuffScratch& s) {
  const int t = threadIdx.x;
  if (t < kHuffSyms) lens[t] = 0;
  if (t == 0) s.n_used = 0;
  if (t < 17) s.count[t] = 0;
  const unsigned mine = t < kHuffSyms ? freq[t] : 0u;
  if (t < 4 * ((kHuffSyms + 3) / 4)) reinterpret_cast<unsigned*>(s.key)[t] = mine > 0 ? mine : 0xffffffffu;
  const bool wide = __syncthreads_or(mine >= (1u << 23));  // 257 smaller counts add up in 32 bits
  if (mine > 0) {
    // Rank among the used symbols in the order (count, descending symbol): those before t must be smaller, those
    // after t smaller or equal. Four counts per shared-memory load; 0xffffffff never counts.
    const unsigned f = mine;
    const int own = t >> 2;
    int r = 0;
    auto below = [&](const uint4 g, unsigned lim) {
      r += (g.x < lim) + (g.y < lim) + (g.z < lim) + (g.w < lim);
    };
#pragma unroll 4
    for (int j = 0; j < own; j++) below(s.key[j], f);
    const uint4 g = s.key[own];
    const unsigned o[4] = {g.x, g.y, g.z, g.w};
#pragma unroll
    for (int e = 0; e < 4; e++) r += (e < (t & 3) && o[e] < f) || (e > (t & 3) && o[e] <= f);
#pragma unroll 4
    for (int j = own + 1; j < (kHuffSyms + 3) / 4; j++) below(s.key[j], f + 1);
    s.order[r] = t;
    if (wide) s.weight[r] = f;
    else reinterpret_cast<unsigned*>(s.weight)[r] = f;
    atomicAdd(&s.n_used, 1);
  }
  __syncthreads();
  const int n = s.n_used;
  if (n == 1) {
    if (t == 0) lens[s.order[0]] = 1;
  } else if (n > 1) {
    if (t == 0) {
      if (wide) huff_merge(s.weight, s, n);
      else huff_merge(reinterpret_cast<unsigned*>(s.weight), s, n);
    }
    __syncthreads();
    // Depth of each leaf = its number of ancestors (the root is node 2n-2); counts per length, capped at 16.
    const int root = 2 * n - 2;
    if (t < n) {
      int d = 0;
      for (int j = t; j != root; j = s.parent[j]) d++;
      atomicAdd(&s.count[min(d, 16)], 1);
    }
    __syncthreads();
    if (t == 0) {
      // Kraft fix-up (huffman.rs:60-78): lengthen codes until the 16-bit limit holds.
      unsigned long long total = 0;
      for (int l = 1; l <= 16; l++) total += (unsigned long long)s.count[l] << (16 - l);
      while (total > (1ull << 16)) {
        s.count[16] -= 1;
        for (int l = 15; l >= 1; l--) {
          if (s.count[l] > 0) {
            s.count[l] -= 1;
            s.count[l + 1] += 2;
            break;
          }
        }
        total -= 1;
      }
    }
    __syncthreads();
    // Lengths 16, 15, .. 1 go to the sorted positions 0, 1, .. in turn (huffman.rs:80-85).
    if (t < n) {
      int start = 0, l = 16;
      while (l > 1 && t >= start + s.count[l]) start += s.count[l--];
      lens[s.order[t]] = (unsigned char)l;
    }
  }
  __syncthreads();
}

}  // namespace rcg
