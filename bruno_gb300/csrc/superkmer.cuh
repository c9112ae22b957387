/*
 * superkmer.cuh -- counting by super-k-mers.
 *
 * Consecutive k-mers of a read mostly share their minimizer (kmer.cuh), so a read falls into
 * runs of k-mers with one minimizer, super-k-mers (Li et al., "Memory efficient minimum
 * substring partitioning", VLDB 2013; Deorowicz et al., KMC 2, Bioinformatics 31, 2015).  A
 * run of n k-mers is one record of n + k - 1 bases, the base before it and the base after it,
 * instead of n records of one k-mer each; every occurrence of a k-mer lands in the partition
 * of its minimizer.
 *
 *   k_sk_extract   reads -> records, unordered, with the records and k-mers of every minimizer
 *                  bin tallied
 *   k_sk_estimate  a sample of the minimizers' k-mers -> HyperLogLog registers
 *   k_sk_plan_*    bins -> partitions of about equal k-mer counts (neighbouring bins share one)
 *   k_sk_scatter   records -> partition order; k_sk_split (many small records) in two passes
 *   k_sk_count     one CTA a partition: equal records merged into one with a weight, their
 *                  k-mers counted in shared memory, the k-mers to keep written to the table, or
 *                  (one-call builds) the graph's nodes made of them
 *   k_sk_expand    a crowded partition's records -> its k-mers with their weights, cut by their key
 *                  into parts that k_sk_count then counts like partitions
 *
 * 50 Mbp at 30x (1.2G k-mers, k = 31): extraction 4.9, split 2.8, count 12.1 ms, where k-mer records
 * took 9.9 (extraction), 5.8 (split), 11.6 (count) and 3.3 (filter).  k = 63, 352M k-mers: 1.9, 0.8
 * and 8.3 against 4.6, 5.3 and 11.1.
 *
 * Included by build.cu only, after its helpers (warp_sum, sm_cas128, CandArgs, ...).
 */
#pragma once

/* A record: NW 64-bit words, bases from the top of word 0, two bits each: the base before the
 * first k-mer (0 without one), the n + k - 1 bases of the k-mers, the base after the last (0
 * without one).  At most k - MZ_M + 1 k-mers share one occurrence of a minimizer, so 2k - 13 bases
 * (49 for k = 31, 113 for k = 63) leave the last word's low 30 bits for
 * [bin:22 | has right:1 | has left:1 | n - 1:6].  The record is on the strand its minimizer is
 * canonical on, so both strands of a place give the same record. */
template <class KT> struct SkRec;
template <> struct SkRec<KW1> { static constexpr int NW = 2; };
template <> struct SkRec<KW2> { static constexpr int NW = 4; };
constexpr uint64_t SK_LEFT = 1ull << 6, SK_RIGHT = 1ull << 7;
constexpr int SK_BIN_SHIFT = 8, SK_BIN_BITS = 22;
constexpr uint64_t SK_BIN_MASK = (1ull << SK_BIN_BITS) - 1;
/* A read of k + 1 bases has a (k+1)-mer and no (k+2)-mer: under the (k+1)-mer filter its two k-mers
 * are one or two records of n = 2 or 1 whose low bits are SK_EDGE + n: their occurrences count for the
 * edge between them, and for no biedge (EDGES: there can be such records) */
constexpr unsigned SK_EDGE = 60;
template <bool EDGES = true>
__device__ __forceinline__ unsigned sk_n(uint64_t last) {
  const unsigned x = (unsigned)(last & 63u);
  return EDGES && x > SK_EDGE ? x - SK_EDGE : x + 1u;
}
template <bool EDGES = true>
__device__ __forceinline__ bool sk_edge(uint64_t last) { return EDGES && (last & 63u) > SK_EDGE; }
/* the entry codes of such an edge, the ones that no (k+2)-mer has: 1 (neither base), 0 and 26..31 */
__device__ __forceinline__ unsigned sk_edge_code(unsigned in5, unsigned out5) {
  const unsigned x = in5 ? in5 - 1u : out5 + 3u;
  return x < 2u ? x : x + 24u;
}
__device__ __forceinline__ bool sk_edge_bases(unsigned code, unsigned &in5, unsigned &out5) {
  if (code >= 2u && code < 26u) return false;
  const unsigned x = code < 2u ? code : code - 24u;
  in5 = x < 4u ? x + 1u : 0u;
  out5 = x < 4u ? 0u : x - 3u;
  return true;
}

/* a sample's minimizer bins: bin0 + (mz_mix >> shift); the k-mers of records whose mix has no
 * bit of smask feed the estimate */
struct SkSample { unsigned int bin0, shift, smask, pad; };

constexpr int SK_TPB = 256;      /* extraction: 8 warps a block, each on its own tiles */
constexpr int SK_WORDS = 32;     /* a tile: one word of 16 bases a lane */
constexpr int SK_HALO = 4;       /* words past the tile that a window of 49 m-mers may touch */
constexpr int SK_READS = 16;     /* reads of a tile at most (the shortest that count take two words) */

/* word t of a tile is bases[sk_pad + t]: a record of the other strand is cut out from its end, up to
 * 2 * NW words before */
template <int NW> constexpr int sk_pad = 2 * NW + 1;
template <int NW>
struct SkWarp {
  uint32_t pmin[16][SK_WORDS + SK_HALO];     /* prefix minima inside blocks; then the runs' minimizers */
  uint32_t bases[2 * NW + 1 + SK_WORDS + 2 * NW + 3]; /* 16 bases a word, first base on top; word t at sk_pad + t */
  uint32_t marks[SK_WORDS + 1];              /* bit i: a run starts, or the read's k-mers end, at base i */
  uint16_t starts[16 * SK_WORDS];            /* run starts of the tile */
  unsigned long long addr[SK_READS];
  int len[SK_READS], nk[SK_READS];           /* bases, k-mers */
};

/* bases (j >= 0) of a record */
template <int NW>
__device__ __forceinline__ unsigned sk_base(const uint64_t *w, int j) {
  return (unsigned)(w[j >> 5] >> (62 - 2 * (j & 31))) & 3u;
}

/* the n bases (1..16) at device address s, packed from the top; .y nonzero: one is not A, C, G, T */
__device__ __forceinline__ uint2 sk_pack(uintptr_t s, int n) {
  const uintptr_t e = s + n, s4 = s & ~(uintptr_t)3;
  uint32_t v[5];
  #pragma unroll
  for (int q = 0; q < 5; ++q) v[q] = s4 + 4 * q < e ? __ldg((const uint32_t *)(s4 + 4 * q)) : 0u;
  const unsigned sh = 8u * (unsigned)(s & 3);
  uint32_t packed = 0, err = 0;
  #pragma unroll
  for (int q = 0; q < 4; ++q) {
    const uint32_t w = __funnelshift_r(v[q], v[q + 1], sh);
    const uint32_t c = ((w >> 1) ^ (w >> 2)) & 0x03030303u;   /* A0 C1 G2 T3, either case */
    /* the four codes as selector nibbles give back the letters they stand for */
    const uint32_t y = c | (c >> 4);
    const uint32_t want = __byte_perm(0x54474341u, 0u, (y & 0xFFu) | ((y >> 8) & 0xFF00u));
    uint32_t d = (w & 0xDFDFDFDFu) ^ want;
    const int left = n - 4 * q;   /* bytes of the read in this word */
    if (left < 4) d &= left <= 0 ? 0u : (1u << (8 * left)) - 1;
    err |= d;
    packed = (packed << 8) | ((c * 0x40100401u) >> 24);
  }
  return make_uint2(packed, err);
}

/* 16 bases reversed */
__device__ __forceinline__ uint32_t rev_pairs32(uint32_t x) {
  x = __brev(x);
  return ((x >> 1) & 0x55555555u) | ((x & 0x55555555u) << 1);
}

/* no record: the unused end of a chunk that a warp reserved (n - 1 is at most 48, SK_EDGE + n at most 62) */
constexpr uint64_t SK_NONE = 63;

/* HyperLogLog registers fed with the k-mers of the records listed; registers are read before they
 * are raised, since most updates raise nothing */
template <class KT>
__global__ void __launch_bounds__(128) k_sk_estimate(const uint64_t *recs, const uint32_t *list, uint64_t cap, int k,
                                                     const SkSample *samples, uint32_t S, unsigned int *hll,
                                                     const DevCounters *ctr) {
  constexpr int NW = SkRec<KT>::NW;
  if (ctr->err) return;   /* records past their room: the caller makes room and comes again */
  const uint64_t n_list = min((unsigned long long)cap, ctr->n_sk_est);
  for (uint64_t x = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; x < n_list; x += (uint64_t)gridDim.x * blockDim.x) {
    const uint64_t *rec = recs + (uint64_t)list[x] * NW;
    const uint64_t last = rec[NW - 1];
    const uint32_t bin = (uint32_t)((last >> SK_BIN_SHIFT) & SK_BIN_MASK);
    uint32_t lo = 0, hi = S;
    while (hi - lo > 1) { const uint32_t m = (lo + hi) >> 1; if (samples[m].bin0 <= bin) lo = m; else hi = m; }
    unsigned int *reg = hll + (uint64_t)lo * HLL_M;
    const int n = (int)sk_n(last);
    KT f{}, r{};
    for (int j = 1; j < n + k; ++j) {
      const unsigned c = sk_base<NW>(rec, j);
      f = KOps<KT>::append(f, c, k);
      r = KOps<KT>::prepend(3u - c, r, k);
      if (j < k) continue;
      const KT t = table_key(KOps<KT>::lt(f, r) ? f : r);
      const uint64_t h = sizeof(KT) == 8 ? ((const uint64_t *)&t)[0] << 2 : ((const uint64_t *)&t)[0];
      const unsigned idx = (unsigned)(h >> (64 - HLL_P));
      const unsigned rho = (unsigned)__clzll((h << HLL_P) | (1ull << (HLL_P - 1))) + 1u;
      if (rho > *(volatile unsigned int *)&reg[idx]) atomicMax(&reg[idx], rho);
    }
  }
}

struct SkExtract {
  const uint64_t *rstart, *rend;
  uint64_t r0, r1;                  /* reads */
  const uint64_t *first;            /* a batch: the first read (from r0 on) of samples s0, s0 + 1, ... */
  uint32_t s0, n_first;
  int k;
  uint32_t chunk;                   /* output records a warp reserves at once */
  const SkSample *samples;
  uint64_t *out;
  uint64_t cap;
  unsigned long long *hist;         /* per bin: k-mers << 32 | records */
  uint32_t *est;                    /* records for the estimate */
  uint64_t est_cap;
  unsigned long long *s_inst, *s_used;
  DevCounters *ctr;
};

/* Reads -> records.  A warp takes tiles of whole reads, 32 words of 16 bases at most (of a longer
 * read, a piece whose k-mers fit).  Each lane packs one word (a read with a base other than A, C,
 * G, T is dropped), orders the 16 m-mers that start in it, and finds the minimum of every window
 * of k - MZ_M + 1 m-mers from block prefix and suffix minima (van Herk 1992): a window that starts
 * in block a and ends in block b is a's suffix from the start, the whole blocks between, and b's
 * prefix up to the end.  BL (16, 8 or 4) is the block, at most k - MZ_M, so that no window lies
 * inside one block.  Where the minimum changes a run starts; the tile's runs are listed, and each
 * lane builds the records of every 32nd run from the packed words.  Everything stays inside the
 * warp: with one tile a block of 256 threads the block's barriers cost a quarter of its time (6.4 ms
 * at 1.2G k-mers, now 4.9).  Bound by issue (0.64 of the SMs' peak, 104 instructions a k-mer); four
 * blocks an SM instead of three spill (5.2 ms).  Output places come in chunks that a warp reserves (one counter
 * cannot take an atomic per tile); a chunk's unused end is marked SK_NONE.  EDGES: the (k+1)-mer
 * filter's, with reads of k + 1 bases (as a switch it cost the others 2%). */
template <class KT, int BL, bool EDGES>
__global__ void __launch_bounds__(SK_TPB, 3) k_sk_extract(SkExtract a) {
  constexpr int NW = SkRec<KT>::NW, NB = 16 / BL, PAD = sk_pad<NW>;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  SkWarp<NW> &S = reinterpret_cast<SkWarp<NW> *>(smem_raw)[threadIdx.x >> 5];
  const int lane = threadIdx.x & 31, k = a.k;
  const unsigned le = ~0u >> (31 - lane);   /* this lane and the ones below */
  const int w1 = k - MZ_M;                  /* a window's last m-mer, from its first */
  const int cw = w1 % BL, qw = w1 / BL;
  const int piece = (16 * SK_WORDS - k - 1) & ~15;   /* k-mers of a long read's piece */
  for (int i = lane; i < 16 * SK_HALO; i += 32) S.pmin[i / SK_HALO][SK_WORDS + i % SK_HALO] = ~0u;
  if (lane == 0) S.marks[SK_WORDS] = 0;
  if (lane < PAD) S.bases[lane] = 0;   /* (what a record cuts from there is masked off) */
  uint32_t cpos = 0, cend = 0;   /* the warp's chunk of the output (fewer than 2^32 records) */
  /* an even share of the reads, sample by sample */
  uint64_t pos, end;
  {
    const uint64_t warp = blockIdx.x * (SK_TPB / 32) + (threadIdx.x >> 5), warps = gridDim.x * (SK_TPB / 32);
    pos = (a.r1 - a.r0) * warp / warps;
    end = (a.r1 - a.r0) * (warp + 1) / warps;
  }
  while (pos < end) {
    uint64_t ra = a.r0 + pos;
    uint32_t n_reads = (uint32_t)(end - pos);   /* reads of the sample's share not yet taken */
    unsigned smp = 0;
    if (a.first) {
      uint32_t lo = 0, hi = a.n_first;
      while (hi - lo > 1) { const uint32_t m = (lo + hi) >> 1; if (__ldg(a.first + m) <= pos) lo = m; else hi = m; }
      smp = a.s0 + lo;
      if (lo + 1 < a.n_first) n_reads = (uint32_t)(min(end, __ldg(a.first + lo + 1)) - pos);
    }
    pos += n_reads;
    unsigned inst = 0, used = 0, edges = 0;   /* edges: k-mers of reads of k + 1 bases */
    uint64_t sp = 0;           /* the read ra + lane */
    uint32_t len = 0;
    if (lane < n_reads) { sp = a.rstart[ra + lane]; len = (uint32_t)(a.rend[ra + lane] - sp); }
    uint32_t q0 = 0;           /* first k-mer of the long read's next piece */
    bool long_ok = false;
    while (n_reads) {
      /* (1) the tile's reads: as many as fit the words, or a piece of a long one */
      __syncwarp();   /* the tile before has been read */
      const uint32_t L0 = __shfl_sync(~0u, len, 0);
      unsigned first;
      uint32_t n_words, reads = 1;
      bool pre = false, post = false;
      if (L0 > 16 * SK_WORDS) {
        const uint64_t s0 = __shfl_sync(~0u, sp, 0);
        const uint32_t nk = L0 - k + 1;
        if (q0 == 0) {   /* the whole read's bases checked before its first piece */
          unsigned bad = 0;
          for (uint32_t p = 16 * lane; p < L0; p += 16 * SK_WORDS) bad |= sk_pack(s0 + p, (int)min(16u, L0 - p)).y;
          long_ok = !__any_sync(~0u, bad);
        }
        const int n = (int)min((uint32_t)piece, nk - q0);
        pre = q0 > 0;
        post = q0 + n < nk;
        if (lane == 0) {
          S.addr[0] = s0 + q0;
          S.nk[0] = n;
          S.len[0] = n + k - 1 + (post ? 1 : 0);
          S.bases[PAD - 1] = pre ? sk_pack(s0 + q0 - 1, 1).x >> 30 : 0u;
        }
        first = long_ok ? 1u : 0u;
        n_words = long_ok ? (uint32_t)(n + k - 1 + (post ? 1 : 0) + 15) >> 4 : 0u;
        q0 += n;
        if (!long_ok || q0 >= nk) q0 = 0; else reads = 0;
      } else {
        const uint32_t L = len >= (uint32_t)k + (EDGES ? 1 : 2) ? min(len, 16u * SK_WORDS + 1) : 0u;
        const uint32_t nw = (L + 15) >> 4;
        uint32_t x = nw;
        #pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
          const uint32_t y = __shfl_up_sync(~0u, x, o);
          if (lane >= o) x += y;
        }
        /* x never falls, so the reads that fit come first */
        const bool fits = lane < n_reads && x <= SK_WORDS, kept = fits && nw;
        const unsigned mf = __ballot_sync(~0u, fits), mk = __ballot_sync(~0u, kept);
        reads = __popc(mf);
        n_words = mf ? __shfl_sync(~0u, x, 31 - __clz(mf)) : 0u;
        if (kept) {
          const int d = __popc(mk & (le >> 1));
          S.addr[d] = sp; S.len[d] = (int)L; S.nk[d] = (int)L - k + 1;
        }
        first = __reduce_or_sync(~0u, kept ? 1u << (x - nw) : 0u);
      }
      ra += reads;
      n_reads -= reads;
      if (reads) {   /* the next tile's reads */
        len = 0;
        if (lane < n_reads) { sp = a.rstart[ra + lane]; len = (uint32_t)(a.rend[ra + lane] - sp); }
      }
      if (n_words == 0) continue;
      __syncwarp();
      /* (2) the lane's word: 16 bases packed and checked */
      const bool mine = (uint32_t)lane < n_words;
      const int rd = __popc(first & le) - 1, w0 = 31 - __clz(first & le), p0 = 16 * (lane - w0);
      const unsigned above = first & ~le;
      const int w2 = above ? __ffs(above) - 1 : (int)n_words;
      uint2 pk = make_uint2(0u, 0u);
      int L = 0;
      if (mine) {
        L = S.len[rd];
        pk = sk_pack(S.addr[rd] + p0, min(16, L - p0));
      }
      S.bases[PAD + lane] = pk.x;
      if (lane < 2 * NW + 3) S.bases[PAD + SK_WORDS + lane] = 0;
      const unsigned bad = __ballot_sync(~0u, pk.y != 0);
      const bool good = mine && (bad & (~0u >> (32 - w2)) & (~0u << w0)) == 0;
      /* (3) the orders of the 16 m-mers that start in the word, then block minima */
      const uint32_t nextw = __shfl_down_sync(~0u, pk.x, 1);
      uint32_t h[16];
      {
        const uint64_t W = ((uint64_t)pk.x << 32) | (lane < 31 ? nextw : 0u), R = rev_pairs(~W);
        /* (m-mers past the read's last are in no window of its k-mers) */
        #pragma unroll
        for (int i = 0; i < 16; ++i)
          h[i] = mz_order((uint32_t)(W >> (64 - 2 * MZ_M - 2 * i)) & MZ_MASK, (uint32_t)(R >> (2 * i)) & MZ_MASK);
        uint32_t m = ~0u;
        #pragma unroll
        for (int i = 0; i < 16; ++i) {
          m = i % BL == 0 ? h[i] : min(m, h[i]);
          S.pmin[i][lane] = m;
        }
        #pragma unroll
        for (int i = 14; i >= 0; --i)
          if (i % BL != BL - 1) h[i] = min(h[i], h[i + 1]);
      }
      __syncwarp();
      #pragma unroll
      for (int bb = 0; bb < NB; ++bb) {
        /* whole blocks inside the windows of this block: qw - 1 of them, or qw once the end has
         * crossed into the next block */
        uint32_t mid = ~0u;
        for (int q = 1; q < qw; ++q) {
          const int g = bb + q;
          mid = min(mid, S.pmin[(g % NB) * BL + BL - 1][lane + g / NB]);
        }
        const int g = bb + qw;
        const uint32_t mid2 = min(mid, S.pmin[(g % NB) * BL + BL - 1][lane + g / NB]);
        /* the windows' ends: BL - cw of them in the block qw further on, cw in the one after that */
        const uint32_t *e1 = &S.pmin[(g % NB) * BL + cw][lane + g / NB];
        const uint32_t *e2 = &S.pmin[((g + 1) % NB) * BL][lane + (g + 1) / NB] - (BL - cw) * (SK_WORDS + SK_HALO);
        #pragma unroll
        for (int i = 0; i < BL; ++i) {
          const bool same = i < BL - cw;
          h[bb * BL + i] = min(h[bb * BL + i], min(same ? mid : mid2, (same ? e1 : e2)[i * (SK_WORDS + SK_HALO)]));
        }
      }
      /* (4) run starts, and the end of the read's k-mers */
      uint32_t prev = __shfl_up_sync(~0u, h[15], 1);
      uint32_t st = 0, marks = 0;
      if (good) {
        const int nk = S.nk[rd] - p0;   /* k-mer positions from the word on */
        #pragma unroll
        for (int i = 0; i < 16; ++i) {
          st |= h[i] != prev ? 1u << i : 0u;
          prev = h[i];
        }
        const bool edge = EDGES && L == k + 1 && !pre && !post;   /* (not a piece of a longer read) */
        if (p0 == 0) { st |= 1u; used += !pre && !edge; }
        st &= nk >= 16 ? 0xFFFFu : nk > 0 ? (1u << nk) - 1 : 0u;
        marks = st;
        if (nk >= 0 && nk < 16) marks |= 1u << nk;
        (edge ? edges : inst) += (unsigned)max(0, min(16, nk));
      }
      S.marks[lane] = marks;
      const uint32_t cnt = __popc(st);
      uint32_t x = cnt;
      #pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const uint32_t y = __shfl_up_sync(~0u, x, o);
        if (lane >= o) x += y;
      }
      const uint32_t total = __shfl_sync(~0u, x, 31);
      uint32_t at = x - cnt;
      __syncwarp();   /* every window has been read: the runs' minimizers instead */
      #pragma unroll
      for (int i = 0; i < 16; ++i) S.pmin[i][lane] = h[i];
      for (uint32_t b = st; b; b &= b - 1) S.starts[at++] = (uint16_t)(16 * lane + __ffs(b) - 1);
      /* the tile's places: the rest of the chunk, then a new one */
      const uint32_t rest = min(total, cend - cpos), o1 = cpos;
      uint32_t o2 = 0;
      cpos += rest;
      if (rest < total) {
        const uint32_t ch = max(a.chunk, total - rest);
        if (lane == 0) o2 = (uint32_t)atomicAdd(&a.ctr->n_sk, (unsigned long long)ch);
        o2 = __shfl_sync(~0u, o2, 0);
        cpos = o2 + (total - rest);
        cend = o2 + ch;
      }
      __syncwarp();
      /* (5) the records */
      const SkSample X = a.samples[smp];
      for (uint32_t y = lane; y < total; y += 32) {
        const int t = S.starts[y] >> 4, i = S.starts[y] & 15;
        const uint32_t mz = S.pmin[i][t];
        const unsigned ft = first & (~0u >> (31 - t));
        const int r = __popc(ft) - 1, wr = 31 - __clz(ft), p = 16 * (t - wr) + i, nk = S.nk[r];
        int run;   /* to the next mark: there is one, the end of the read's k-mers */
        const uint32_t m = S.marks[t] >> i >> 1;
        if (m) run = __ffs(m);
        else {
          run = 16 - i;
          int u = t + 1;
          while (u < SK_WORDS && S.marks[u] == 0) { run += 16; ++u; }
          run += __ffs(S.marks[u]) - 1;   /* (marks[SK_WORDS] exists and is never reached) */
        }
        const uint32_t mix = mz_mix(mz), bin = X.bin0 + (mix >> X.shift);
        uint32_t o = y < rest ? o1 + y : o2 + (y - rest);
        for (int d = 0; d < run; ) {   /* a minimizer that recurs may run on: cut at what a record holds */
          const int n = min(run - d, k - MZ_M + 1), nb = n + k + 1, q = p + d - 1;   /* q: the base before the first k-mer */
          bool hl = q >= 0 || pre, hr = p + d + n < nk || post;
          const bool other = mz & 1u;   /* on the other strand: cut out from the end, then reversed */
          const int b0 = 16 * (PAD + wr) + (other ? q + nb - 32 * NW : q), tw = b0 >> 4;
          const unsigned sh = 2u * (unsigned)(b0 & 15);
          uint32_t v[2 * NW];
          uint32_t cur = S.bases[tw];
          #pragma unroll
          for (int u = 0; u < 2 * NW; ++u) {
            const uint32_t nxt = S.bases[tw + u + 1];
            v[u] = __funnelshift_l(nxt, cur, sh);
            cur = nxt;
          }
          if (other) {
            #pragma unroll
            for (int u = 0; u < NW; ++u) {
              const uint32_t x = rev_pairs32(~v[u]);
              v[u] = rev_pairs32(~v[2 * NW - 1 - u]);
              v[2 * NW - 1 - u] = x;
            }
            const bool s = hl; hl = hr; hr = s;
          }
          const int bits = 2 * (hr ? nb : nb - 1);   /* past the last base, and the absent base before: zero */
          #pragma unroll
          for (int u = 0; u < 2 * NW; ++u) v[u] &= __funnelshift_lc(0u, ~0u, (unsigned)max(0, 32 * (u + 1) - bits));
          if (!hl) v[0] &= ~0u >> 2;
          const bool edge = EDGES && S.len[r] == k + 1 && !pre && !post;
          v[2 * NW - 1] |= (bin << SK_BIN_SHIFT) | (hr ? (uint32_t)SK_RIGHT : 0u) | (hl ? (uint32_t)SK_LEFT : 0u) |
                           (edge ? SK_EDGE + n : (uint32_t)(n - 1));
          if (o < a.cap) {
            ulonglong2 *dst = reinterpret_cast<ulonglong2 *>(a.out + (uint64_t)o * NW);
            #pragma unroll
            for (int u = 0; u < NW; u += 2)
              __stcs(dst + u / 2, make_ulonglong2(((uint64_t)v[2 * u] << 32) | v[2 * u + 1],
                                                  ((uint64_t)v[2 * u + 2] << 32) | v[2 * u + 3]));
          } else {
            atomicOr(&a.ctr->err, (unsigned long long)DERR_TABLE_FULL);
          }
          atomicAdd(&a.hist[bin], ((unsigned long long)n << 32) | 1ull);
          if ((mix & X.smask) == 0 && o < a.cap) {   /* (a record that was not stored is not read either) */
            const unsigned long long e = atomicAdd(&a.ctr->n_sk_est, 1ull);
            if (e < a.est_cap) a.est[e] = o;
          }
          d += n;
          if (d < run) o = (uint32_t)atomicAdd(&a.ctr->n_sk, 1ull);
        }
      }
    }
    const unsigned long long iw = warp_sum(inst), uw = warp_sum(used);
    if (EDGES) {
      const unsigned long long ew = warp_sum(edges);
      if (lane == 0 && ew) atomicAdd(&a.ctr->n_sk_edges, ew);
    }
    if (lane == 0) {
      if (iw) atomicAdd(&a.ctr->n_instances, iw);
      if (uw) atomicAdd(&a.ctr->n_reads_used, uw);
      if (a.s_inst && iw) atomicAdd(&a.s_inst[smp], iw);
      if (a.s_used && uw) atomicAdd(&a.s_used[smp], uw);
    }
  }
  for (uint32_t o = cpos + lane; o < cend; o += 32)
    if (o < a.cap) a.out[(uint64_t)o * NW + NW - 1] = SK_NONE;
}

/* ------------------------------------------------------------ bins -> partitions
 * Partition of a bin = (k-mers of its sample's bins before it) / T, T = the sample's k-mers over
 * its partitions: neighbouring bins share a partition of T k-mers give or take a bin, so a
 * partition's size does not depend on how evenly minimizers spread. */
struct SkPlan {   /* a sample */
  unsigned long long inst0, T;        /* k-mers of the samples before, k-mers a partition */
  unsigned int bin0, pbase, parts, pad;   /* first bin, first partition, partitions */
};
/* records of one bin at most: its k-mers, at most 49 a record, have 32 bits of its tally */
constexpr unsigned long long SK_MAX_BIN = 1ull << 26;
constexpr int SK_PLAN_TPB = 256, SK_PLAN_PER = 16, SK_PLAN_CHUNK = SK_PLAN_TPB * SK_PLAN_PER;

__global__ void __launch_bounds__(SK_PLAN_TPB) k_sk_plan_sum(const unsigned long long *hist, uint32_t nbins,
                                                             ulonglong2 *sums, DevCounters *ctr) {
  unsigned long long inst = 0, rec = 0;
  bool big = false;
  for (uint32_t j = threadIdx.x; j < SK_PLAN_CHUNK; j += SK_PLAN_TPB) {
    const uint32_t b = blockIdx.x * SK_PLAN_CHUNK + j;
    if (b >= nbins) break;
    const unsigned long long v = hist[b];
    inst += v >> 32; rec += v & 0xFFFFFFFFull;
    big |= (v & 0xFFFFFFFFull) > SK_MAX_BIN;
  }
  inst = warp_sum(inst); rec = warp_sum(rec);
  __shared__ unsigned long long si[SK_PLAN_TPB / 32], sr[SK_PLAN_TPB / 32];
  if ((threadIdx.x & 31) == 0) { si[threadIdx.x >> 5] = inst; sr[threadIdx.x >> 5] = rec; }
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int q = 1; q < SK_PLAN_TPB / 32; ++q) { inst += si[q]; rec += sr[q]; }
    sums[blockIdx.x] = make_ulonglong2(inst, rec);
  }
  if (big) atomicOr(&ctr->err, (unsigned long long)DERR_SKEW);
}

/* part[b] = partition of bin b (over all samples); off[P], cur[P] = first record of partition P
 * (nparts + 1 and nparts of them) */
__global__ void __launch_bounds__(SK_PLAN_TPB) k_sk_plan_apply(const unsigned long long *hist, uint32_t nbins,
                                                               const ulonglong2 *sums, const SkPlan *plan, uint32_t S,
                                                               uint32_t nparts, uint32_t *part, uint32_t *off,
                                                               uint32_t *cur) {
  __shared__ unsigned long long si[SK_PLAN_TPB], sr[SK_PLAN_TPB];
  const int tid = threadIdx.x;
  unsigned long long bi = 0, br = 0;   /* sums of the blocks before */
  for (uint32_t q = tid; q < blockIdx.x; q += SK_PLAN_TPB) { bi += sums[q].x; br += sums[q].y; }
  const uint32_t b0 = blockIdx.x * SK_PLAN_CHUNK + tid * SK_PLAN_PER, b1 = min(nbins, b0 + SK_PLAN_PER);
  unsigned long long ti = 0, tr = 0;
  for (uint32_t b = b0; b < b1; ++b) { const unsigned long long v = hist[b]; ti += v >> 32; tr += v & 0xFFFFFFFFull; }
  /* the block's base: every thread's share of the earlier sums; then the threads' exclusive scan */
  si[tid] = bi; sr[tid] = br;
  __syncthreads();
  for (int o = SK_PLAN_TPB / 2; o > 0; o >>= 1) {
    if (tid < o) { si[tid] += si[tid + o]; sr[tid] += sr[tid + o]; }
    __syncthreads();
  }
  bi = si[0]; br = sr[0];
  __syncthreads();
  si[tid] = ti; sr[tid] = tr;
  __syncthreads();
  for (int o = 1; o < SK_PLAN_TPB; o <<= 1) {
    const unsigned long long vi = tid >= o ? si[tid - o] : 0, vr = tid >= o ? sr[tid - o] : 0;
    __syncthreads();
    si[tid] += vi; sr[tid] += vr;
    __syncthreads();
  }
  unsigned long long inst = bi + si[tid] - ti, rec = br + sr[tid] - tr;
  if (b0 >= nbins) return;
  /* the sample of a bin, and the bin's partition from the k-mers before it */
  auto sample_of_bin = [&](uint32_t b) {
    uint32_t lo = 0, hi = S;
    while (hi - lo > 1) { const uint32_t m = (lo + hi) >> 1; if (plan[m].bin0 <= b) lo = m; else hi = m; }
    return lo;
  };
  auto part_of = [&](const SkPlan &X, unsigned long long before) {
    return X.pbase + (uint32_t)min((before - X.inst0) / X.T, (unsigned long long)(X.parts - 1));
  };
  uint32_t s = sample_of_bin(b0);
  SkPlan X = plan[s];
  /* the partition of the bin before b0: partitions after it, up to b0's own, start at b0 */
  uint32_t next;   /* first partition whose start is not yet known */
  if (b0 == 0) next = 0;
  else {
    const uint32_t sp = b0 > X.bin0 ? s : sample_of_bin(b0 - 1);
    const SkPlan Y = sp == s ? X : plan[sp];
    next = part_of(Y, inst - (hist[b0 - 1] >> 32)) + 1;
  }
  for (uint32_t b = b0; b < b1; ++b) {
    while (s + 1 < S && plan[s + 1].bin0 <= b) X = plan[++s];
    const uint32_t P = part_of(X, inst);
    part[b] = P;
    for (; next <= P; ++next) { off[next] = (uint32_t)rec; cur[next] = (uint32_t)rec; }
    const unsigned long long v = hist[b];
    inst += v >> 32; rec += v & 0xFFFFFFFFull;
  }
  if (b1 == nbins) {
    for (; next < nparts; ++next) { off[next] = (uint32_t)rec; cur[next] = (uint32_t)rec; }
    off[nparts] = (uint32_t)rec;
  }
}

/* Records -> partition order: one returning atomic on the partition's cursor and one store a
 * record.  A partition's open line stays in L2 until its records have filled it (2^18 open
 * 128-byte lines are 32 MB of the 129 MB), so the scattered stores leave as whole lines.  Bound by the
 * single stores and atomics (133M records of 16 bytes, 2^18 partitions: 3.55 ms, where reading and
 * writing them takes 0.63; with places from bin counts and no atomics, to 2^21 open lines, 6.65). */
constexpr int SK_SCATTER_U = 4;
template <int NW>
__global__ void __launch_bounds__(256) k_sk_scatter(const uint64_t *rec, uint64_t n, const uint32_t *part,
                                                    uint32_t *cur, uint64_t *out, const DevCounters *ctr) {
  if (ctr->err) return;   /* the bins cannot be counted this way: the caller falls back */
  const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
  for (uint64_t i0 = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i0 < n; i0 += stride * SK_SCATTER_U) {
    ulonglong2 r[SK_SCATTER_U][NW / 2];
    uint32_t P[SK_SCATTER_U], o[SK_SCATTER_U];
    #pragma unroll
    for (int u = 0; u < SK_SCATTER_U; ++u) {
      const uint64_t i = i0 + u * stride;
      if (i >= n) continue;
      #pragma unroll
      for (int q = 0; q < NW / 2; ++q) r[u][q] = __ldcs(reinterpret_cast<const ulonglong2 *>(rec + i * NW) + q);
    }
    bool has[SK_SCATTER_U];
    #pragma unroll
    for (int u = 0; u < SK_SCATTER_U; ++u) has[u] = i0 + u * stride < n && (r[u][NW / 2 - 1].y & 63u) != SK_NONE;
    #pragma unroll
    for (int u = 0; u < SK_SCATTER_U; ++u)
      if (has[u]) P[u] = __ldg(part + ((r[u][NW / 2 - 1].y >> SK_BIN_SHIFT) & SK_BIN_MASK));
    #pragma unroll
    for (int u = 0; u < SK_SCATTER_U; ++u)
      if (has[u]) o[u] = atomicAdd(&cur[P[u]], 1u);
    #pragma unroll
    for (int u = 0; u < SK_SCATTER_U; ++u) {
      if (!has[u]) continue;
      #pragma unroll
      for (int q = 0; q < NW / 2; ++q) reinterpret_cast<ulonglong2 *>(out + (uint64_t)o[u] * NW)[q] = r[u][q];
    }
  }
}

/* The same in two passes, to groups of 2^lg partitions and from these to partitions: a block orders a
 * tile of records by group (partition) in shared memory and writes a run of its own to each, one
 * atomic a run.  Bound by its phases: a block of a tile in registers and in shared memory leaves two
 * to an SM (133M records, 2^18 partitions, both passes: 2.80 ms; tiles of 2048 records, whose runs
 * are half as long, 3.41; of 8192, one block an SM, 3.10; 1024 threads a tile of 4096 3.14). */
constexpr int SK_SPLIT_TPB = 512, SK_SPLIT_N = 1024;   /* groups, and partitions of a group, at most */
template <int NW> constexpr int SK_SPLIT_TILE = 16384 / (2 * NW);
template <int NW> constexpr size_t SK_SPLIT_BYTES = (size_t)SK_SPLIT_TILE<NW> * (NW * 8 + 2) + SK_SPLIT_N * 8;
template <int NW>
__global__ void __launch_bounds__(SK_SPLIT_TPB, 2) k_sk_split(const uint64_t *rec, uint64_t n, const uint32_t *n_dev,
                                                           const uint32_t *part, int lg, int fine, uint32_t *cur,
                                                           uint64_t *out, uint64_t room, const DevCounters *ctr) {
  constexpr int TILE = SK_SPLIT_TILE<NW>, U = TILE / SK_SPLIT_TPB;
  extern __shared__ __align__(16) uint64_t s_rec[];
  uint32_t *s_cnt = reinterpret_cast<uint32_t *>(s_rec + (size_t)TILE * NW), *s_dst = s_cnt + SK_SPLIT_N;
  uint16_t *s_d = reinterpret_cast<uint16_t *>(s_dst + SK_SPLIT_N);
  __shared__ uint32_t s_warp[SK_SPLIT_TPB / 32];
  if (ctr->err) return;   /* the bins cannot be counted this way: the caller falls back */
  const int tid = threadIdx.x, lane = tid & 31;
  const uint64_t total = n_dev ? *n_dev : n;   /* (the second pass: no unused places) */
  const uint64_t i0 = (uint64_t)blockIdx.x * TILE;
  if (n_dev)   /* unused places behind, as the extraction leaves them: the records may be ordered again */
    for (uint64_t i = max(total, i0) + tid; i < min(room, i0 + TILE); i += SK_SPLIT_TPB) out[i * NW + NW - 1] = SK_NONE;
  if (i0 >= total) return;
  for (int i = tid; i < SK_SPLIT_N; i += SK_SPLIT_TPB) s_cnt[i] = 0;
  /* the second pass: partitions counted from the first of the tile's first group */
  uint32_t p0 = 0;
  if (fine) p0 = __ldg(part + ((rec[i0 * NW + NW - 1] >> SK_BIN_SHIFT) & SK_BIN_MASK)) >> lg << lg;
  __syncthreads();
  ulonglong2 r[U][NW / 2];
  uint32_t d[U], at[U];
  #pragma unroll
  for (int u = 0; u < U; ++u) {
    const uint64_t i = i0 + u * SK_SPLIT_TPB + tid;
    d[u] = ~0u;
    if (i >= total) continue;
    #pragma unroll
    for (int q = 0; q < NW / 2; ++q) r[u][q] = __ldcs(reinterpret_cast<const ulonglong2 *>(rec + i * NW) + q);
  }
  #pragma unroll
  for (int u = 0; u < U; ++u) {
    if (i0 + u * SK_SPLIT_TPB + tid >= total || (r[u][NW / 2 - 1].y & 63u) == SK_NONE) continue;
    const uint32_t P = __ldg(part + ((r[u][NW / 2 - 1].y >> SK_BIN_SHIFT) & SK_BIN_MASK));
    d[u] = fine ? P - p0 : P >> lg;
  }
  #pragma unroll
  for (int u = 0; u < U; ++u) {
    if (d[u] == ~0u) continue;
    if (d[u] < SK_SPLIT_N) {
      at[u] = atomicAdd(&s_cnt[d[u]], 1u);
    } else {   /* past the second of the tile's groups: by itself */
      const uint64_t o = atomicAdd(&cur[p0 + d[u]], 1u);
      #pragma unroll
      for (int q = 0; q < NW / 2; ++q) reinterpret_cast<ulonglong2 *>(out + o * NW)[q] = r[u][q];
      d[u] = ~0u;
    }
  }
  __syncthreads();
  /* where each group's records start in the tile, and where they go */
  constexpr int PER = SK_SPLIT_N / SK_SPLIT_TPB;
  uint32_t c[PER], sum = 0;
  #pragma unroll
  for (int q = 0; q < PER; ++q) { c[q] = s_cnt[tid * PER + q]; sum += c[q]; }
  uint32_t x = sum;
  #pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const uint32_t y = __shfl_up_sync(~0u, x, o);
    if (lane >= o) x += y;
  }
  if (lane == 31) s_warp[tid >> 5] = x;
  __syncthreads();
  uint32_t run = x - sum, all = 0;
  for (int q = 0; q < SK_SPLIT_TPB / 32; ++q) {
    run += q < (tid >> 5) ? s_warp[q] : 0u;
    all += s_warp[q];
  }
  #pragma unroll
  for (int q = 0; q < PER; ++q) {
    s_cnt[tid * PER + q] = run;
    if (c[q]) s_dst[tid * PER + q] = atomicAdd(&cur[p0 + tid * PER + q], c[q]) - run;   /* (modulo 2^32) */
    run += c[q];
  }
  __syncthreads();
  #pragma unroll
  for (int u = 0; u < U; ++u) {
    if (d[u] == ~0u) continue;
    const uint32_t o = s_cnt[d[u]] + at[u];
    #pragma unroll
    for (int q = 0; q < NW / 2; ++q) reinterpret_cast<ulonglong2 *>(s_rec + (size_t)o * NW)[q] = r[u][q];
    s_d[o] = (uint16_t)d[u];
  }
  __syncthreads();
  for (uint32_t y = tid; y < all; y += SK_SPLIT_TPB) {
    const uint32_t o = s_dst[s_d[y]] + y;
    #pragma unroll
    for (int q = 0; q < NW / 2; ++q)
      reinterpret_cast<ulonglong2 *>(out + (uint64_t)o * NW)[q] = reinterpret_cast<const ulonglong2 *>(s_rec + (size_t)y * NW)[q];
  }
}
/* cursors of the groups of 2^lg partitions */
__global__ void k_sk_groups(const uint32_t *off, uint32_t nparts, int lg, uint32_t *cur) {
  const uint32_t g = blockIdx.x * blockDim.x + threadIdx.x;
  if ((uint64_t)g << lg < nparts) cur[g] = off[g << lg];
}

/* ------------------------------------------------------------ counting
 * One CTA a partition.  Its records come in rounds; equal records (the same place read without
 * an error, from either strand: two thirds of them at 30x) are merged in a small hash of record
 * numbers, then the distinct ones' k-mers, cut into items of SK_ITEM k-mers so that every thread
 * has work, are counted with the record's weight in a hash of k-mers in shared memory: per slot
 * the k-mer and two entry words, in two arrays (a k-mer with more biedges goes on in later slots
 * keyed k-mer | CONT).  The k-mers to keep are then placed in a region of the table of their own
 * number over the load, in the table's slot format, and listed for the filter.
 *
 * keep_all: every k-mer is kept (the raw counts or other thresholds may still be asked for);
 * otherwise a k-mer that the filter's quick rule drops (its total below the (k+1)-mer lower bound;
 * filter_quick) is tallied and left out: at 30x and 0.5% errors three k-mers of four. */
/* Bound by issue and by the block's phases (0.61 of the SMs' peak, 21 of 32 lanes at work: probe runs
 * and entries of uneven length; a quarter of the stalls are barriers).  1.2G k-mers, k = 31: 12.1 ms
 * with 384 threads (256: 12.6, 320: 12.2), items of 3 (4 and 5: 3% more) and two probes before a k-mer
 * waits (three: 12.4, four: 12.6); making the nodes is 1.45 ms of it, and saves the filter's 3.3. */
constexpr int SK_COUNT_TPB = 384;
constexpr int SK_ITEM = 3;
template <class KT> constexpr int SK_ITEMS = ((sizeof(KT) == 8 ? 17 : 49) + SK_ITEM - 1) / SK_ITEM;   /* items a record at most */
constexpr double SK_MAX_INV_LOAD = 4.0;
constexpr uint32_t SK_LATE = 256;
struct SkCount {
  const uint64_t *recs;
  const uint32_t *off;              /* first record of every partition */
  const uint32_t *todo;             /* the partitions to count; NULL: those of `cls`, or all */
  const ClassRun *cls;              /* a batch's partitions of one size class, as runs of samples */
  uint32_t ncls;
  uint32_t slots;                   /* k-mer slots in shared memory */
  uint32_t late;                    /* where the late k-mers wait, in shared-memory words */
  uint32_t round, hsize;            /* records a round (at most 1024), entries of their hash (a power of two) */
  int k;
  int keep_all, thresholding;
  uint32_t t[6];                    /* the filter's bounds, clamped to 65536 (counts end at 65535) */
  double inv_load;                  /* table slots a kept slot */
  uint64_t *table;
  uint64_t cap;                     /* table slots of the sample(s) */
  uint2 *info;                      /* per partition: its first slot, its slots */
  uint32_t *over;                   /* partitions that overflowed the shared-memory slots */
  uint32_t *cand;                   /* the slots the filter must read (not with nodes) */
  int nodes;                        /* local_insert_by_freqencies is done here, on the kept k-mers */
  uint32_t *chain_list, *branch_list;   /* slots of the chain and branch nodes */
  uint64_t list_cap;
  unsigned long long *s_tally;
  const SGeom *sg;
  uint32_t nsamples;
  unsigned long long *bump;         /* per sample: table slots taken so far */
  uint32_t sub0;                    /* parts of crowded partitions: the first one's place in info, */
  const uint32_t *sub_smp;          /* their samples */
  uint64_t *past;                   /* their k-mer records that an entry no longer takes (SkPast) */
  uint64_t past_cap;
  DevCounters *ctr;
};

/* entries of the record hash: a power of two, a third of them free at least */
__host__ __device__ constexpr uint32_t sk_hash_size(uint32_t round) {
  uint32_t h = 64;
  while (2 * h < 3 * round) h *= 2;
  return h;
}
/* Shared memory: slots (key, two entries); then a round's records, weights, record hash (its memory
 * then holds the item list, 2 bytes an item) and late k-mers, or the
 * list of kept slots and the bitmap of a region of at most SK_MAX_INV_LOAD slots a kept one */
template <class KT>
__host__ __device__ constexpr uint32_t sk_late_at(uint32_t slots, uint32_t round) {   /* in 8-byte words, even */
  const size_t items = (size_t)round * SK_ITEMS<KT> * 2, hash = (size_t)sk_hash_size(round) * 4;
  const size_t b = (size_t)slots * (Slot<KT>::KEYW * 8 + 8) + (size_t)round * (SkRec<KT>::NW * 8 + 4) +
                   (items > hash ? items : hash);
  return (uint32_t)((b + 15) / 16 * 2);
}
template <class KT>
__host__ __device__ constexpr size_t sk_count_bytes(uint32_t slots, uint32_t round) {
  const size_t r = (size_t)sk_late_at<KT>(slots, round) * 8 + SK_LATE * (Slot<KT>::KEYW * 8 + 8);
  const size_t l = (size_t)slots * (Slot<KT>::KEYW * 8 + 8 + 2) + 8 + (size_t)(slots * SK_MAX_INV_LOAD) / 8 + 8;
  return r > l ? r : l;
}

/* A k-mer's probe sequence in the shared-memory slots: an odd step of its own, so that runs do not
 * cluster (a lane with a long run holds up its warp, and the last late k-mer its block) */
struct SkSeq {
  uint32_t j, step;
  __device__ __forceinline__ SkSeq(uint32_t h, uint32_t slots) {
    h ^= h >> 16;
    h *= 0xC2B2AE35u;
    j = __umulhi(h, slots);
    step = (h & 30u) | 1u;
  }
  __device__ __forceinline__ SkSeq(KW1 x, uint32_t slots)
      : SkSeq((uint32_t)x.v * 0x9E3779B1u ^ (uint32_t)(x.v >> 32) * 0x85EBCA6Bu, slots) {}
  __device__ __forceinline__ SkSeq(KW2 x, uint32_t slots)
      : SkSeq((uint32_t)x.lo * 0x9E3779B1u ^ (uint32_t)(x.lo >> 32) * 0x85EBCA6Bu ^ (uint32_t)x.hi * 0x27D4EB2Fu ^
                  (uint32_t)(x.hi >> 32) * 0x165667B1u, slots) {}
  __device__ __forceinline__ void next(uint32_t slots) {
    j += step;
    if (j >= slots) j -= slots;
  }
};

/* The shared-memory slots: k <= 31 one 16-byte (key, entries 0-1), read at once and claimed with its
 * first entry by one 128-bit CAS; k > 31 keys and entry pairs in two arrays. */
template <class KT> struct SkSlots;
template <> struct SkSlots<KW1> {
  uint64_t *p;
  uint32_t n;
  __device__ __forceinline__ SkSlots(uint64_t *mem, uint32_t slots) : p(mem), n(slots) {}
  __device__ __forceinline__ void clear(uint32_t i) const { reinterpret_cast<ulonglong2 *>(p)[i] = make_ulonglong2(KEY_EMPTY, 0ull); }
  __device__ __forceinline__ uint32_t *entries(uint32_t j) const { return reinterpret_cast<uint32_t *>(p + 2 * j + 1); }
  __device__ __forceinline__ KW1 key(uint32_t j) const { return {p[2 * j]}; }
  __device__ __forceinline__ uint64_t pair(uint32_t j) const { return p[2 * j + 1]; }
  /* slot j's key and entries as they are, or after claiming it for `want` with `fresh` (claimed) */
  __device__ __forceinline__ KW1 visit(uint32_t j, KW1 want, uint32_t fresh, uint64_t &e, bool &claimed) const {
    const uint32_t a = (uint32_t)__cvta_generic_to_shared(p + 2 * j);
    KW1 x;
    asm volatile("ld.volatile.shared.v2.u64 {%0, %1}, [%2];" : "=l"(x.v), "=l"(e) : "r"(a) : "memory");
    if ((int64_t)x.v < 0) {   /* empty: no key has its top bit set */
      x.v = sm_cas128(a, KEY_EMPTY, 0ull, want.v, (uint64_t)fresh, e);
      claimed = (int64_t)x.v < 0;
    }
    return x;
  }
};
template <> struct SkSlots<KW2> {
  uint64_t *p, *q;
  uint32_t n;
  __device__ __forceinline__ SkSlots(uint64_t *mem, uint32_t slots) : p(mem), q(mem + 2 * slots), n(slots) {}
  __device__ __forceinline__ void clear(uint32_t i) const {
    reinterpret_cast<ulonglong2 *>(p)[i] = make_ulonglong2(KEY_EMPTY, KEY_EMPTY);
    q[i] = 0;
  }
  __device__ __forceinline__ uint32_t *entries(uint32_t j) const { return reinterpret_cast<uint32_t *>(q + j); }
  __device__ __forceinline__ KW2 key(uint32_t j) const { return {p[2 * j], p[2 * j + 1]}; }
  __device__ __forceinline__ uint64_t pair(uint32_t j) const { return q[j]; }
  __device__ __forceinline__ KW2 visit(uint32_t j, KW2 want, uint32_t, uint64_t &e, bool &) const {
    const uint32_t a = (uint32_t)__cvta_generic_to_shared(p + 2 * j);
    KW2 x;
    asm volatile("ld.volatile.shared.v2.u64 {%0, %1}, [%2];" : "=l"(x.lo), "=l"(x.hi) : "r"(a) : "memory");
    if (key_is_empty(x)) {
      KW2 o;
      o.lo = sm_cas128(a, KEY_EMPTY, KEY_EMPTY, want.lo, want.hi, o.hi);
      x = key_is_empty(o) ? want : o;
    }
    e = *(volatile const uint64_t *)(q + j);
    return x;
  }
};

constexpr uint32_t SK_MAX_PROBE = 512;   /* a longer run: the partition is too full */

/* A slot's second entry word carries SK_MORE (its E_BIG bit: no count here reaches 2^24) once the
 * k-mer goes on in a continuation slot. */
constexpr uint32_t SK_MORE = E_BIG;
__device__ __forceinline__ uint32_t sk_count_of(uint32_t w) { return w >> E_COUNT_SHIFT; }

/* `fresh` is an entry word: a code and the occurrences to count.  One entry word of a slot tried for
 * it; `w` is what the word was seen to hold.  SAT: a count from 2^25 on stays where it is (a block's
 * threads, with weights of 2^10 at most, cannot bring it to 2^26 before they see it), and `past` says so */
template <bool SAT = false>
__device__ __forceinline__ bool sk_try_entry(uint32_t *e, uint32_t w, uint32_t fresh, unsigned &claims, bool &past) {
  if (w == 0) {
    w = atomicCAS(e, 0u, fresh);
    if (w == 0) { ++claims; return true; }
  }
  if (entry_code(w) != entry_code(fresh)) return false;
  const uint32_t add = fresh & ~((1u << E_COUNT_SHIFT) - 1);
  if (SAT) {
    past = atomicAdd(e, add) >> 31;
    if (past) atomicSub(e, add);
  } else {
    atomicAdd(e, add);
  }
  return true;
}

/* k-mer records whose occurrences an entry no longer takes, for counts that must be exact (rec: NULL
 * where only the filter reads them) */
struct SkPast { uint64_t *rec; uint64_t cap; DevCounters *ctr; };

/* an entry word's occurrences into the shared-memory slots of a k-mer, continuation slots and all
 * (any lanes may call it); false if the slots are full */
template <class KT, bool SAT>
__device__ __noinline__ bool sk_insert(SkSlots<KT> sl, KT want, uint32_t fresh, unsigned &claims, SkPast over = SkPast{}) {
  constexpr int NW = SkRec<KT>::NW, KWD = Slot<KT>::KEYW;
  const KT kmer = want;
  auto done = [&](bool past) {
    if (!SAT || !past || !over.rec) return true;
    const unsigned long long o = atomicAdd(&over.ctr->n_sk_past, 1ull);
    if (o < over.cap) {
      KOps<KT>::store(over.rec + o * NW, kmer);
      over.rec[o * NW + KWD] = fresh;
    }
    return true;
  };
  bool past = false;
  SkSeq p(want, sl.n);
  for (uint32_t probe = 0; probe < SK_MAX_PROBE; ++probe, p.next(sl.n)) {
    uint64_t seen;
    bool claimed = false;
    const KT key = sl.visit(p.j, want, fresh, seen, claimed);
    if (claimed) { ++claims; return true; }
    if (KOps<KT>::eq(key, want)) {
      uint32_t *e = sl.entries(p.j);
      if (sk_try_entry<SAT>(e, *(volatile uint32_t *)e, fresh, claims, past)) return done(past);
      if (sk_try_entry<SAT>(e + 1, *(volatile uint32_t *)(e + 1), fresh, claims, past)) return done(past);
      atomicOr(e + 1, SK_MORE);
      ((uint64_t *)&want)[KOps<KT>::WORDS - 1] |= KEY_CONT;
    }
  }
  return false;
}

/* fn(entry words 0 and 1) for the k-mer of slot q, then for its continuation slots, in order */
template <class KT, class F>
__device__ __forceinline__ void sk_entries(const SkSlots<KT> &sl, uint32_t q, KT key, F fn) {
  uint64_t e = sl.pair(q);
  fn(e & ~((uint64_t)SK_MORE << 32));
  if (!((e >> 32) & SK_MORE)) return;
  SkSeq p(key, sl.n);   /* the k-mer's own sequence, from slot q on */
  ((uint64_t *)&key)[KOps<KT>::WORDS - 1] |= KEY_CONT;
  p.j = q;
  do {   /* its next slot lies further on */
    KT x;
    do {
      p.next(sl.n);
      x = sl.key(p.j);
    } while (!KOps<KT>::eq(x, key) && !key_is_empty(x));
    if (key_is_empty(x)) return;
    e = sl.pair(p.j);
    fn(e & ~((uint64_t)SK_MORE << 32));
  } while ((e >> 32) & SK_MORE);
}

/* a k-mer with a longer probe run, or whose slot's two entries are taken, waits here until the
 * round's others are counted: its warp's other lanes would wait for it */
template <class KT> struct SkLate { KT key; uint64_t fresh; };

/* the first ten bases of a k-mer */
__device__ __forceinline__ uint32_t sk_top20(KW1 x, int k) { return (uint32_t)(x.v >> (2 * k - 20)) & 0xFFFFFu; }
__device__ __forceinline__ uint32_t sk_top20(KW2 x, int k) { return (uint32_t)KOps<KW2>::shr(x, 2 * k - 20).lo & 0xFFFFFu; }

/* local_insert_by_freqencies for one k-mer (filter_kmer's steps over entries in shared memory): the
 * node's counters, 0 if no entry is kept, 1 for a chain node, 2 for a branch node.  The entries'
 * flags 0..3 are tallied in the bytes of `few`, others in hist.
 *
 * EF: the blocked driver's (k+1)-mer filter instead.  Every (k+1)-mer of a read is an out edge of its
 * first k-mer and an in edge of its second, so an edge's occurrences over the k-mer's entries are
 * those of its (k+1)-mer: no table of (k+1)-mers.  Twice those where the (k+1)-mer is its own reverse
 * complement (both its k-mers are this one); and where the k-mer is, its out edge in b is its in edge
 * in the complement of b, seen from the other strand.  Edges outside the bounds leave the entries;
 * entries then alike are one, entries without edges none (flag 0 tallies what is left).  Edges of reads of
 * k + 1 bases (sk_edge_bases) count for the (k+1)-mers alone. */
template <class KT, bool EF>
__device__ __forceinline__ int sk_node(const SkSlots<KT> &sl, uint32_t q, KT key, const SkCount &a, uint64_t *pw,
                                       uint32_t &few, unsigned int *hist) {
  const int k = a.k;
  const unsigned first = KOps<KT>::first(key, k), last = KOps<KT>::last(key);
  /* a palindrome's ends are complements: eight bases at the ends of the k-mer and of its two
   * (k-1)-mers rule all but one in 2^16 out before the whole is compared */
  const uint32_t tail = (uint32_t)((const uint64_t *)&key)[0], head = sk_top20(key, k), rt = rev_pairs32(~tail);
  bool oddk = (k & 1) != 0, kpal = false, high = false, low = false;
  if (oddk) {
    if ((head >> 4) == rev_pairs32(~(tail >> 2)) >> 16) high = km1_high_palindrome(key, k);
    if (((head >> 2) & 0xFFFFu) == rt >> 16) low = km1_low_palindrome(key, k);
  } else if ((head >> 4) == rt >> 16) {
    kpal = k_palindrome(key, k);
  }
  uint32_t kf = 0, ok = 0;   /* ok: bit c (4 + c): the (k+1)-mers over in (out) base c are kept */
  if (EF || a.thresholding) {
    uint32_t k1[8] = {0, 0, 0, 0, 0, 0, 0, 0};
    sk_entries<KT>(sl, q, key, [&](uint64_t x) {
      #pragma unroll
      for (int z = 0; z < 2; ++z) {
        const uint32_t w = (uint32_t)(x >> (32 * z));
        if (w == 0) continue;
        const uint32_t c = sk_count_of(w), half = (c + 1) >> 1;
        const unsigned code = entry_code(w);
        unsigned in5 = code_in5(code), out5 = code_out5(code);
        if (EF) sk_edge_bases(code, in5, out5);
        kf += c;
        const uint32_t vi = !EF && oddk && high && !kpal && last == 4u - in5 ? half : c;
        const uint32_t vo = !EF && oddk && low && !kpal && first == 4u - out5 ? half : c;
        #pragma unroll
        for (unsigned b = 0; b < 4; ++b) {
          k1[b] += in5 == b + 1 ? vi : 0u;
          k1[4 + b] += out5 == b + 1 ? vo : 0u;
        }
      }
    });
    kf = min(0xFFFFu, kf);
    #pragma unroll
    for (int b = 0; b < 8; ++b) {
      uint32_t v = k1[b];
      if (EF && kpal) v += k1[7 - b];
      if (EF && (b < 4 ? high && last == 3u - b : low && first == 7u - b)) v >>= 1;
      v = min(0xFFFFu, v);
      ok |= v >= a.t[2] && v < a.t[3] ? 1u << b : 0u;
    }
  }
  uint32_t nc[9] = {0, 0, 0, 0, 0, 0, 0, 0, 0};
  bool any = false;
  uint32_t left = 0;   /* EF: the codes of the entries that are left */
  sk_entries<KT>(sl, q, key, [&](uint64_t x) {
    #pragma unroll
    for (int z = 0; z < 2; ++z) {
      const uint32_t w = (uint32_t)(x >> (32 * z));
      if (w == 0) continue;
      const uint32_t c16 = min(0xFFFFu, sk_count_of(w));
      const unsigned code = entry_code(w);
      unsigned in5 = code_in5(code), out5 = code_out5(code), f = 0;
      if (EF) {
        if (sk_edge_bases(code, in5, out5)) continue;
        if (!((ok << 1) >> in5 & 1u)) in5 = 0;
        if (!((ok >> 3) >> out5 & 1u)) out5 = 0;
        if (in5 == 0 && out5 == 0) continue;
        left |= 1u << biedge_code(in5, out5);
      } else if (a.thresholding) {   /* an absent base counts as a (k+1)-mer outside the bounds */
        if (c16 < a.t[4] || c16 >= a.t[5]) f |= 4;
        if (kf < a.t[0] || kf >= a.t[1]) f |= 8;
        if (!((ok << 1) >> in5 & 1u) || !in5) f |= 2;
        if (!((ok >> 3) >> out5 & 1u) || !out5) f |= 1;
      }
      if (EF) ;
      else if (f < 4) few += 1u << (8 * f);   /* (at most 25 entries a k-mer) */
      else atomicAdd(&hist[f], 1u);
      if (f >= 3) continue;
      if (f == 1) out5 = 0;
      if (f == 2) in5 = 0;
      any = true;
      #pragma unroll
      for (unsigned b = 0; b < 4; ++b) {
        nc[b] += out5 == b + 1 ? c16 : 0u;
        nc[4 + b] += in5 == b + 1 ? c16 : 0u;
      }
      nc[8] += c16;
    }
  });
  if (!any) return 0;
  if (EF) few += __popc(left);
  unsigned din = 0, dout = 0;   /* IsBranchPoint / IsChainNode (debruijn_graph_filters.hpp:57-220) */
  bool k1pal = false;
  #pragma unroll
  for (unsigned b = 0; b < 4; ++b) {
    dout += nc[b] > 0;
    din += nc[4 + b] > 0;
    if (oddk && nc[b] > 0 && low && (first == 3u - b || first == b)) k1pal = true;
    if (oddk && nc[4 + b] > 0 && high && (last == 3u - b || last == b)) k1pal = true;
  }
  #pragma unroll
  for (int b = 0; b < 9; ++b) nc[b] = min(0xFFFFu, nc[b]);
  pw[0] = (uint64_t)(nc[0] | (nc[1] << 16)) | ((uint64_t)(nc[2] | (nc[3] << 16)) << 32);
  pw[1] = (uint64_t)(nc[4] | (nc[5] << 16)) | ((uint64_t)(nc[6] | (nc[7] << 16)) << 32);
  pw[2] = nc[8];
  return din >= 2 || dout >= 2 || kpal || k1pal ? 2 : 1;
}

/* Equal records merge into the first that claimed an entry of the record hash, which then has their
 * number as its weight (a third of the entries stays free; every thread of the block calls it) */
template <int NW>
__device__ __forceinline__ void sk_merge(const uint64_t *s_rec, uint32_t *s_wt, uint32_t *s_hash, uint32_t hmask,
                                         uint32_t nr, uint32_t tid, uint32_t nt) {
  for (uint32_t i = tid; i < nr; i += nt) {
    ulonglong2 rec[NW / 2];
    uint64_t z = 0;
    #pragma unroll
    for (int q = 0; q < NW / 2; ++q) {
      rec[q] = reinterpret_cast<const ulonglong2 *>(s_rec + (size_t)i * NW)[q];
      z = (z ^ rec[q].x) * 0x9E3779B97F4A7C15ull ^ rec[q].y ^ (z >> 29);
    }
    z *= 0xD6E8FEB86659FD93ull;
    uint32_t h = (uint32_t)(z >> 52) & hmask;
    for (;;) {
      const uint32_t o = atomicCAS(&s_hash[h], ~0u, i);
      if (o == ~0u) { atomicAdd(&s_wt[i], 1u); break; }
      bool same = true;
      #pragma unroll
      for (int q = 0; q < NW / 2; ++q) {
        const ulonglong2 v = reinterpret_cast<const ulonglong2 *>(s_rec + (size_t)o * NW)[q];
        same &= v.x == rec[q].x && v.y == rec[q].y;
      }
      if (same) { atomicAdd(&s_wt[o], 1u); break; }
      h = (h + 1) & hmask;
    }
  }
}

/* lex_less: the smaller strand's biedge, reverse-complemented on a flip */
__device__ __forceinline__ unsigned sk_code(bool fwd, unsigned in5, unsigned out5, bool edge) {
  const unsigned in = fwd ? in5 : out5 ? 5u - out5 : 0u, out = fwd ? out5 : in5 ? 5u - in5 : 0u;
  return edge ? sk_edge_code(in, out) : biedge_code(in, out);
}

/* ------------------------------------------------------------ crowded partitions
 * A minimizer that many places share (a tail of one base, an adapter, a satellite: k-mers that hold it
 * and some of what lies around) can put more k-mers into a partition than a block's slots, or more
 * records than one block should count.  Such a partition is cut by its k-mers' keys: its records go
 * through blocks of SK_CHUNK, which merge the equal ones and write each k-mer with its weight to one of
 * 2^lg parts, first counted, then placed; a part holds some thousand k-mers, is counted by a block and
 * has a region of its own, which lookups find by the key.  160M k-mers, adapters in 2% of the reads:
 * 5.9 ms a build (4.9 without the adapters); by k-mer records, where such an input used to go after the
 * count had been tried at three sizes, 29.9, of which the k-mer records themselves take 17.1.  Bound by
 * the latency of few blocks: these adapters' 70 chunks take 0.04 ms to count and 0.05 to place, their
 * parts 0.15 to count. */
struct SkChunk { uint32_t r0, n, sub0, lg; };   /* records, first part, log2 of the parts */
template <int NW> constexpr uint32_t SK_CHUNK = 2048 / NW;
/* records of a partition at most that one block counts (a typical one: 500), and below 2^26 k-mers */
constexpr uint32_t SK_MAX_RECORDS = 1u << 15;

template <class KT, bool WRITE>
__global__ void __launch_bounds__(256) k_sk_expand(const uint64_t *recs, const SkChunk *chunks, int k,
                                                   unsigned long long *cur, uint64_t *out) {
  constexpr int NW = SkRec<KT>::NW;
  constexpr uint32_t N = SK_CHUNK<NW>, H = 2 * N;
  __shared__ __align__(16) uint64_t s_rec[N * NW];
  __shared__ uint32_t s_wt[N], s_hash[H];
  const SkChunk ch = chunks[blockIdx.x];
  const uint32_t tid = threadIdx.x, nt = blockDim.x;
  for (uint32_t i = tid; i < ch.n * (NW / 2); i += nt)
    reinterpret_cast<ulonglong2 *>(s_rec)[i] = reinterpret_cast<const ulonglong2 *>(recs + (uint64_t)ch.r0 * NW)[i];
  for (uint32_t i = tid; i < N; i += nt) s_wt[i] = 0;
  for (uint32_t i = tid; i < H; i += nt) s_hash[i] = ~0u;
  __syncthreads();
  sk_merge<NW>(s_rec, s_wt, s_hash, H - 1, ch.n, tid, nt);
  __syncthreads();
  for (uint32_t i = tid; i < ch.n; i += nt) {
    const uint32_t weight = s_wt[i] << E_COUNT_SHIFT;
    if (!weight) continue;
    const uint64_t *w = s_rec + (size_t)i * NW;
    const uint64_t last = w[NW - 1];
    const int nk = (int)sk_n(last), n_out = nk - ((last & SK_RIGHT) ? 0 : 1);
    KT f = KOps<KT>::extract(w, 1, k), r = KOps<KT>::rc(f, k);
    unsigned in5 = (last & SK_LEFT) ? sk_base<NW>(w, 0) + 1u : 0u;
    for (int d = 0; d < nk; ++d) {
      const unsigned c = d < n_out ? sk_base<NW>(w, d + k + 1) : 0u;
      const bool fwd = KOps<KT>::lt(f, r);
      const KT key = fwd ? f : r;
      const uint32_t fresh = (sk_code(fwd, in5, d < n_out ? c + 1u : 0u, sk_edge(last)) << E_CODE_SHIFT) | weight;
      in5 = KOps<KT>::first(f, k) + 1u;
      f = KOps<KT>::append(f, c, k);
      r = KOps<KT>::prepend(3u - c, r, k);
      const unsigned long long o = atomicAdd(&cur[ch.sub0 + (key_sub(table_key(key)) & ((1u << ch.lg) - 1u))], 1ull);
      if constexpr (WRITE) {
        ulonglong2 *to = reinterpret_cast<ulonglong2 *>(out + o * NW);
        if constexpr (NW == 2) {
          to[0] = make_ulonglong2(((const uint64_t *)&key)[0], (uint64_t)fresh);
        } else {
          to[0] = make_ulonglong2(((const uint64_t *)&key)[0], ((const uint64_t *)&key)[KOps<KT>::WORDS - 1]);
          to[1] = make_ulonglong2((uint64_t)fresh, 0ull);
        }
      }
    }
  }
}

struct SkCrowd { uint32_t part, sub0, lg, smp; };
/* the records of the listed partitions */
__global__ void k_sk_crowd_records(const uint32_t *list, uint32_t n, const uint32_t *off, uint2 *out) {
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) out[i] = make_uint2(off[list[i]], off[list[i] + 1] - off[list[i]]);
}
/* crowded partitions' entries of the partition table, and their parts' samples */
__global__ void k_sk_crowd_mark(const SkCrowd *crowd, uint32_t parts, uint2 *info, uint32_t *sub_smp) {
  const SkCrowd x = crowd[blockIdx.x];
  if (threadIdx.x == 0) info[x.part] = make_uint2(parts + x.sub0, SK_SUBS | x.lg);
  for (uint32_t i = threadIdx.x; i < 1u << x.lg; i += blockDim.x) sub_smp[x.sub0 + i] = x.smp;
}
__global__ void k_sk_crowd_off(const unsigned long long *base, uint32_t n, uint32_t *off) {
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) off[i] = (uint32_t)base[i];
}

/* Those records, once the table is written: their occurrences go to the side table of counts past an
 * entry word's own, under the word's address (one sample's table) */
template <class KT>
__global__ void __launch_bounds__(256) k_sk_past(const uint64_t *rec, uint64_t n, uint64_t *table, const SGeom *sg,
                                                 DevCounters *ctr) {
  constexpr int SU = Slot<KT>::U64, KWD = Slot<KT>::KEYW, NE = Slot<KT>::ENTRIES, NW = SkRec<KT>::NW;
  for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (uint64_t)gridDim.x * blockDim.x) {
    const KT x = KOps<KT>::load(rec + i * NW), t = table_key(x);
    const uint32_t fresh = (uint32_t)rec[i * NW + KWD];
    uint32_t *at = nullptr;
    Probe pr = table_probe(sg[0].g, x, t);
    for (uint64_t p = pr.lo; p < pr.hi && !at; ++p, pr.next()) {
      const KT key = KOps<KT>::load(table + pr.i * SU);
      if (key_is_empty(key)) break;
      if (!key_matches(key, t, false) && !key_matches(key, t, true)) continue;
      uint32_t *e = reinterpret_cast<uint32_t *>(table + pr.i * SU + KWD);
      for (int q = 0; q < NE && !at; ++q)
        if (e[q] && entry_code(e[q]) == entry_code(fresh)) at = e + q;
    }
    if (!at) { atomicOr(&ctr->err, (unsigned long long)DERR_INVARIANT); continue; }
    atomicOr(at, E_BIG);
    big_add(ctr, (unsigned long long)(uintptr_t)at, fresh >> E_COUNT_SHIFT);
  }
}

/* SUB: the parts of crowded partitions, from their k-mers' records (off, todo and over are theirs) */
template <class KT, bool EF, bool SUB>
__global__ void __launch_bounds__(SK_COUNT_TPB, sizeof(KT) == 8 ? 4 : 3) k_sk_count(SkCount a) {
  constexpr int SU = Slot<KT>::U64, KWD = Slot<KT>::KEYW, NE = Slot<KT>::ENTRIES, NW = SkRec<KT>::NW;
  extern __shared__ __align__(16) uint64_t sm[];
  __shared__ uint32_t s_items, s_full, s_listed, s_other, s_conts, s_wide, s_base, s_slots, s_late_n, s_smp;
  __shared__ unsigned int s_qh[4], s_claims, s_hist[16], s_nc[2];
  __shared__ unsigned long long s_nbase[2];
  __shared__ unsigned long long s_cand;
  if (a.ctr->err & DERR_SKEW) return;
  uint32_t part = a.todo ? a.todo[blockIdx.x] : blockIdx.x;
  if (!SUB && a.cls && !a.todo) {
    uint32_t lo = 0, hi = a.ncls;
    while (hi - lo > 1) { const uint32_t m = (lo + hi) >> 1; if (__ldg(&a.cls[m].run) <= blockIdx.x) lo = m; else hi = m; }
    part = a.cls[lo].pbase + (blockIdx.x - a.cls[lo].run);
  }
  const int tid = threadIdx.x, lane = tid & 31, k = a.k;
  const uint32_t nt = blockDim.x, slots = a.slots, round = a.round;
  const SkSlots<KT> sl(sm, slots);
  uint64_t *s_rec = sm + (size_t)slots * (KWD + 1);
  uint32_t *s_wt = reinterpret_cast<uint32_t *>(s_rec + (size_t)round * NW), *s_hash = s_wt + round;
  uint16_t *s_list = reinterpret_cast<uint16_t *>(s_hash);
  SkLate<KT> *s_late = reinterpret_cast<SkLate<KT> *>(sm + a.late);
  if (!SUB && a.off[part + 1] - a.off[part] > SK_MAX_RECORDS) {
    if (tid == 0) a.over[atomicAdd(&a.ctr->n_over, 1ull)] = part;
    return;
  }
  for (uint32_t i = tid; i < slots; i += nt) sl.clear(i);
  if (tid < 4) s_qh[tid] = 0;
  if (tid < 16) s_hist[tid] = 0;
  if (tid < 2) s_nc[tid] = 0;
  if (tid == 0) { s_full = 0; s_listed = 0; s_other = 0; s_conts = 0; s_wide = 0; s_claims = 0; }
  const uint32_t hmask = a.hsize - 1;
  unsigned claims = 0;
  const uint32_t r1 = a.off[part + 1];
  if constexpr (SUB) {
    __syncthreads();
    for (uint32_t i = a.off[part] + tid; i < r1; i += nt) {
      const uint64_t *w = a.recs + (uint64_t)i * NW;
      if (!*(volatile uint32_t *)&s_full && !sk_insert<KT, true>(sl, KOps<KT>::load(w), (uint32_t)w[KWD], claims, SkPast{a.past, a.past_cap, a.ctr}))
        s_full = 1;
    }
  }
  for (uint32_t r0 = a.off[part]; !SUB && r0 < r1; r0 += round) {
    const uint32_t nr = min(round, r1 - r0);
    for (uint32_t i = tid; i < nr * (NW / 2); i += nt)
      reinterpret_cast<ulonglong2 *>(s_rec)[i] = __ldcs(reinterpret_cast<const ulonglong2 *>(a.recs + (uint64_t)r0 * NW) + i);
    for (uint32_t i = tid; i < nr; i += nt) s_wt[i] = 0;
    for (uint32_t i = tid; i <= hmask; i += nt) s_hash[i] = ~0u;
    if (tid == 0) { s_items = 0; s_late_n = 0; }
    __syncthreads();
    sk_merge<NW>(s_rec, s_wt, s_hash, hmask, nr, tid, nt);
    __syncthreads();
    /* the distinct records' k-mers as items of SK_ITEM */
    for (uint32_t i0 = 0; i0 < nr; i0 += nt) {
      const uint32_t i = i0 + tid;
      const unsigned n = i < nr && s_wt[i] ? sk_n<EF>(s_rec[(size_t)i * NW + NW - 1]) : 0u;
      const uint32_t ni = (n + SK_ITEM - 1) / SK_ITEM;
      uint32_t x = ni;
      #pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const uint32_t y = __shfl_up_sync(~0u, x, o);
        if (lane >= o) x += y;
      }
      uint32_t at = 0;
      if (lane == 31 && x) at = atomicAdd(&s_items, x);
      at = __shfl_sync(~0u, at, 31) + x - ni;
      for (uint32_t q = 0; q < ni; ++q) s_list[at + q] = (uint16_t)(i | (q << 10));
    }
    __syncthreads();
    const uint32_t items = s_items;
    /* the warp's lanes stay together: every loop's bound is the warp's or fixed */
    for (uint32_t y0 = tid & ~31u; y0 < items; y0 += nt) {
      const bool has = y0 + lane < items;
      const uint32_t it = has ? s_list[y0 + lane] : 0u, id = it & 1023u;
      const int o0 = SK_ITEM * (int)(it >> 10);
      const uint64_t *w = s_rec + (size_t)id * NW;
      const uint64_t last = w[NW - 1];
      const int nk = (int)sk_n<EF>(last), n = has ? min(nk - o0, SK_ITEM) : 0;
      const uint32_t weight = (s_wt[id] << E_COUNT_SHIFT) | (sk_edge<EF>(last) ? 1u : 0u);   /* (lowest bit: an edge) */
      KT f = KOps<KT>::extract(w, o0 + 1, k), r = KOps<KT>::rc(f, k);
      /* in5, out5 of the k-mers: the base before (0: none), then the bases after from the top of `next` */
      unsigned in5 = o0 > 0 || (last & SK_LEFT) ? sk_base<NW>(w, o0) + 1u : 0u;
      const int b = o0 + k + 1;
      const uint64_t n0 = w[b >> 5] << (2 * (b & 31)), n1 = (b >> 5) + 1 < NW ? w[(b >> 5) + 1] : 0ull;
      uint32_t next = (uint32_t)((n0 | ((b & 31) ? n1 >> (64 - 2 * (b & 31)) : 0ull)) >> 32);
      const int n_out = nk - o0 - ((last & SK_RIGHT) ? 0 : 1);   /* k-mers of the item that have a base after */
      for (int d = 0; __any_sync(~0u, d < n); ++d) {
        bool todo = d < n;
        const unsigned c = next >> 30, out5 = d < n_out ? c + 1u : 0u;
        next <<= 2;
        const bool fwd = KOps<KT>::lt(f, r);
        const KT key = fwd ? f : r;
        const unsigned code = sk_code(fwd, in5, out5, EF && (weight & 1u));
        const uint32_t fresh = (code << E_CODE_SHIFT) | (weight & ~1u);
        in5 = KOps<KT>::first(f, k) + 1u;
        f = KOps<KT>::append(f, c, k);
        r = KOps<KT>::prepend(3u - c, r, k);
        /* the k-mer's slot within two probes, then its entry among the slot's two */
        SkSeq p(key, slots);
        uint64_t seen = 0;
        bool seek = todo;
        #pragma unroll
        for (int probe = 0; probe < 2; ++probe) {
          if (seek) {
            bool claimed = false;
            const KT x = sl.visit(p.j, key, fresh, seen, claimed);
            if (claimed) { ++claims; todo = false; }
            seek = !claimed && !KOps<KT>::eq(x, key);
            if (seek) p.next(slots);
          }
        }
        if (todo && !seek) {
          uint32_t *e = sl.entries(p.j);
          uint32_t cur = (uint32_t)seen;
          if (cur != 0 && entry_code(cur) != code) { cur = (uint32_t)(seen >> 32); ++e; }
          bool past;
          todo = !sk_try_entry(e, cur, fresh, claims, past);
        }
        if (todo) {   /* the rest, later */
          const uint32_t at = atomicAdd(&s_late_n, 1u);
          if (at < SK_LATE) s_late[at] = SkLate<KT>{key, fresh};
          else if (!*(volatile uint32_t *)&s_full && !sk_insert<KT, false>(sl, key, fresh, claims)) s_full = 1;
        }
        __syncwarp();
      }
    }
    __syncthreads();
    const uint32_t late = min(s_late_n, SK_LATE);
    for (uint32_t y = tid; y < late; y += nt)
      if (!*(volatile uint32_t *)&s_full && !sk_insert<KT, false>(sl, s_late[y].key, (uint32_t)s_late[y].fresh, claims)) s_full = 1;
    __syncthreads();
    if (s_full) break;
  }
  __syncthreads();
  if (s_full) {   /* counted again with more slots: nothing of it is tallied or written */
    if (tid == 0) a.over[atomicAdd(&a.ctr->n_over, 1ull)] = part;
    return;
  }
  /* which k-mers to keep, by slot: the listed ones from the front of the list, others (keep_all) from
   * its back (the list and the region's bitmap take the memory of the records and all behind it) */
  uint16_t *kept = reinterpret_cast<uint16_t *>(s_rec);
  uint64_t qh = 0;   /* quick drops' flags 3 | 8 | 4 as 16-bit fields (a thread sees under 2^11 slots) */
  uint32_t my_conts = 0;
  uint32_t t_low = a.thresholding ? a.t[2] : 0u;
  if (EF && !(k & 1)) t_low = (t_low + 1) / 2;   /* (a palindrome's edges occur up to twice as often as it) */
  const bool no_bounds = a.t[0] == 0 && a.t[1] > 0xFFFFu && a.t[4] == 0 && a.t[5] > 0xFFFFu;   /* flags 3 only */
  for (uint32_t q0 = tid & ~31u; q0 < slots; q0 += nt) {
    const uint32_t q = q0 + lane;   /* slots are a multiple of 32 */
    const KT key = sl.key(q);
    bool listed = false, keep = false;
    if (!key_is_empty(key)) {
      if (key_cont(key)) {
        ++my_conts;
      } else {
        const uint64_t e = sl.pair(q);
        const uint32_t c0 = sk_count_of((uint32_t)e), c1 = sk_count_of((uint32_t)(e >> 32));
        const bool more = ((e >> 32) & SK_MORE) != 0;
        uint32_t kf = c0 + c1;
        if (more && kf < t_low) {   /* the total needs the continuation slots */
          kf = 0;
          sk_entries<KT>(sl, q, key, [&](uint64_t x) { kf += sk_count_of((uint32_t)x) + sk_count_of((uint32_t)(x >> 32)); });
        }
        kf = min(0xFFFFu, kf);
        listed = kf >= t_low;
        keep = listed || a.keep_all;
        if (!EF && !listed) {
          if (no_bounds && !more) {
            qh += 1 + (c1 != 0);
          } else {
            const uint32_t kout = (kf < a.t[0] || kf >= a.t[1]) ? 2u : 0u;
            sk_entries<KT>(sl, q, key, [&](uint64_t x) {
              #pragma unroll
              for (int z = 0; z < 2; ++z) {
                const uint32_t c16 = min(0xFFFFu, sk_count_of((uint32_t)(x >> (32 * z))));
                if (c16) qh += 1ull << (16 * (kout | ((c16 < a.t[4] || c16 >= a.t[5]) ? 1u : 0u)));
              }
            });
          }
        }
      }
    }
    const unsigned ml = __ballot_sync(~0u, listed), below = (1u << lane) - 1;
    uint32_t at = 0;
    if (ml) {
      if (lane == 0) at = atomicAdd(&s_listed, (uint32_t)__popc(ml));
      at = __shfl_sync(~0u, at, 0);
      if (listed) kept[at + __popc(ml & below)] = (uint16_t)q;
    }
    if (a.keep_all) {
      const unsigned mo = __ballot_sync(~0u, keep && !listed);
      if (lane == 0 && mo) at = atomicAdd(&s_other, (uint32_t)__popc(mo));
      at = __shfl_sync(~0u, at, 0);
      if (keep && !listed) kept[slots - 1 - (at + __popc(mo & below))] = (uint16_t)q;
    }
  }
  my_conts = (uint32_t)warp_sum(my_conts);
  claims = (unsigned)warp_sum(claims);
  if (lane == 0) {
    if (my_conts) atomicAdd(&s_conts, my_conts);
    if (claims) atomicAdd(&s_claims, claims);
  }
  #pragma unroll
  for (int f = 0; f < 4; ++f) {
    const unsigned long long h = warp_sum((qh >> (16 * f)) & 0xFFFFull);
    if (lane == 0 && h) atomicAdd(&s_qh[f], (unsigned)h);
  }
  __syncthreads();
  const uint32_t listed = s_listed, nkept = listed + s_other;
  /* table slots: one a kept k-mer, and a k-mer of more entries than that holds has three continuation
   * slots here for every one it takes there.  Two slots at least of the region stay empty, which
   * ends every probe run. */
  const uint32_t tslots = nkept + s_conts / (NE / 2), want_R = (uint32_t)(tslots * a.inv_load) + 2u;
  /* the first nodes, one a thread, before the reservations: region, chain and branch indices are
   * then taken at once, by three warps */
  int kind = 0;
  KT t{};
  uint64_t pw[3] = {0, 0, 0};
  uint32_t few = 0, at = 0;
  auto make_node = [&](uint32_t x) {   /* every thread of the block */
    kind = 0;
    if (x < nkept) {
      const KT key = sl.key(kept[x]);
      kind = sk_node<KT, EF>(sl, kept[x], key, a, pw, few, s_hist);
      t = table_key(key);
    }
    const unsigned mc = __ballot_sync(~0u, kind == 1), mb = __ballot_sync(~0u, kind == 2);
    uint32_t oc = 0, ob = 0;
    if (lane == 0) {
      oc = mc ? atomicAdd(&s_nc[0], (unsigned)__popc(mc)) : 0u;
      ob = mb ? atomicAdd(&s_nc[1], (unsigned)__popc(mb)) : 0u;
    }
    oc = __shfl_sync(~0u, oc, 0) + __popc(mc & ((1u << lane) - 1));
    ob = __shfl_sync(~0u, ob, 0) + __popc(mb & ((1u << lane) - 1));
    at = kind == 2 ? ob : oc;
    /* the flags' bytes, summed over the warp in 16-bit halves */
    const uint32_t f02 = __reduce_add_sync(~0u, few & 0x00FF00FFu), f13 = __reduce_add_sync(~0u, (few >> 8) & 0x00FF00FFu);
    few = 0;
    if (lane < 4) {
      const uint32_t f = ((lane & 1 ? f13 : f02) >> (lane & 2 ? 16 : 0)) & 0xFFFFu;
      if (f) atomicAdd(&s_hist[lane], f);
    }
  };
  auto reserve = [&](int list, uint32_t smp) {   /* one thread: the block's chain (0) or branch (1) indices */
    const uint32_t n = s_nc[list];
    if (!n) return;
    s_nbase[list] = atomicAdd(list ? &a.ctr->n_branch : &a.ctr->n_chain, (unsigned long long)n);
    if (a.s_tally) atomicAdd(&a.s_tally[(uint64_t)smp * T_NUM + (list ? T_BRANCH : T_CHAIN)], (unsigned long long)n);
  };
  if (EF || a.nodes) {
    make_node(tid);
    __syncthreads();
  }
  if ((EF || a.nodes) && (tid == 32 || tid == 64))
    reserve(tid / 32 - 1, SUB ? a.sub_smp[part] : sample_of_part(a.sg, a.nsamples, part));
  if (tid == 0) {
    const uint32_t R = want_R;
    const uint32_t smp = SUB ? a.sub_smp[part] : sample_of_part(a.sg, a.nsamples, part);
    const TableGeom &g = a.sg[smp].g;
    const unsigned long long lo = atomicAdd(&a.bump[smp], (unsigned long long)R);
    s_cand = a.cand ? atomicAdd(&a.ctr->n_cand, (unsigned long long)listed) : 0ull;
    const bool fits = lo + R <= g.nslots;
    if (!fits) atomicOr(&a.ctr->err, (unsigned long long)DERR_TABLE_FULL);
    s_slots = fits ? R : 0;
    s_smp = smp;
    s_base = (uint32_t)(g.base + lo);
    a.info[SUB ? a.sub0 + part : part] = make_uint2((uint32_t)(g.base + lo), R);
    if (!a.cand) atomicAdd(&a.ctr->n_cand, (unsigned long long)listed);
    if (tslots) atomicAdd(&a.ctr->n_slots_claimed, (unsigned long long)tslots);
    if (!EF && s_claims) atomicAdd(&a.ctr->n_entries, (unsigned long long)s_claims);
    if (a.s_tally && s_claims) atomicAdd(&a.s_tally[(uint64_t)smp * T_NUM + T_ENTRIES], (unsigned long long)s_claims);
  }
  if (tid < 4 && s_qh[tid]) atomicAdd(&a.ctr->quick_hist[3 + 4 * tid], (unsigned long long)s_qh[tid]);
  /* the places taken in the region, a bit each, behind the list */
  uint32_t *taken = reinterpret_cast<uint32_t *>(kept) + (slots + 1) / 2;
  for (uint32_t i = tid; i < (want_R + 31u) / 32; i += nt) taken[i] = 0;
  __syncthreads();
  const uint32_t R = s_slots;
  if (R == 0) return;
  uint64_t *dst = a.table + (uint64_t)s_base * SU;
  auto place = [&](uint32_t pos) {   /* the first free place from pos on */
    for (;;) {
      const uint32_t bit = 1u << (pos & 31);
      if (!(atomicOr(&taken[pos >> 5], bit) & bit)) return pos;
      if (++pos == R) pos = 0;
    }
  };
  if (EF || a.nodes) {   /* the nodes themselves */
    for (uint32_t x0 = 0;;) {
      if (kind) {
        const unsigned long long o = s_nbase[kind - 1] + at;
        const uint32_t pos = place(bin_home(t, R));
        const uint64_t aux = kind == 1 ? o : 0xFFFFFFFFull;
        pw[2] |= (uint64_t)((kind == 1 ? NF_CHAIN : NF_BRANCH) | (s_smp << NF_SAMPLE_SHIFT)) << 16 | aux << 32;
        t = as_node(t);
        ulonglong2 *to = reinterpret_cast<ulonglong2 *>(dst + (uint64_t)pos * SU);
        if constexpr (KWD == 1) {
          to[0] = make_ulonglong2(((const uint64_t *)&t)[0], pw[0]);
          to[1] = make_ulonglong2(pw[1], pw[2]);
        } else {
          to[0] = make_ulonglong2(((const uint64_t *)&t)[0], ((const uint64_t *)&t)[KWD - 1]);
          to[1] = make_ulonglong2(pw[0], pw[1]);
          to[2] = make_ulonglong2(pw[2], 0ull);
          to[3] = make_ulonglong2(0ull, 0ull);
        }
        if (o < a.list_cap) (kind == 1 ? a.chain_list : a.branch_list)[o] = s_base + pos;
        else atomicOr(&a.ctr->err, (unsigned long long)DERR_TABLE_FULL);
      }
      x0 += nt;
      if (x0 >= nkept) break;
      __syncthreads();
      if (tid < 2) s_nc[tid] = 0;
      __syncthreads();
      make_node(x0 + tid);
      __syncthreads();
      if (tid == 32 || tid == 64) reserve(tid / 32 - 1, s_smp);
      __syncthreads();
    }
  }
  for (uint32_t x = tid; x < (EF || a.nodes ? 0u : nkept); x += nt) {
    const uint32_t q = x < listed ? kept[x] : kept[slots - 1 - (x - listed)];
    const KT key = sl.key(q), t = table_key(key);
    const uint32_t pos = place(bin_home(t, R));
    ulonglong2 *to = reinterpret_cast<ulonglong2 *>(dst + (uint64_t)pos * SU);
    const uint64_t e = sl.pair(q);
    #pragma unroll
    for (int i = 0; i < SU; i += 2) {
      uint64_t v[2] = {0, 0};
      #pragma unroll
      for (int z = 0; z < 2; ++z)
        if (i + z < KWD) v[z] = ((const uint64_t *)&t)[i + z];
        else if (i + z == KWD) v[z] = e & ~((uint64_t)SK_MORE << 32);
      to[i / 2] = make_ulonglong2(v[0], v[1]);
    }
    if ((e >> 32) & SK_MORE) {
      int n = KWD;
      sk_entries<KT>(sl, q, key, [&](uint64_t x) {
        if (n > KWD && n < SU) dst[(uint64_t)pos * SU + n] = x;
        if (n == SU) s_wide = 1;
        ++n;
      });
    }
    if (x < listed) a.cand[s_cand + x] = s_base + pos;
  }
  __syncthreads();
  if (tid < 16 && s_hist[tid]) atomicAdd(&a.ctr->flag_hist[tid], (unsigned long long)s_hist[tid]);
  if (s_wide)   /* k-mers of more entries than a table slot holds: continuation slots behind the first */
    for (uint32_t x = tid; x < nkept; x += nt) {
      const uint32_t q = x < listed ? kept[x] : kept[slots - 1 - (x - listed)];
      const KT key = sl.key(q);
      KT t = table_key(key);
      ((uint64_t *)&t)[KWD - 1] |= KEY_CONT;
      uint64_t *to = nullptr;
      int n = 0;
      sk_entries<KT>(sl, q, key, [&](uint64_t e) {
        const int i = n % (SU - KWD);
        if (n >= SU - KWD && i == 0) {
          to = dst + (uint64_t)place(bin_home(table_key(key), R)) * SU;
          KOps<KT>::store(to, t);
          for (int z = KWD; z < SU; ++z) to[z] = 0;
        }
        if (to) to[KWD + i] = e;
        ++n;
      });
    }
  __syncthreads();
  for (uint32_t pos = tid; pos < R; pos += nt) {
    if (taken[pos >> 5] >> (pos & 31) & 1u) continue;
    #pragma unroll
    for (int i = 0; i < SU; i += 2)
      reinterpret_cast<ulonglong2 *>(dst + (uint64_t)pos * SU)[i / 2] =
          make_ulonglong2(i < KWD ? KEY_EMPTY : 0ull, i + 1 < KWD ? KEY_EMPTY : 0ull);
  }
}

/* the slots of every sample's share of the table past the ones its regions took, for calls that
 * scan a batch's table (used: per sample, the slots taken) */
__global__ void k_sk_fill_gaps(uint64_t *table, const SGeom *sg, const uint64_t *cap, uint32_t S) {
  for (uint32_t q = blockIdx.y; q < S; q += gridDim.y) {
    const uint64_t lo = (sg[q].g.base + sg[q].g.nslots) * 4, hi = (sg[q].g.base + cap[q]) * 4;
    for (uint64_t i = lo + (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < hi; i += (uint64_t)gridDim.x * blockDim.x)
      table[i] = (i & 3) == 0 ? KEY_EMPTY : 0ull;
  }
}
