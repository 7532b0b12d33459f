// mic_bin_sort.cu -- K1: cell location (findMarkerCells, markers.c:41-106) and the stable
// counting sort that orders the device marker columns by cell.
//
// Cell location uses integer compares on the IEEE bit patterns of X, Y and the gridlines
// (valid because every compared value is non-negative): the same answer as the reference's
// bisection, with no FP64 instructions on a GPU whose FP64 rate is 1/60 of FP32.
//
// Sorting: key = 4*(cellY*NCX + cellX) + 2*qy + qx, where (qx, qy) is the marker's quadrant of
// its cell (X >= xc[cellX+1], Y >= yc[cellY+1]: the stagger test of findCellStag2D) and NCX the
// basic cells in x (NX - 1, or NX on a grid periodic in x: markers.c:49, 73); out-of-domain
// markers get key 4*NCX*(NY-1).  Cells stay contiguous and inside a cell the markers
// of each quadrant are contiguous, so every staggered (cell-centre) cell's markers are four
// runs.  An LSD radix sort with 8-bit digits (stable by construction) orders (key, index) pairs.
// The digit counts of every pass come with the cell location (they do not depend on the order), and
// a pass is one kernel: each block ranks a tile's items per digit in index order (warp match), finds
// what the tiles before it hold of each digit by looking back at their published counts, and writes
// the tile out in digit order.  Ties keep the current device order, so the result equals a CPU
// stable sort of the current order.  cell_start[] brackets each cell's markers.
#include "mic_internal.cuh"

using namespace mic;

namespace {

constexpr int kSortThreads = 256;
constexpr int kRadixBits = 8;
constexpr int kBuckets = 1 << kRadixBits;
constexpr int kMaxPasses = 4;
// Items per thread of a pass: 16 (tiles of 4,096) where that fills the GPU; 4 up to 524,288 markers,
// so that the small sorts spread over more SMs (65,536 markers: 64 tiles instead of 16).
constexpr int kItemsLarge = 16, kItemsSmall = 4;
constexpr int64_t kSmallSort = 1 << 19;
inline int items_for(int64_t n) { return n <= kSmallSort ? kItemsSmall : kItemsLarge; }
inline int64_t tiles_for(int64_t n) {
  const int64_t t = (int64_t)kSortThreads * items_for(n);
  return (n + t - 1) / t;
}
// scratch of one sort (ints): tile tickets of the passes, digit counts of the passes, and per pass
// each tile's published counts
constexpr int kOffTicket = 0, kOffCounts = 32, kOffTiles = kOffCounts + kMaxPasses * kBuckets;
inline int64_t sort_ints(int64_t tiles, int passes) { return kOffTiles + (int64_t)passes * tiles * kBuckets; }
inline int passes_for(int64_t ncells) {  // digits of the largest key, 4 ncells
  int bits = 1;
  while ((1LL << bits) <= 4 * ncells) ++bits;
  return (bits + kRadixBits - 1) / kRadixBits;
}

// Largest i in [0, n-2] with g[i] <= v (markers.c:47-69), on bit patterns.
__device__ __forceinline__ int bisect_bits(const long long *__restrict__ g, int n, long long v) {
  int lo = 0, hi = n - 1;
  while (hi - lo > 1) {
    int mid = (lo + hi) >> 1;
    if (v >= __ldg(g + mid))
      lo = mid;
    else
      hi = mid;
  }
  return lo;
}

// The same index from a hint, the marker's cell before this binning: most markers stay in it or
// move to a neighbour, whose intervals g[h] <= v < g[h+1] (the last index takes every v >= g[n-2])
// are tested first; otherwise, or for a hint out of [0, n-2], the bisection.  The tested interval
// characterises the largest i with g[i] <= v, so the result is the bisection's for any hint.
__device__ __forceinline__ int locate_bits(const long long *__restrict__ g, int n, long long v, int hint) {
  if (hint >= 0 && hint <= n - 2) {
    if (__ldg(g + hint) <= v) {
      if (hint == n - 2 || v < __ldg(g + hint + 1)) return hint;
      // v >= g[hint + 1]
      if (hint + 1 == n - 2 || v < __ldg(g + hint + 2)) return hint + 1;
    } else if (hint >= 1 && __ldg(g + hint - 1) <= v) {
      return hint - 1;  // g[hint - 1] <= v < g[hint]
    }
  }
  return bisect_bits(g, n, v);
}

// digit counts of a warp's keys into shared memory; neighbouring markers share their high digits,
// so a warp of one digit adds once
__device__ __forceinline__ void count_digits(int (*h)[kBuckets], int passes, bool valid, int k) {
  const unsigned in = __ballot_sync(0xffffffffu, valid);
  if (in == 0) return;
  for (int p = 0; p < passes; ++p) {
    const int d = (k >> (p * kRadixBits)) & (kBuckets - 1);
    const int d0 = __shfl_sync(0xffffffffu, d, __ffs(in) - 1);
    if (__all_sync(0xffffffffu, !valid || d == d0)) {
      if ((threadIdx.x & 31) == 0) atomicAdd(&h[p][d0], __popc(in));
    } else if (valid) {
      atomicAdd(&h[p][d], 1);
    }
  }
}
__device__ __forceinline__ void clear_digits(int (*h)[kBuckets], int passes) {
  for (int b = threadIdx.x; b < passes * kBuckets; b += blockDim.x) (&h[0][0])[b] = 0;
}
__device__ __forceinline__ void add_digits(int (*h)[kBuckets], int passes, int *counts) {
  for (int b = threadIdx.x; b < passes * kBuckets; b += blockDim.x)
    if ((&h[0][0])[b]) atomicAdd(counts + b, (&h[0][0])[b]);
}

// (a grid of a few blocks per SM walks the markers, so that few digit counts are added in memory)
__global__ void k_find_cells(Params P, const double *__restrict__ X, const double *__restrict__ Y,
                             int *__restrict__ cellX, int *__restrict__ cellY, int *__restrict__ cpu,
                             int *__restrict__ key, int64_t n, int passes, int *counts, Status *st) {
  if (!after_previous()) return;
  __shared__ unsigned long long s_out;
  __shared__ int h[kMaxPasses][kBuckets];
  if (threadIdx.x == 0) s_out = 0;
  clear_digits(h, passes);
  __syncthreads();
  for (int64_t base = blockIdx.x * (int64_t)blockDim.x; base < n; base += (int64_t)gridDim.x * blockDim.x) {
    const int64_t m = base + threadIdx.x;
    int k = 0;
    if (m < n) {
      const long long bx = dbits(X[m]);
      const long long by = dbits(Y[m]);
      const long long ux = (bx == (long long)0x8000000000000000ULL) ? 0LL : bx;
      const long long uy = (by == (long long)0x8000000000000000ULL) ? 0LL : by;
      const long long blx = dbits(P.LX), bly = dbits(P.LY);
      // X >= 0 && Y >= 0 && X <= LX && Y <= LY; NaN fails every test
      const bool in = ux >= 0 && uy >= 0 && ux <= blx && uy <= bly;
      const int hx = cellX[m], hy = cellY[m];  // the cell before this binning (any value)
      int cx = -1, cy = -1;
      k = 4 * P.NCX * (P.NY - 1);
      if (in) {
        cx = locate_bits(P.xbits, P.NCX + 1, ux, hx);  // lines 0..NCX (periodic: line NX = LX)
        cy = locate_bits(P.ybits, P.NY, uy, hy);
        const int qx = ux >= nonneg_bits(P.xc[cx + 1]), qy = uy >= nonneg_bits(P.yc[cy + 1]);
        k = 4 * (cy * P.NCX + cx) + 2 * qy + qx;
      } else {
        atomicAdd(&s_out, 1ULL);
      }
      cellX[m] = cx;
      cellY[m] = cy;
      cpu[m] = 0;
      key[m] = k;
    }
    count_digits(h, passes, m < n, k);
  }
  __syncthreads();
  add_digits(h, passes, counts);
  if (threadIdx.x == 0 && s_out) atomicAdd(&st->n_out, s_out);
}

// In-place exclusive scan of an int array of length len, in blocks of 2048; block totals go
// to aux[] and are scanned by the same routine recursively from the host.
constexpr int kScanThreads = 256;
constexpr int kScanPer = 8;
constexpr int kScanBlock = kScanThreads * kScanPer;

__global__ void k_scan_block(int *__restrict__ data, int64_t len, int *__restrict__ block_sums) {
  __shared__ int warp_tot[kScanThreads / 32];
  const int64_t base = (int64_t)blockIdx.x * kScanBlock + (int64_t)threadIdx.x * kScanPer;
  int v[kScanPer];
  int sum = 0;
#pragma unroll
  for (int k = 0; k < kScanPer; ++k) {
    v[k] = (base + k < len) ? data[base + k] : 0;
    sum += v[k];
  }
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  int incl = sum;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    int t = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane >= o) incl += t;
  }
  if (lane == 31) warp_tot[warp] = incl;
  __syncthreads();
  if (warp == 0) {
    int w = (lane < kScanThreads / 32) ? warp_tot[lane] : 0;
    int wi = w;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      int t = __shfl_up_sync(0xffffffffu, wi, o);
      if (lane >= o) wi += t;
    }
    if (lane < kScanThreads / 32) warp_tot[lane] = wi - w;
    if (lane == kScanThreads / 32 - 1 && block_sums) block_sums[blockIdx.x] = wi;
  }
  __syncthreads();
  int run = warp_tot[warp] + incl - sum;
#pragma unroll
  for (int k = 0; k < kScanPer; ++k) {
    if (base + k < len) data[base + k] = run;
    run += v[k];
  }
}

__global__ void k_scan_add(int *__restrict__ data, int64_t len, const int *__restrict__ block_offsets) {
  const int64_t base = (int64_t)blockIdx.x * kScanBlock;
  const int add = block_offsets[blockIdx.x];
  for (int k = threadIdx.x; k < kScanBlock; k += blockDim.x)
    if (base + k < len) data[base + k] += add;
}

// One pass of the sort.  Tiles are taken in order from a ticket, so the tiles a block waits for are
// running or done.  A tile publishes per digit its own count, then (after looking back) the count of
// all tiles up to it; a later tile adds counts backwards until it meets one of the latter, eight
// tiles' words in flight at a time.  The wait is bounded (limit: rounds that find nothing new): a
// block that gives up leaves its items where they are, adds to *lost, and sets
// *flag, a word in the host's memory that stays set until the markers are uploaded or reset; every
// call that waits for the device reads it there and returns MIC_ERR_CELL.  What the pass then leaves
// is no order, so k_cell_start puts the identity in its place: the markers stay as they were.
// Bound by the ranking (a chain of warp matches and shared-memory counts: half the issue slots, 15%
// of HBM's rate); matching by eight ballots instead took 159 against 129 us, eight items a thread
// 150.  The five launches of a pass (digit counts, three of their scan, scatter) became one: 16.8 M
// markers 224 -> 129 us a pass, 65,536 markers 42 -> 10.
constexpr unsigned kHas = 1u << 30, kUpTo = 2u << 30, kCount = kHas - 1;  // (2^30 markers of 440 B fit no GPU)

template <int IT>
__global__ void __launch_bounds__(kSortThreads, 3) k_radix_pass(const int *__restrict__ key_in, const int *__restrict__ val_in,
                                                            int use_iota, int *__restrict__ key_out,
                                                            int *__restrict__ val_out, int64_t n, int shift,
                                                            const int *__restrict__ counts, unsigned *tiles, int *ticket,
                                                            int limit, unsigned long long *lost, int *flag) {
  if (!after_previous()) return;
  constexpr int W = kSortThreads / 32, T = kSortThreads * IT;
  __shared__ int wcnt[W][kBuckets];        // per warp and digit: count, then offset in the tile's digit
  __shared__ int s_key[T], s_val[T];       // the tile in digit order
  __shared__ int local[kBuckets], at[kBuckets];  // digit's first item in the tile; its place in the output
  __shared__ int wsum[2][W];
  __shared__ int s_tile, s_lost;
  const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
  if (t == 0) {
    s_tile = atomicAdd(ticket, 1);
    s_lost = 0;
  }
#pragma unroll
  for (int w = 0; w < W; ++w) wcnt[w][t] = 0;
  __syncthreads();
  const int tile = s_tile;
  const int64_t first = (int64_t)tile * T, base = first + warp * (32 * IT) + lane;
  int k[IT], v[IT], rank[IT];
#pragma unroll
  for (int r = 0; r < IT; ++r) {
    const int64_t i = base + r * 32;
    k[r] = i < n ? key_in[i] : 0;
    v[r] = i < n ? (use_iota ? (int)i : val_in[i]) : 0;
  }
  const unsigned before = (1u << lane) - 1u;
#pragma unroll
  for (int r = 0; r < IT; ++r) {
    const bool valid = base + r * 32 < n;
    const int d = valid ? (k[r] >> shift) & (kBuckets - 1) : kBuckets;  // invalid: a group of their own
    const unsigned peers = __match_any_sync(0xffffffffu, d);
    const int c = valid ? wcnt[warp][d] : 0, mine = __popc(peers & before);
    rank[r] = c + mine;
    __syncwarp();
    if (valid && mine == 0) wcnt[warp][d] = c + __popc(peers);
    __syncwarp();
  }
  __syncthreads();
  // thread t: digit t
  int count = 0;
#pragma unroll
  for (int w = 0; w < W; ++w) {
    const int c = wcnt[w][t];
    wcnt[w][t] = count;
    count += c;
  }
  volatile unsigned *slot = tiles + t;
  slot[(int64_t)tile * kBuckets] = (tile == 0 ? kUpTo : kHas) | (unsigned)count;
  // first places: of the digit among all markers, and in the tile
  int a = counts[t], b = count;
  const int a0 = a, b0 = b;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int x = __shfl_up_sync(0xffffffffu, a, o), y = __shfl_up_sync(0xffffffffu, b, o);
    if (lane >= o) {
      a += x;
      b += y;
    }
  }
  if (lane == 31) {
    wsum[0][warp] = a;
    wsum[1][warp] = b;
  }
  __syncthreads();
  a -= a0;
  b -= b0;
#pragma unroll
  for (int w = 0; w < W; ++w)
    if (w < warp) {
      a += wsum[0][w];
      b += wsum[1][w];
    }
  int run = 0;
  if (tile > 0) {
    constexpr int LB = 8;
    int p = tile - 1, rounds = 0;
    bool done = false;
    while (!done) {
      if (rounds >= limit) {
        s_lost = 1;
        break;
      }
      unsigned w[LB];
#pragma unroll
      for (int i = 0; i < LB; ++i) w[i] = p - i >= 0 ? (unsigned)slot[(int64_t)(p - i) * kBuckets] : (2u << 30);
      int moved = 0;
      bool open = true;
#pragma unroll
      for (int i = 0; i < LB; ++i) {
        if (open && !done && (w[i] & ~kCount)) {
          run += (int)(w[i] & kCount);
          ++moved;
          done = (w[i] & kUpTo) != 0;
        } else {
          open = false;
        }
      }
      p -= moved;
      rounds += moved == 0;
    }
    slot[(int64_t)tile * kBuckets] = kUpTo | (unsigned)(run + count);
  }
  local[t] = b;
  at[t] = a + run - b;
  __syncthreads();
  const int items = (int)min((int64_t)T, n - first);
  if (s_lost) {  // (a later tile's counts are wrong too; its places are bounded below)
    if (t == 0) {
      atomicAdd(lost, (unsigned long long)items);
      if (flag) *static_cast<volatile int *>(flag) = 1;
    }
    for (int i = t; i < items; i += kSortThreads) {
      key_out[first + i] = key_in[first + i];
      val_out[first + i] = use_iota ? (int)(first + i) : val_in[first + i];
    }
    return;
  }
#pragma unroll
  for (int r = 0; r < IT; ++r) {
    if (base + r * 32 < n) {
      const int d = (k[r] >> shift) & (kBuckets - 1);
      const int q = local[d] + wcnt[warp][d] + rank[r];
      s_key[q] = k[r];
      s_val[q] = v[r];
    }
  }
  __syncthreads();
#pragma unroll
  for (int r = 0; r < IT; ++r) {
    const int i = t + r * kSortThreads;
    if (i < items) {
      const int key = s_key[i];
      const int64_t q = (int64_t)at[(key >> shift) & (kBuckets - 1)] + i;
      if (q >= 0 && q < n) {
        key_out[q] = key;
        val_out[q] = s_val[i];
      }
    }
  }
}

// the passes of one sort on stream s; *kin / *vin: where the sorted keys and indices end up.  A
// launch is counted and timed through ctx when it is given.
void radix_launch(mic_ctx *ctx, cudaStream_t s, int **kin, int **kout, int **vin, int **vout, int64_t n, int passes,
                  int *scratch, int limit, unsigned long long *lost, int *flag) {
  const int64_t tiles = tiles_for(n);
  for (int p = 0; p < passes; ++p) {
    unsigned *words = reinterpret_cast<unsigned *>(scratch + kOffTiles + (int64_t)p * tiles * kBuckets);
    const int *counts = scratch + kOffCounts + p * kBuckets;
    if (ctx) mic_prof_begin(ctx, "k_radix_pass", s);
    if (items_for(n) == kItemsSmall)
      launch_after(k_radix_pass<kItemsSmall>, (unsigned)tiles, kSortThreads, 0, s, *kin, *vin, p == 0, *kout, *vout,
                   n, p * kRadixBits, counts, words, scratch + kOffTicket + p, limit, lost, flag);
    else
      launch_after(k_radix_pass<kItemsLarge>, (unsigned)tiles, kSortThreads, 0, s, *kin, *vin, p == 0, *kout, *vout,
                   n, p * kRadixBits, counts, words, scratch + kOffTicket + p, limit, lost, flag);
    if (ctx) mic_prof_end(ctx, s);
    int *x = *kin;
    *kin = *kout;
    *kout = x;
    x = *vin;
    *vin = *vout;
    *vout = x;
  }
}

// From the sorted (cell, quadrant) keys: qs[q] = first sorted position with key >= q for
// q in [0, 4*ncells+4] (when qs is given) and cs[c] = qs[4c] for c in [0, ncells+1].  After a sort
// that gave up: the identity as the order, no marker in any cell, and *lost all markers.
__global__ void k_cell_start(const int *__restrict__ skey, int64_t n, int ncells, int *__restrict__ cs,
                             int *__restrict__ qs, unsigned long long *lost, int *perm) {
  if (!after_previous()) return;
  // one thread per (cell, quadrant) key q in [0, 4 ncells + 4]: the run of key q starts at the
  // first sorted position whose key is >= q (n when there is none), so empty stretches of cells
  // cost nothing extra.  cs[c] = qs[4c].  The search starts at the position q would have with
  // markers spread evenly over the keys and gallops outwards (steps 1, 2, 4, ...) until it
  // brackets the answer, then bisects the bracket: a few loads, near those of the neighbouring
  // threads, where a bisection of the whole array takes log2 n.  Invariant of the final
  // bisection: every position below lo holds a key < q, and hi is n or holds a key >= q.
  const int64_t q = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  const int64_t qmax = 4LL * ncells + 4;
  if (q > qmax) return;
  int64_t lo = 0, hi = n;
  const unsigned long long gave_up = *lost;  // (used at the end: the search ends whatever the keys are)
  if (n > 0) {
    const int64_t g = q * n / (qmax + 1);  // in [0, n)
    if (skey[g] < q) {
      lo = g + 1;
      for (int64_t step = 1;; step <<= 1) {
        const int64_t p = g + step;
        if (p >= n) break;  // hi stays n
        if (skey[p] >= q) {
          hi = p;
          break;
        }
        lo = p + 1;
      }
    } else {
      hi = g;
      for (int64_t step = 1;; step <<= 1) {
        const int64_t p = g - step;
        if (p < 0) break;  // lo stays 0
        if (skey[p] < q) {
          lo = p + 1;
          break;
        }
        hi = p;
      }
    }
  }
  while (lo < hi) {
    const int64_t mid = (lo + hi) >> 1;
    if (skey[mid] < q)
      lo = mid + 1;
    else
      hi = mid;
  }
  if (gave_up) {
    if (q == 0) *lost = (unsigned long long)n;
    for (int64_t k = q; k < n; k += qmax + 1) perm[k] = (int)k;
    lo = 0;
  }
  if (qs) qs[q] = (int)lo;
  if ((q & 3) == 0) cs[q >> 2] = (int)lo;
}

struct GatherCols {
  const double *src_f[C_F64_COUNT];
  double *dst_f[C_F64_COUNT];
  const int *src_i[C_I32_COUNT];
  int *dst_i[C_I32_COUNT];
  int nf;  // double columns moved: the device-only grain column only once grain sizes were set
};

// The gather of every column into the sorted order.  GEO: also the projection geometry of each
// marker, from the position and cell just gathered: this kernel is bound by HBM and the
// geometry by the FP64 pipe, so together they cost little more than the gather alone.
// Every load comes before the first store.  The compiler cannot tell the column buffers apart,
// so a load written after a store could not issue before it: interleaved, each thread would
// wait out one memory latency per column (30 in a row) and the gather would be bound by latency.
// The geometry's grid-line loads come before the stores for the same reason.
template <bool GEO>
__global__ void k_reorder(GatherCols g, const int *__restrict__ perm, int64_t n, Params P, GeoOut go) {
  if (!after_previous()) return;
  const int64_t k = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (k >= n) return;
  const int p = perm[k];
  double vf[C_F64_COUNT];
  int vi[C_I32_COUNT];
#pragma unroll
  for (int c = 0; c < C_F64_COUNT; ++c) vf[c] = (c < g.nf) ? __ldg(g.src_f[c] + p) : 0.0;
#pragma unroll
  for (int c = 0; c < C_I32_COUNT; ++c) vi[c] = __ldg(g.src_i[c] + p);
  if (GEO) geometry_marker(P, vf[C_X], vf[C_Y], vi[C_CELLX], vi[C_CELLY], go, k);
#pragma unroll
  for (int c = 0; c < C_F64_COUNT; ++c)
    if (c < g.nf) g.dst_f[c][k] = vf[c];
#pragma unroll
  for (int c = 0; c < C_I32_COUNT; ++c) g.dst_i[c][k] = vi[c];
}

// perm[k] = device slot of caller marker k (k < n); slots from n on stay in place
__global__ void k_restore_perm(const int *__restrict__ id, int64_t n, int64_t cap, int *__restrict__ perm) {
  const int64_t s = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (s >= cap) return;
  if (s < n)
    perm[id[s]] = (int)s;
  else
    perm[s] = (int)s;
}

// aux: free space for the block totals of this level and all coarser levels
int scan_exclusive(mic_ctx *ctx, int *data, int64_t len, int *aux) {
  const int64_t nb = (len + kScanBlock - 1) / kScanBlock;
  if (nb <= 1) {
    {
      MIC_KERNEL(ctx, "k_scan_block");
      k_scan_block<<<1, kScanThreads, 0, ctx->stream>>>(data, len, nullptr);
    }
    return cudaGetLastError() == cudaSuccess ? MIC_OK : MIC_ERR_CUDA;
  }
  int *sums = aux;
  {
    MIC_KERNEL(ctx, "k_scan_block");
    k_scan_block<<<(unsigned)nb, kScanThreads, 0, ctx->stream>>>(data, len, sums);
  }
  int e = scan_exclusive(ctx, sums, nb, aux + nb + 1);
  if (e) return e;
  {
    MIC_KERNEL(ctx, "k_scan_add");
    k_scan_add<<<(unsigned)nb, kScanThreads, 0, ctx->stream>>>(data, len, sums);
  }
  return cudaGetLastError() == cudaSuccess ? MIC_OK : MIC_ERR_CUDA;
}

int ensure_sort_scratch(mic_ctx *ctx, int64_t need) {
  if (ctx->sort_cap >= need) return MIC_OK;
  cudaFree(ctx->sort_buf);
  ctx->sort_buf = nullptr;
  ctx->sort_cap = 0;
  if (cudaMalloc((void **)&ctx->sort_buf, sizeof(int) * need) != cudaSuccess) return MIC_ERR_NOMEM;
  ctx->sort_cap = need;
  return MIC_OK;
}

}  // namespace

// Bins every marker, sorts the columns by cell (stable) and rebuilds cell_start.
int mic_bin_and_sort(mic_ctx *ctx, int64_t *n_out, bool step) {
  const int64_t n = ctx->n;
  const int passes = passes_for(ctx->ncells);
  const int64_t ints = n > 0 ? sort_ints(tiles_for(n), passes) : 0;
  int e = n > 0 ? ensure_sort_scratch(ctx, ints) : MIC_OK;
  if (e) return e;
  mic_clear_list clear;
  clear.add(&ctx->d_status->n_out, 2 * sizeof(unsigned long long));  // and bad_cell
  if (n > 0) clear.add(ctx->sort_buf, sizeof(int) * ints);
  if (step) mic_clear_yield(ctx, clear, true);
  if ((e = mic_clear(ctx, clear))) return e;
  if (n == 0) {
    MIC_CUDA_TRY(cudaMemsetAsync(ctx->cell_start, 0, sizeof(int) * ((size_t)ctx->ncells + 2), ctx->stream));
    MIC_CUDA_TRY(cudaMemsetAsync(ctx->quad_start, 0, sizeof(int) * (4 * (size_t)ctx->ncells + 5), ctx->stream));
    ctx->sorted = 1;
    ctx->wn_valid = 0;
    if (n_out) *n_out = 0;
    return MIC_OK;
  }
  {
    MIC_KERNEL(ctx, "k_find_cells");
    const int block = tuned_block(ctx, TU_FIND_CELLS);
    const unsigned full = grid_for(n, block), most = 2048 / block * sm_count(ctx);
    launch_after(k_find_cells, full < most ? full : most, block, 0, ctx->stream, ctx->P, ctx->f64[C_X], ctx->f64[C_Y],
                 ctx->i32[C_CELLX], ctx->i32[C_CELLY], ctx->i32[C_CPU], ctx->key, n, passes,
                 ctx->sort_buf + kOffCounts, ctx->d_status);
  }
  MIC_CUDA_TRY(cudaGetLastError());
  int *kin = ctx->key, *kout = ctx->key_alt, *vin = ctx->perm, *vout = ctx->perm_alt;
  radix_launch(ctx, ctx->stream, &kin, &kout, &vin, &vout, n, passes, ctx->sort_buf, ctx->sort_limit,
               &ctx->d_status->bad_cell, ctx->h_lost);
  MIC_CUDA_TRY(cudaGetLastError());
  // kin / vin now hold the sorted keys and the permutation
  {
    MIC_KERNEL(ctx, "k_cell_start");
    launch_after(k_cell_start, grid_for(4LL * ctx->ncells + 5), kBlock, 0, ctx->stream, kin, n, ctx->ncells,
                 ctx->cell_start, ctx->quad_start, &ctx->d_status->bad_cell, vin);
  }
  MIC_CUDA_TRY(cudaGetLastError());
  GatherCols g;
  g.nf = ctx->has_grain ? C_F64_COUNT : C_AOS_F64;
  for (int c = 0; c < C_F64_COUNT; ++c) {
    g.src_f[c] = ctx->f64[c];
    g.dst_f[c] = ctx->f64_alt[c];
  }
  for (int c = 0; c < C_I32_COUNT; ++c) {
    g.src_i[c] = ctx->i32[c];
    g.dst_i[c] = ctx->i32_alt[c];
  }
  {
    MIC_KERNEL(ctx, "k_reorder");
    launch_after(k_reorder<true>, grid_for(n, tuned_block(ctx, TU_REORDER)), tuned_block(ctx, TU_REORDER), 0,
                 ctx->stream, g, vin, n, ctx->P, geo_out(ctx));
  }
  MIC_CUDA_TRY(cudaGetLastError());
  for (int c = 0; c < g.nf; ++c) {
    double *t = ctx->f64[c];
    ctx->f64[c] = ctx->f64_alt[c];
    ctx->f64_alt[c] = t;
  }
  for (int c = 0; c < C_I32_COUNT; ++c) {
    int *t = ctx->i32[c];
    ctx->i32[c] = ctx->i32_alt[c];
    ctx->i32_alt[c] = t;
  }
  ctx->sorted = 1;
  ctx->geo_valid = 1;  // computed by the gather
  ctx->wn_valid = 0;
  if (n_out) {
    e = mic_fetch_status(ctx);
    *n_out = (int64_t)ctx->h_status->n_out;
    if (e) return e;
  }
  return MIC_OK;
}

// exclusive prefix sum of data[0, len) in place; aux: mic_scan_aux_ints(len) ints of scratch
int mic_scan_exclusive(mic_ctx *ctx, int *data, int64_t len, int *aux) { return scan_exclusive(ctx, data, len, aux); }

int64_t mic_scan_aux_ints(int64_t len) {
  int64_t aux = 0, l = len;
  while (l > 1) {
    l = (l + kScanBlock - 1) / kScanBlock;
    aux += l + 1;
  }
  return aux + 16;
}

// Columns [0, n) back to the caller's marker order (slot k holds caller marker k); slots
// [n, cap) keep their contents.  The next pass bins and sorts again.
int mic_restore_caller_order(mic_ctx *ctx) {
  const int64_t cap = ctx->cap;
  if (cap == 0) return MIC_OK;
  {
    MIC_KERNEL(ctx, "k_restore_perm");
    k_restore_perm<<<grid_for(cap), kBlock, 0, ctx->stream>>>(ctx->i32[C_ID], ctx->n, cap, ctx->perm);
  }
  GatherCols g;
  g.nf = ctx->has_grain ? C_F64_COUNT : C_AOS_F64;
  for (int c = 0; c < C_F64_COUNT; ++c) {
    g.src_f[c] = ctx->f64[c];
    g.dst_f[c] = ctx->f64_alt[c];
  }
  for (int c = 0; c < C_I32_COUNT; ++c) {
    g.src_i[c] = ctx->i32[c];
    g.dst_i[c] = ctx->i32_alt[c];
  }
  {
    MIC_KERNEL(ctx, "k_reorder");
    launch_after(k_reorder<false>, grid_for(cap), kBlock, 0, ctx->stream, g, ctx->perm, cap, ctx->P, GeoOut{});
  }
  MIC_CUDA_TRY(cudaGetLastError());
  for (int c = 0; c < g.nf; ++c) {
    double *t = ctx->f64[c];
    ctx->f64[c] = ctx->f64_alt[c];
    ctx->f64_alt[c] = t;
  }
  for (int c = 0; c < C_I32_COUNT; ++c) {
    int *t = ctx->i32[c];
    ctx->i32[c] = ctx->i32_alt[c];
    ctx->i32_alt[c] = t;
  }
  mic_invalidate_sort(ctx);
  return MIC_OK;
}

int mic_ensure_sorted(mic_ctx *ctx) {
  if (ctx->sorted) return MIC_OK;
  return mic_bin_and_sort(ctx, nullptr);
}

extern "C" int mic_find_marker_cells(mic_ctx *ctx, int64_t *n_out) {
  if (!ctx) return MIC_ERR_ARG;
  cudaSetDevice(ctx->device);
  int64_t no = 0;
  int e = mic_bin_and_sort(ctx, &no);
  if (n_out) *n_out = no;
  return e;
}

// ---- binning and stable sort for callers that cannot allocate ------------------------
//
// Some callers of this code cannot call cudaMalloc: a host that has finished its
// start-up and forbids device allocation afterwards (fixed-memory production runs),
// code that runs between the capture calls of a stream it does not own, or a plug-in
// whose host application owns the allocator.  mic_bin_sort_noalloc serves them: the
// caller passes device pointers for its inputs and outputs, and the sort's scratch (keys,
// the second value buffer, the digit histograms and the scan's block totals) lives in the
// file-scope device array below, reserved once when the library loads on a device and
// held until the process exits.  Every call shares that array, so calls whose work
// overlaps on the GPU (different streams, or different host threads on one device) race
// and must be ordered by the caller.

#include <mutex>

namespace {

constexpr int64_t kNoallocMaxMarkers = MIC_NOALLOC_MAX_MARKERS;
constexpr int64_t kNoallocMaxCells = MIC_NOALLOC_MAX_CELLS;
// the sort's own scratch at the largest tile count: tiles of the small sort up to kSmallSort
// markers, of the large one beyond; the largest key has three digits
constexpr int64_t kNoallocTiles = kSmallSort / (kSortThreads * kItemsSmall);
static_assert(kNoallocTiles >= kNoallocMaxMarkers / (kSortThreads * kItemsLarge), "tiles of the largest sort");
constexpr int kNoallocPasses = 3;
static_assert(4 * kNoallocMaxCells < (1LL << (kNoallocPasses * kRadixBits)), "digits of the largest key");
constexpr int64_t kNoallocSort = kOffTiles + kNoallocPasses * kNoallocTiles * kBuckets;
// layout (in 4-byte words): key | key_alt | val_alt | sort, then two 8-byte counters
constexpr int64_t kOffKey = 0;
constexpr int64_t kOffKeyAlt = kOffKey + kNoallocMaxMarkers;
constexpr int64_t kOffValAlt = kOffKeyAlt + kNoallocMaxMarkers;
constexpr int64_t kOffSort = kOffValAlt + kNoallocMaxMarkers;
constexpr int64_t kWords = (kOffSort + kNoallocSort + 63) / 64 * 64;
constexpr size_t kNoallocBytes = (size_t)kWords * 4 + 256;

static __device__ __align__(256) unsigned char g_noalloc_scratch[kNoallocBytes];

// host-side: device address of g_noalloc_scratch per CUDA context (the symbol itself is only a
// host stand-in and must never be handed to a kernel).  The cache is keyed on the context's
// process-unique id, not on the device ordinal: after cudaDeviceReset, or under another context
// of the same device, the address is looked up again instead of reusing a stale one.
std::mutex g_noalloc_mu;
constexpr int kNoallocCache = 64;
unsigned long long g_noalloc_ctx[kNoallocCache];  // context ids (0 = empty slot)
unsigned char *g_noalloc_ptr[kNoallocCache];
int g_noalloc_next;  // next slot to fill (round robin once all are used)

// the current context's id through the driver entry points (no link against libcuda); 0 when
// they are unavailable, and then the address is looked up on every call
typedef int (*CtxGetCurrentFn)(void **);
typedef int (*CtxGetIdFn)(void *, unsigned long long *);
unsigned long long current_context_id() {
  static CtxGetCurrentFn get_current = nullptr;
  static CtxGetIdFn get_id = nullptr;
  static std::once_flag once;
  std::call_once(once, [] {
    void *f = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPointByVersion("cuCtxGetCurrent", &f, 12000, cudaEnableDefault, &q) == cudaSuccess &&
        q == cudaDriverEntryPointSuccess)
      get_current = (CtxGetCurrentFn)f;
    f = nullptr;
    if (cudaGetDriverEntryPointByVersion("cuCtxGetId", &f, 12000, cudaEnableDefault, &q) == cudaSuccess &&
        q == cudaDriverEntryPointSuccess)
      get_id = (CtxGetIdFn)f;
    cudaGetLastError();
  });
  void *ctx = nullptr;
  unsigned long long id = 0;
  if (!get_current || !get_id || get_current(&ctx) != 0 || !ctx || get_id(ctx, &id) != 0) return 0;
  return id;
}

__global__ void k_find_cells_grid(const double *__restrict__ X, const double *__restrict__ Y,
                                  const double *__restrict__ xg, const double *__restrict__ yg, int NX, int NY,
                                  double LX, double LY, int *__restrict__ cellX, int *__restrict__ cellY,
                                  int *__restrict__ key, int64_t n, int passes, int *counts,
                                  unsigned long long *n_out) {
  __shared__ unsigned long long s_out;
  __shared__ int h[kMaxPasses][kBuckets];
  if (threadIdx.x == 0) s_out = 0;
  clear_digits(h, passes);
  __syncthreads();
  const int64_t m = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  int k = 0;
  if (m < n) {
    const long long ux = nonneg_bits(X[m]), uy = nonneg_bits(Y[m]);
    const bool in = ux >= 0 && uy >= 0 && ux <= dbits(LX) && uy <= dbits(LY);
    int cx = -1, cy = -1;
    k = 4 * (NX - 1) * (NY - 1);
    if (in) {
      int lo = 0, hi = NX - 1;
      while (hi - lo > 1) {
        const int mid = (lo + hi) >> 1;
        if (ux >= nonneg_bits(xg[mid])) lo = mid; else hi = mid;
      }
      cx = lo;
      lo = 0;
      hi = NY - 1;
      while (hi - lo > 1) {
        const int mid = (lo + hi) >> 1;
        if (uy >= nonneg_bits(yg[mid])) lo = mid; else hi = mid;
      }
      cy = lo;
      // quadrant of the cell: the same test as the context binning (cell centres from x, y)
      const int qx = ux >= nonneg_bits((xg[cx] + xg[cx + 1]) / 2.0);
      const int qy = uy >= nonneg_bits((yg[cy] + yg[cy + 1]) / 2.0);
      k = 4 * (cy * (NX - 1) + cx) + 2 * qy + qx;
    } else {
      atomicAdd(&s_out, 1ULL);
    }
    cellX[m] = cx;
    cellY[m] = cy;
    key[m] = k;
  }
  count_digits(h, passes, m < n, k);
  __syncthreads();
  add_digits(h, passes, counts);
  if (threadIdx.x == 0 && s_out) atomicAdd(n_out, s_out);
}

// Device address of the scratch array in the current context.  The first call in a context
// (on each device, with that device current) looks it up with cudaGetSymbolAddress, which also
// makes the runtime set the context up; later calls in the same context reuse it.
int noalloc_scratch(unsigned char **out) {
  std::lock_guard<std::mutex> lock(g_noalloc_mu);
  const unsigned long long id = current_context_id();
  if (id)
    for (int k = 0; k < kNoallocCache; ++k)
      if (g_noalloc_ctx[k] == id) {
        *out = g_noalloc_ptr[k];
        return MIC_OK;
      }
  unsigned char *p = nullptr;
  if (cudaGetSymbolAddress((void **)&p, g_noalloc_scratch) != cudaSuccess || !p) {
    cudaGetLastError();
    return MIC_ERR_CUDA;
  }
  // the lookup may have created the context: take its id now
  const unsigned long long id2 = id ? id : current_context_id();
  if (id2) {
    g_noalloc_ctx[g_noalloc_next] = id2;
    g_noalloc_ptr[g_noalloc_next] = p;
    g_noalloc_next = (g_noalloc_next + 1) % kNoallocCache;
  }
  *out = p;
  return MIC_OK;
}

}  // namespace

extern "C" int mic_bin_sort_noalloc(const double *X, const double *Y, int64_t n, const double *x, const double *y,
                                    int NX, int NY, double LX, double LY, int32_t *cellX, int32_t *cellY,
                                    int32_t *perm, int32_t *cell_start, void *stream, int64_t *n_out) {
  if (n < 0 || NX < 3 || NY < 3 || !x || !y || !cell_start) return MIC_ERR_ARG;
  if (n > 0 && (!X || !Y || !cellX || !cellY || !perm)) return MIC_ERR_ARG;
  if (n > kNoallocMaxMarkers) return MIC_ERR_CAPACITY;
  const int64_t ncells = (int64_t)(NX - 1) * (NY - 1);
  if (ncells > kNoallocMaxCells) return MIC_ERR_CAPACITY;
  int device = 0;
  if (cudaGetDevice(&device) != cudaSuccess) return MIC_ERR_NO_DEVICE;
  unsigned char *base = nullptr;
  int e = noalloc_scratch(&base);
  if (e) return e;
  cudaStream_t s = (cudaStream_t)stream;
  int *words = reinterpret_cast<int *>(base);
  int *key = words + kOffKey, *key_alt = words + kOffKeyAlt, *val_alt = words + kOffValAlt;
  int *sort = words + kOffSort;
  // markers outside the domain, and markers a sort that gave up has not placed
  unsigned long long *d_out = reinterpret_cast<unsigned long long *>(base + (size_t)kWords * 4), *d_lost = d_out + 1;
  // the counters keep the previous call's values: clear them
  if (cudaMemsetAsync(d_out, 0, 2 * sizeof(unsigned long long), s) != cudaSuccess) return MIC_ERR_CUDA;
  if (n > 0) {
    const int passes = passes_for(ncells);
    if (cudaMemsetAsync(sort, 0, sizeof(int) * sort_ints(tiles_for(n), passes), s) != cudaSuccess) return MIC_ERR_CUDA;
    k_find_cells_grid<<<grid_for(n), kBlock, 0, s>>>(X, Y, x, y, NX, NY, LX, LY, cellX, cellY, key, n, passes,
                                                     sort + kOffCounts, d_out);
    if (cudaGetLastError() != cudaSuccess) return MIC_ERR_CUDA;
    // the last pass must write the caller's perm[]: pick the buffers accordingly (the first reads none)
    int *kin = key, *kout = key_alt, *vin = (passes & 1) ? val_alt : perm, *vout = (passes & 1) ? perm : val_alt;
    radix_launch(nullptr, s, &kin, &kout, &vin, &vout, n, passes, sort, kLookRounds, d_lost, nullptr);
    if (cudaGetLastError() != cudaSuccess) return MIC_ERR_CUDA;
    launch_after(k_cell_start, grid_for(4LL * ncells + 5), kBlock, 0, s, kin, n, (int)ncells, cell_start, nullptr,
                 d_lost, vin);
  } else {
    if (cudaMemsetAsync(cell_start, 0, sizeof(int32_t) * (size_t)(ncells + 2), s) != cudaSuccess)
      return MIC_ERR_CUDA;
  }
  if (cudaGetLastError() != cudaSuccess) return MIC_ERR_CUDA;
  if (n_out) {
    unsigned long long h[2] = {0, 0};
    if (cudaMemcpyAsync(h, d_out, sizeof(h), cudaMemcpyDeviceToHost, s) != cudaSuccess) return MIC_ERR_CUDA;
    if (cudaStreamSynchronize(s) != cudaSuccess) return MIC_ERR_CUDA;
    *n_out = (int64_t)h[0];
    if (h[1]) return MIC_ERR_CELL;
  }
  return MIC_OK;
}
