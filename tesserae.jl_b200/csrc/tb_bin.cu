// tb_bin.cu -- particle binning into grid blocks: the device counterpart of
// update!(::GPUBlockStrategy, x) (Tesserae.jl src/Parallel/gpu_block_strategy.jl:142-166),
// producing the block order of the reference CPU strategy bit for bit: block id
// ascending, particle id ascending inside a block (cpu_block_strategy.jl:174-190).
//
//   count    one thread per particle: findblock, warp-aggregated count atomics
//   scan     packed (count | nonempty << 32) 64-bit sums: offsets, cursors, the
//            compacted block list and the totals [nactive, nassigned], and the
//            node blocks the transfer touches; one launch up to 16 tiles of 1024
//            blocks, a tile reduction before it above
//   scatter  a warp takes 4 chunks of 32 ids and reserves one run per (chunk,
//            distinct block) with a single atomic, writing the particles in lane order
//   fixup    one warp per non-empty block: the block's segment is a set of runs,
//            one per scatter chunk, each ascending; the runs are ranked by chunk id
//            and copied in order; blocks of more than 128 runs by the CTA (bitonic
//            in shared memory, or in a global scratch region above 2048 runs)
// The result is deterministic regardless of atomic order.
#include "tb_launch.cuh"

namespace tb {

namespace {

__device__ __forceinline__ unsigned lanemask_lt() {
    unsigned m;
    asm("mov.u32 %0, %%lanemask_lt;" : "=r"(m));
    return m;
}

template <int D, class T>
__global__ void __launch_bounds__(256) bin_count_kernel(DMesh<D, T> M, const T* __restrict__ x0,
                                                        const T* __restrict__ x1, const T* __restrict__ x2,
                                                        long long n, int* __restrict__ blockids,
                                                        int* __restrict__ counts) {
    chain_wait();
    const long long p = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    int b = -1;
    if (p < n) {
        T x[3];
        x[0] = x0[p];
        x[1] = x1[p];
        if constexpr (D == 3) x[2] = x2[p];
        b = findblock<D, T>(M, x);
        blockids[p] = b;
    }
    const unsigned peers = __match_any_sync(0xffffffffu, b);
    const int leader = __ffs(peers) - 1;
    if (b > 0 && int(threadIdx.x & 31) == leader) atomicAdd(&counts[b - 1], __popc(peers));
}

__device__ __forceinline__ unsigned long long pack_count(int c) {
    return (unsigned long long)(unsigned)c | ((unsigned long long)(c != 0) << 32);
}

// Inclusive block scan of one 64-bit value per thread (blockDim = 256).
__device__ __forceinline__ unsigned long long block_incl_scan(unsigned long long v, unsigned long long* warp_tot,
                                                              unsigned long long& total) {
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, nw = blockDim.x >> 5;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        unsigned long long t = __shfl_up_sync(0xffffffffu, v, o);
        if (lane >= o) v += t;
    }
    if (lane == 31) warp_tot[wid] = v;
    __syncthreads();
    if (wid == 0) {
        unsigned long long w = lane < nw ? warp_tot[lane] : 0ull;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            unsigned long long t = __shfl_up_sync(0xffffffffu, w, o);
            if (lane >= o) w += t;
        }
        if (lane < nw) warp_tot[lane] = w;
    }
    __syncthreads();
    total = warp_tot[nw - 1];
    unsigned long long r = v + (wid > 0 ? warp_tot[wid - 1] : 0ull);
    __syncthreads();
    return r;
}

__global__ void __launch_bounds__(256) scan_reduce_kernel(const int* __restrict__ counts, int nb,
                                                          unsigned long long* __restrict__ partials) {
    chain_wait();
    __shared__ unsigned long long wt[8];
    const int base = blockIdx.x * SCAN_TILE + threadIdx.x * 4;
    unsigned long long s = 0;
#pragma unroll
    for (int k = 0; k < 4; ++k)
        if (base + k < nb) s += pack_count(counts[base + k]);
    unsigned long long total;
    block_incl_scan(s, wt, total);
    if (threadIdx.x == 0) partials[blockIdx.x] = total;
}

// Offsets, cursors, the compacted block list and the totals from the counts. A
// CTA sums what lies before its own tile itself: the tile partials
// (scan_reduce_kernel), or, with ONE, the counts (up to SCAN_ONE tiles a CTA reads
// at most 60 counts per thread, which costs less than a second launch; a third
// launch for the prefix of the partials was 2 us of every step).
// With touch.cur it also marks the node blocks that this step's transfer reaches
// (every block within one block per axis of one that holds particles) and lists
// those marked now or in the previous transfer; the order of the list does not
// matter. *touch.count must be zero; *touch.next_count is zeroed for the next
// step, and *bnd_count for this one's P2G.
template <bool ONE>
__global__ void __launch_bounds__(256) scan_kernel(const int* __restrict__ counts, int nb,
                                                   const unsigned long long* __restrict__ partials,
                                                   int* __restrict__ offsets, int* __restrict__ cursors,
                                                   int* __restrict__ blocklist, int* __restrict__ totals,
                                                   unsigned long long* __restrict__ bnd_count, TouchArgs touch) {
    chain_wait();
    __shared__ unsigned long long wt[8];
    const int tile0 = blockIdx.x * SCAN_TILE, base = tile0 + threadIdx.x * 4;
    unsigned long long before = 0;
    if constexpr (ONE) {
        for (int b = threadIdx.x; b < tile0; b += 256) before += pack_count(counts[b]);
    } else {
        for (int t = threadIdx.x; t < int(blockIdx.x); t += 256) before += partials[t];
    }
    unsigned long long prefix;
    block_incl_scan(before, wt, prefix);
    int c[4];
    unsigned long long s = 0;
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        c[k] = (base + k < nb) ? counts[base + k] : 0;
        s += pack_count(c[k]);
    }
    unsigned long long total;
    unsigned long long incl = block_incl_scan(s, wt, total);
    unsigned long long run = prefix + incl - s;  // exclusive prefix of this thread
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        const int b = base + k;
        if (b < nb) {
            const int start = int(run & 0xffffffffull);
            offsets[b] = start;
            cursors[b] = start;
            if (c[k] != 0) blocklist[int(run >> 32)] = b + 1;
            run += pack_count(c[k]);
            if (b == nb - 1) {
                offsets[nb] = int(run & 0xffffffffull);
                totals[0] = int(run >> 32);
                totals[1] = int(run & 0xffffffffull);
            }
        }
    }
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        if (bnd_count) *bnd_count = 0;
        if (touch.next_count) *touch.next_count = 0;
    }
    if (!touch.cur) return;
    const int lane = threadIdx.x & 31;
#pragma unroll 1
    for (int k = 0; k < 4; ++k) {
        const int B = tile0 + k * 256 + threadIdx.x;  // neighbouring threads, neighbouring blocks
        bool t = false;
        if (B < nb) {
            const int bx = B % touch.nb.x, by = (B / touch.nb.x) % touch.nb.y, bz = B / (touch.nb.x * touch.nb.y);
            int any = 0;
            for (int z = max(bz - 1, 0); z <= min(bz + 1, touch.nb.z - 1); ++z)
                for (int y = max(by - 1, 0); y <= min(by + 1, touch.nb.y - 1); ++y) {
                    const int* row = counts + touch.nb.x * (y + touch.nb.y * z);
                    any |= row[bx];
                    if (bx > 0) any |= row[bx - 1];
                    if (bx + 1 < touch.nb.x) any |= row[bx + 1];
                }
            touch.cur[B] = any != 0;
            t = any != 0 || touch.prev[B] != 0;
        }
        const unsigned m = __ballot_sync(0xffffffffu, t);
        int at = 0;
        if (lane == 0 && m) at = atomicAdd(touch.count, __popc(m));
        at = __shfl_sync(0xffffffffu, at, 0);
        if (t) touch.list[at + __popc(m & lanemask_lt())] = B;
    }
}

// Each warp scatters SCAT_IT chunks of 32 consecutive ids: all their block ids
// are loaded, and all their run reservations issued, before any is waited for
// (one round trip each instead of one per chunk). A chunk still reserves one
// run per block, so the runs the fix-up orders are those of one warp per chunk.
constexpr int SCAT_IT = 4;
__global__ void __launch_bounds__(256) bin_scatter_kernel(const int* __restrict__ blockids, long long n,
                                                          int* __restrict__ cursors, int* __restrict__ perm_tmp) {
    chain_wait();
    const unsigned full = 0xffffffffu;
    const int lane = threadIdx.x & 31;
    const long long c0 = (((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5) * (32ll * SCAT_IT);
    int b[SCAT_IT];
#pragma unroll
    for (int u = 0; u < SCAT_IT; ++u) {
        const long long p = c0 + 32 * u + lane;
        b[u] = p < n ? blockids[p] : -1;
    }
    unsigned peers[SCAT_IT];
    int base[SCAT_IT];
#pragma unroll
    for (int u = 0; u < SCAT_IT; ++u) {
        peers[u] = __match_any_sync(full, b[u]);
        base[u] = 0;
        if (b[u] > 0 && lane == __ffs(peers[u]) - 1) base[u] = atomicAdd(&cursors[b[u] - 1], __popc(peers[u]));
    }
#pragma unroll
    for (int u = 0; u < SCAT_IT; ++u) {
        const int bb = __shfl_sync(full, base[u], __ffs(peers[u]) - 1);
        if (b[u] > 0) perm_tmp[bb + __popc(peers[u] & lanemask_lt())] = int(c0 + 32 * u + lane);
    }
}

constexpr int FIX_THREADS = 256;
constexpr int FIX_SMEM_KEYS = 2048;

__device__ __forceinline__ int next_pow2(int v) {
    int k = 1;
    while (k < v) k <<= 1;
    return k;
}

// Exclusive scan of one int per thread over the CTA (blockDim = FIX_THREADS);
// `total` gets the sum. Two barriers; `wsum` holds the warp sums.
__device__ __forceinline__ int fix_excl_scan(int v, int* wsum, int& total) {
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    int incl = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int t = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += t;
    }
    if (lane == 31) wsum[wid] = incl;
    __syncthreads();
    int wprefix = 0;
    total = 0;
#pragma unroll
    for (int q = 0; q < FIX_THREADS / 32; ++q) {
        const int w = wsum[q];
        wprefix += q < wid ? w : 0;
        total += w;
    }
    __syncthreads();
    return wprefix + incl - v;
}

// A block's segment of the scattered ids is a concatenation of runs, one per
// scatter chunk (32 consecutive ids) that held particles of the block, each
// ascending and contiguous, and no two runs of a segment share a chunk id.
//
// By a warp, up to FIXW_RUNS runs: the run heads are found with ballots, the runs
// ranked by chunk id (every run against every run) and the segment copied
// element-parallel, each element to its run's place.
//
// By the CTA, more runs: the keys (chunk id << 32 | run index) are bitonic-sorted,
// the output start of each run is the prefix sum of the run lengths in sorted
// order, and the segment is copied element-parallel, all in shared memory when
// the padded key count fits; above that (more than FIX_SMEM_KEYS runs) the keys
// are sorted in the block's own region [2s, 2s + 2n) of the global scratch
// (next_pow2(k) <= 2n, segments disjoint) and each thread copies whole runs.
constexpr int FIXW_RUNS = 128;
constexpr int FIXW_U = 8;  // chunks of 32 ids loaded together

struct FixShared {
    unsigned long long sbuf[FIX_SMEM_KEYS];
    int hpos[FIX_SMEM_KEYS + 1];  // run starts, segment order
    int hout[FIX_SMEM_KEYS];      // output start of each run, segment order
    int kcount;
    int wsum[FIX_THREADS / 32];
    int over[FIX_THREADS / 32];  // this round's blocks with too many runs (-1: none)
};

// Segment S[s, s + n) to out, by the whole CTA.
__device__ __forceinline__ void fixup_cta(FixShared& sm, const int* __restrict__ S, int s, int n,
                                          int* __restrict__ perm, unsigned long long* __restrict__ gscratch) {
    unsigned long long* sbuf = sm.sbuf;
    int *hpos = sm.hpos, *hout = sm.hout, *wsum = sm.wsum;
    int& kcount = sm.kcount;
    const int tid = threadIdx.x;
    auto is_head = [](const int* seg, int j, int v) { return j == 0 || (seg[j - 1] >> 5) != (v >> 5); };
    const int* seg = S + s;
    int* out = perm + s;
    // Run heads: the first element, and every element whose warp id differs
    // from its predecessor's.
    int myheads = 0;
    for (int j = tid; j < n; j += FIX_THREADS) myheads += is_head(seg, j, seg[j]);
    int k;
    fix_excl_scan(myheads, wsum, k);
    const int K = next_pow2(k);
    if (K <= FIX_SMEM_KEYS) {
        // 1. heads in segment order: positions and keys
        int rbase = 0;
        for (int j0 = 0; j0 < n; j0 += FIX_THREADS) {
            const int j = j0 + tid;
            const int v = j < n ? seg[j] : 0;
            const int h = (j < n && is_head(seg, j, v)) ? 1 : 0;
            int tot;
            const int r = rbase + fix_excl_scan(h, wsum, tot);
            if (h) {
                hpos[r] = j;
                sbuf[r] = ((unsigned long long)(unsigned)(v >> 5) << 32) | (unsigned)r;
            }
            rbase += tot;
        }
        if (tid == 0) hpos[k] = n;
        for (int t = k + tid; t < K; t += FIX_THREADS) sbuf[t] = ~0ull;
        __syncthreads();
        // 2. bitonic sort of the K keys (ascending)
        for (int size = 2; size <= K; size <<= 1) {
            for (int stride = size >> 1; stride > 0; stride >>= 1) {
                for (int i = tid; i < (K >> 1); i += FIX_THREADS) {
                    const int lo = (i / stride) * 2 * stride + (i % stride);
                    const int hi = lo + stride;
                    const bool asc = (lo & size) == 0;
                    const unsigned long long a = sbuf[lo], c = sbuf[hi];
                    if ((a > c) == asc) {
                        sbuf[lo] = c;
                        sbuf[hi] = a;
                    }
                }
                __syncthreads();
            }
        }
        // 3. output start of each run: lengths summed in sorted order
        int obase = 0;
        for (int i0 = 0; i0 < k; i0 += FIX_THREADS) {
            const int i = i0 + tid;
            int r = 0, len = 0;
            if (i < k) {
                r = int(sbuf[i] & 0xffffffffull);
                len = hpos[r + 1] - hpos[r];
            }
            int tot;
            const int st = obase + fix_excl_scan(len, wsum, tot);
            if (i < k) hout[r] = st;
            obase += tot;
        }
        __syncthreads();
        // 4. element-parallel copy: an element's run is the number of heads at
        //    or before it, minus one
        rbase = 0;
        for (int j0 = 0; j0 < n; j0 += FIX_THREADS) {
            const int j = j0 + tid;
            const int v = j < n ? seg[j] : 0;
            const int h = (j < n && is_head(seg, j, v)) ? 1 : 0;
            int tot;
            const int r = rbase + fix_excl_scan(h, wsum, tot) + h - 1;
            if (j < n) out[hout[r] + (j - hpos[r])] = v + 1;
            rbase += tot;
        }
        __syncthreads();
        return;
    }
    unsigned long long* buf = gscratch + 2ll * s;
    if (tid == 0) kcount = 0;
    __syncthreads();
    for (int j = tid; j < n; j += FIX_THREADS) {
        const int v = seg[j];
        if (is_head(seg, j, v)) {
            const int idx = atomicAdd(&kcount, 1);
            buf[idx] = ((unsigned long long)(unsigned)(v >> 5) << 32) | (unsigned)j;
        }
    }
    __syncthreads();
    for (int t = k + tid; t < K; t += FIX_THREADS) buf[t] = ~0ull;
    __syncthreads();
    // Bitonic sort of the K keys (ascending).
    for (int size = 2; size <= K; size <<= 1) {
        for (int stride = size >> 1; stride > 0; stride >>= 1) {
            for (int i = tid; i < (K >> 1); i += FIX_THREADS) {
                const int lo = (i / stride) * 2 * stride + (i % stride);
                const int hi = lo + stride;
                const bool asc = (lo & size) == 0;
                const unsigned long long a = buf[lo], c = buf[hi];
                if ((a > c) == asc) {
                    buf[lo] = c;
                    buf[hi] = a;
                }
            }
            __syncthreads();
        }
    }
    // Copy the runs in sorted order; each run is at most 32 long.
    int base = 0;
    for (int c0 = 0; c0 < k; c0 += FIX_THREADS) {
        const int r = c0 + tid;
        int len = 0, j0 = 0;
        if (r < k) {
            const unsigned long long e = buf[r];
            j0 = int(e & 0xffffffffull);
            const int w = int(e >> 32);
            len = 1;
            while (j0 + len < n && (seg[j0 + len] >> 5) == w) ++len;
        }
        int total;
        const int excl = base + fix_excl_scan(len, wsum, total);
        for (int t = 0; t < len; ++t) out[excl + t] = seg[j0 + t] + 1;
        base += total;
    }
    __syncthreads();
}

// Segment S[s, s + n) to out, by one warp with its own shared arrays; false (and
// nothing written) if it has more than FIXW_RUNS runs.
__device__ __forceinline__ bool fixup_warp(int* hpos, int* hkey, int* hout, const int* __restrict__ seg, int n,
                                           int* __restrict__ out) {
    const int lane = threadIdx.x & 31;
    const unsigned full = 0xffffffffu, below = (1u << lane) - 1u;
    // A run is at most 32 long, so a longer segment has too many runs: hand it
    // over without walking it, and stop walking at the first run past the limit.
    if (n > FIXW_RUNS * 32) return false;
    int nruns = 0;
    // The segment is read FIXW_U chunks of 32 at a time, all loads of a batch
    // issued before any is used; the predecessor of a chunk's first element
    // is lane 31 of the chunk before.
    int last = -1;
    for (int J0 = 0; J0 < n && nruns <= FIXW_RUNS; J0 += 32 * FIXW_U) {
        int vv[FIXW_U];
#pragma unroll
        for (int u = 0; u < FIXW_U; ++u) {
            const int j = J0 + 32 * u + lane;
            vv[u] = j < n ? seg[j] : 0;
        }
#pragma unroll
        for (int u = 0; u < FIXW_U; ++u) {
            const int j0 = J0 + 32 * u;
            if (j0 >= n) break;
            const int j = j0 + lane, v = vv[u];
            int prev = __shfl_up_sync(full, v, 1);
            if (lane == 0) prev = last;
            last = __shfl_sync(full, v, 31);
            const bool head = j < n && (j == 0 || (prev >> 5) != (v >> 5));
            const unsigned hm = __ballot_sync(full, head);
            const int idx = nruns + __popc(hm & below);
            if (head && idx < FIXW_RUNS) {
                hpos[idx] = j;
                hkey[idx] = v >> 5;
            }
            nruns += __popc(hm);
        }
    }
    if (nruns > FIXW_RUNS) return false;
    if (lane == 0) hpos[nruns] = n;
    __syncwarp();
    // output start of each run: total length of the runs with a smaller chunk id
    for (int r = lane; r < nruns; r += 32) {
        const int key = hkey[r];
        int start = 0, at = hpos[0];
        for (int q = 0; q < nruns; ++q) {
            const int next = hpos[q + 1];
            if (hkey[q] < key) start += next - at;
            at = next;
        }
        hout[r] = start;
    }
    __syncwarp();
    // copy element-parallel: the run of element j is the number of heads at
    // or before j, minus one
    int rbase = 0;
    last = -1;
    for (int J0 = 0; J0 < n; J0 += 32 * FIXW_U) {
        int vv[FIXW_U];
#pragma unroll
        for (int u = 0; u < FIXW_U; ++u) {
            const int j = J0 + 32 * u + lane;
            vv[u] = j < n ? seg[j] : 0;
        }
#pragma unroll
        for (int u = 0; u < FIXW_U; ++u) {
            const int j0 = J0 + 32 * u;
            if (j0 >= n) break;
            const int j = j0 + lane, v = vv[u];
            int prev = __shfl_up_sync(full, v, 1);
            if (lane == 0) prev = last;
            last = __shfl_sync(full, v, 31);
            const bool head = j < n && (j == 0 || (prev >> 5) != (v >> 5));
            const unsigned hm = __ballot_sync(full, head);
            const int r = rbase + __popc(hm & (below | (1u << lane))) - 1;
            if (j < n) out[hout[r] + (j - hpos[r])] = v + 1;
            rbase += __popc(hm);
        }
    }
    __syncwarp();
    return true;
}

// A CTA takes 8 blocks of the list at a time, one per warp, and then together
// those that a warp could not do; one block at a time in crowded scenes (1024
// particles or more per block on average, whose blocks mostly have too many runs),
// fewer than 8 where there are too few blocks to give every CTA 8 (a 74 k particle
// sphere of 27 per cell, most blocks over the limit: 0.31 ms per two steps at one
// block per CTA, 0.40 at eight).
// One launch: as two (warps, then the blocks they listed) the second cost 2 us of
// every step. With `zero`, the counts of all blocks are zeroed (the next step's
// G2P counts into them).
__global__ void __launch_bounds__(FIX_THREADS) bin_fixup_kernel(const int* __restrict__ totals,
                                                                const int* __restrict__ blocklist,
                                                                const int* __restrict__ offsets,
                                                                const int* __restrict__ S, int* __restrict__ perm,
                                                                unsigned long long* __restrict__ gscratch,
                                                                int* __restrict__ zero, int nb) {
    chain_wait();
    constexpr int NWARP = FIX_THREADS / 32;
    __shared__ FixShared sm;
    __shared__ int whpos[NWARP][FIXW_RUNS + 1], whkey[NWARP][FIXW_RUNS], whout[NWARP][FIXW_RUNS];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int nactive = totals[0];
    const int take = (nactive > 0 && totals[1] / nactive >= 1024)
                         ? 1
                         : min(NWARP, (nactive + int(gridDim.x) - 1) / int(gridDim.x));
    for (int b0 = blockIdx.x * take; b0 < nactive; b0 += gridDim.x * take) {
        int over = -1;
        if (w < take && b0 + w < nactive) {
            const int b = blocklist[b0 + w] - 1, s = offsets[b];
            if (!fixup_warp(whpos[w], whkey[w], whout[w], S + s, offsets[b + 1] - s, perm + s)) over = b;
        }
        if (lane == 0) sm.over[w] = over;
        __syncthreads();
        for (int q = 0; q < take; ++q) {
            const int b = sm.over[q];  // uniform over the CTA
            if (b >= 0) fixup_cta(sm, S, offsets[b], offsets[b + 1] - offsets[b], perm, gscratch);
        }
        __syncthreads();
    }
    if (zero)
        for (int b = blockIdx.x * FIX_THREADS + threadIdx.x; b < nb; b += gridDim.x * FIX_THREADS) zero[b] = 0;
}

inline unsigned grid_for(long long n, int threads) { return unsigned((n + threads - 1) / threads); }

// The fix-up is set up early up to this many particles, in all and per mesh block.
// Whole steps with it early / in order, us: spheres in lattice order of 352 per mesh
// block (463 k) 197 / 180, of 386 (1.9 M) 582 / 581, of 147 (195 k) 117 / 111; a block of 57
// (512 k) 116.8 / 117.4, a column in block order of 135 (454 k) 117.3 / 118.4, a sphere in block
// order of 147 132.5 / 133.3. Blocks of 58 in lattice order: 1.7 M 498 / 500, 2.7 M 913 / 899,
// 3.5 M 1033 / 1022, 4.9 M 1489 / 1491; in block order 2.7 M 622 / 616.
constexpr long long FIX_EARLY_N = 1 << 21, FIX_EARLY_PER_BLOCK = 128;

constexpr int SCAN_ONE = 16;  // tiles up to which the scan is one launch

void launch_scan(const int* counts, int nb, unsigned long long* partials, int* offsets, int* cursors, int* blocklist,
                 int* totals, unsigned long long* bnd_count, const TouchArgs& touch, const LaunchCfg& cfg) {
    const int nt = scan_tiles(nb);
    if (nt <= SCAN_ONE) {
        launch_chained(scan_kernel<true>, nt, 256, 0, cfg, counts, nb, partials, offsets, cursors, blocklist, totals,
                                                      bnd_count, touch);
        ++*cfg.launches;
        return;
    }
    launch_chained(scan_reduce_kernel, nt, 256, 0, cfg, counts, nb, partials);
    launch_chained(scan_kernel<false>, nt, 256, 0, cfg, counts, nb, partials, offsets, cursors, blocklist, totals, bnd_count,
                                                   touch);
    *cfg.launches += 2;
}

// ---- sparse grid numbering ----------------------------------------------
// act[B] = 1 for every node block B within one block per axis of a block that
// holds particles (act zeroed before). Several threads may store the same 1.
template <int D>
__global__ void __launch_bounds__(128) sparse_mark_kernel(const int* __restrict__ totals,
                                                          const int* __restrict__ blocklist, int3 nb,
                                                          int* __restrict__ act) {
    const int nactive = totals[0];
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < nactive; i += gridDim.x * blockDim.x) {
        const int b = blocklist[i] - 1;
        const int bx = b % nb.x, by = (b / nb.x) % nb.y, bz = (D == 3) ? b / (nb.x * nb.y) : 0;
        for (int dz = (D == 3 ? -1 : 0); dz <= (D == 3 ? 1 : 0); ++dz)
            for (int dy = -1; dy <= 1; ++dy)
                for (int dx = -1; dx <= 1; ++dx) {
                    const int x = bx + dx, y = by + dy, z = bz + dz;
                    if (x < 0 || y < 0 || z < 0 || x >= nb.x || y >= nb.y || (D == 3 && z >= nb.z)) continue;
                    act[x + nb.x * (y + nb.y * z)] = 1;
                }
    }
}

// bnum[B] = (rank of B among the active blocks) + 1, or 0; the count to nact[0].
__global__ void __launch_bounds__(256) sparse_number_kernel(const int* __restrict__ act,
                                                            const int* __restrict__ offsets, int nb,
                                                            const int* __restrict__ totals, int* __restrict__ bnum,
                                                            int* __restrict__ nact) {
    for (int B = blockIdx.x * blockDim.x + threadIdx.x; B < nb; B += gridDim.x * blockDim.x) {
        bnum[B] = act[B] ? offsets[B] + 1 : 0;
        if (B == 0) nact[0] = totals[0];
    }
}

}  // namespace

cudaError_t launch_sparsity(int dim, const int* nbv, int nblocks, const BinBuffers& b, const SparseScratch& sc,
                            int* bnum, int* blist, int* nact, const LaunchCfg& cfg) {
    cudaError_t e = cudaMemsetAsync(sc.act, 0, sizeof(int) * size_t(nblocks), cfg.stream);
    if (e != cudaSuccess) return e;
    KernelScope ks(cfg, "sparsity");
    const int3 nb = make_int3(nbv[0], nbv[1], nbv[2]);
    const int mgrid = std::max(1, std::min((nblocks + 127) / 128, cfg.num_sms * 8));
    if (dim == 3) sparse_mark_kernel<3><<<mgrid, 128, 0, cfg.stream>>>(b.totals, b.blocklist, nb, sc.act);
    else sparse_mark_kernel<2><<<mgrid, 128, 0, cfg.stream>>>(b.totals, b.blocklist, nb, sc.act);
    // the binning's scan over the activity: offsets = ranks, blocklist = the active list
    launch_scan(sc.act, nblocks, sc.partials, sc.offsets, sc.cursors, blist, sc.totals, nullptr, TouchArgs{}, cfg);
    sparse_number_kernel<<<std::max(1, std::min((nblocks + 255) / 256, cfg.num_sms * 8)), 256, 0, cfg.stream>>>(
        sc.act, sc.offsets, nblocks, sc.totals, bnum, nact);
    *cfg.launches += 2;
    return cudaGetLastError();
}

template <int D, class T>
cudaError_t launch_bin_count(const DMesh<D, T>& M, const T* const* x, long long n, const BinBuffers& b,
                             const LaunchCfg& cfg) {
    cudaError_t e = cudaMemsetAsync(b.counts, 0, sizeof(int) * size_t(M.nblocks), cfg.stream);
    if (e != cudaSuccess) return e;
    if (n > 0) {
        KernelScope ks(cfg, "bin_count");
        launch_chained(bin_count_kernel<D, T>, grid_for(n, 256), 256, 0, cfg, M, x[0], x[1], D == 3 ? x[2] : x[1], n,
                                                                         b.blockids, b.counts);
        ++*cfg.launches;
    }
    return cudaGetLastError();
}

cudaError_t launch_bin_rest(int nb, long long n, const BinBuffers& b, const LaunchCfg& cfg, const TouchArgs& touch,
                            bool zero_counts) {
    {
        KernelScope ks(cfg, "bin_scan");
        launch_scan(b.counts, nb, b.partials, b.offsets, b.cursors, b.blocklist, b.totals, b.bnd_count, touch, cfg);
    }
    if (n > 0) {
        {
            KernelScope ks(cfg, "bin_scatter");
            launch_chained(bin_scatter_kernel, grid_for(n, 256 * SCAT_IT), 256, 0, cfg, b.blockids, n, b.cursors,
                                                                                  b.perm_tmp);
        }
        KernelScope ks(cfg, "bin_fixup");
        const int grid = std::max(1, std::min(nb, cfg.num_sms * 5));
        LaunchCfg fix = cfg;
        fix.early = cfg.early && n <= FIX_EARLY_N && n <= FIX_EARLY_PER_BLOCK * nb;
        launch_chained(bin_fixup_kernel, grid, FIX_THREADS, 0, fix, b.totals, b.blocklist, b.offsets, b.perm_tmp, b.perm,
                                                               b.sort_scratch, zero_counts ? b.counts : nullptr, nb);
        *cfg.launches += 2;
    }
    return cudaGetLastError();
}

template <int D, class T>
cudaError_t launch_bin(const DMesh<D, T>& M, const T* const* x, long long n, const BinBuffers& b,
                       const LaunchCfg& cfg, const TouchArgs& touch, bool zero_counts) {
    cudaError_t e = launch_bin_count<D, T>(M, x, n, b, cfg);
    if (e != cudaSuccess) return e;
    return launch_bin_rest(M.nblocks, n, b, cfg, touch, zero_counts);
}

#define TB_INST_BIN(D, T)                                                                                     \
    template cudaError_t launch_bin<D, T>(const DMesh<D, T>&, const T* const*, long long, const BinBuffers&, \
                                          const LaunchCfg&, const TouchArgs&, bool);                          \
    template cudaError_t launch_bin_count<D, T>(const DMesh<D, T>&, const T* const*, long long,              \
                                                const BinBuffers&, const LaunchCfg&);
TB_INST_BIN(3, double)
TB_INST_BIN(3, float)
TB_INST_BIN(2, double)
TB_INST_BIN(2, float)

}  // namespace tb
