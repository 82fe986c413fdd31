// fbk_bins.cu — the build front end (src/graph/build.rs:84-328) over minimizer bins: every
// k-mer of the reads is counted in shared memory, once, and the Count-Min Sketch gate is
// applied to distinct k-mers instead of to their occurrences.
//
//   1. k_bin_runs cuts every read into runs of consecutive windows that share their
//      minimizer (the smallest hash of the canonical m-mers in the middle of the window; a
//      window and its reverse complement have the same one) and logs each run — its first
//      base, its window count and whether the windows before and after it exist — with the
//      bin of its minimizer;
//   2. the runs are scattered by bin (k_bin_scan*, k_bin_scatter): all occurrences of a
//      k-mer lie in one bin;
//   3. the windows of bins with many times the others' are scattered again, by their keys
//      (split_heavy); k_bin_agg takes those and groups of consecutive bins, about as many as
//      fill a hash table in shared memory, reads their windows' bases from the packed bank
//      again and adds up, per distinct canonical k-mer, its 8 edge counts (build.rs:243-289
//      without the gate).
//      A key seen twice or more becomes a row of a dense array; of a key seen once, only
//      its place in the bank is kept, as a bit of a bitmap over the bases;
//   4. every distinct key enters the pass-1 sketch with its whole count at once
//      (k_bin_sketch, k_singles), the sketch being the two-level threshold ladder of
//      fbk_k_ladder.cu: t_solid is 2 here, the default (build.rs:141);
//   5. the gate (build.rs:259-267): a key seen twice passes by itself, so only the keys
//      seen once ask the sketch (k_singles), each once, and the windows that fail are a
//      bitmap.  A push of the reference needs both windows of a transition to pass: the
//      neighbours of a key seen once are the next bits of the bitmap, and a row's edge
//      that was crossed twice leads to a key seen twice.  What is left, the edges of rows
//      that were crossed once, asks the sketch for the neighbour k-mer (k_bin_gate).
//   The rows that remain are the accumulator (KmerAcc) and are converted as a table is.
//
// Why this shape: the occurrence-wise passes (fbk_k_ladder.cu, fbk_k_roll.cu, fbk_k_pass.cu)
// spend 8 random L2 loads on the gate and a table probe and 2 L2 atomics per occurrence, and
// an SM serves one such lane a cycle.  Shared memory serves 32 lanes in 3-4 cycles, and the
// gate's loads fall on the distinct k-mers (4-10 times fewer at 100x).  Device time at 5 Mbp
// and 100x (485 M bases; 418 / 373 / 305 / 232 M windows), 2^24 columns, 0.5% errors:
//   k                     21     33     55     77
//   over occurrences    20.4   23.3   20.8   21.3 ms
//   here                11.9   13.1   11.6   11.8
//     runs, scatter      3.4    2.6    1.9    1.9
//     aggregate          5.2    5.8    6.2    6.3
//     sketch, gate       2.2    2.7    2.9    3.2
// The same entry takes a sketch that the caller keeps (AGG_COUNT) and the estimator's sample
// loop (bins_first).
#include <algorithm>
#include <cmath>

#include "fbk_device.cuh"
#include "fbk_internal.h"
#include "fbk_table.cuh"

namespace fbk {
namespace {

// A logged run: bits 0-31 first base, 32-43 windows, 44 / 45 the window before / after it
// exists in the read, 46-63 bin.
constexpr uint32_t RUN_MAX_BINS = 1u << 18;
constexpr uint32_t RUN_SPLIT = 2048;  // a run is cut where the window number is a multiple of this
__device__ __forceinline__ uint64_t run_pack(uint64_t off, uint32_t n, bool left, bool right, uint32_t bin) {
    return (off & 0xFFFFFFFFull) | ((uint64_t)n << 32) | ((uint64_t)left << 44) | ((uint64_t)right << 45) | ((uint64_t)bin << 46);
}

// The m-mers compared for a window: positions [skip, skip + w) of its k - m + 1.  The
// middle is symmetric under reverse complement, so both strands see the same set.
struct MinPlan {
    uint32_t m, w, skip;
};
// m: short enough that a window has many of them (long runs: fewer to log, count and scatter),
// long enough that a genome repeats few by chance, as a minimizer's places all go to one bin.
// At 5 and 12 Mbp (5 Mbp, 100x, whole build): k = 21, m = 9 13.2 ms, 10 12.5, 11 12.6, 12 12.9;
// k = 25, m = 11 12.3, 12 12.4, 14 12.7; k = 31, m = 13 12.5, 15 12.6; k = 45 the same for both.
// w at most 32: runs of about (w + 1) / 2 windows, short enough that the keys of one
// minimizer stay a small part of a group (at k = 77 and 100x about 15 distinct k-mers per
// genome position, 240 per minimizer of a group of 1700).
MinPlan min_plan(uint32_t k) {
    MinPlan p;
    p.m = k >= 40 ? 15 : std::min(13u, std::max(10u, (k - 3) / 2));
    const uint32_t full = k - p.m + 1;
    p.w = full <= 32 ? full : 32 - ((full ^ 32u) & 1u);
    p.skip = (full - p.w) / 2;
    return p;
}

// Reverses the order of the 16 2-bit groups of x.
__device__ __forceinline__ uint32_t rev2_32(uint32_t x) {
    x = __brev(x);
    return ((x >> 1) & 0x55555555u) | ((x & 0x55555555u) << 1);
}

constexpr int RUN_CHUNKS = 6;  // windows per tile: 6 x 32
constexpr uint32_t RUN_QUEUE = 64;  // runs of a warp that wait for their bin, a power of two

// The hashes of up to 32 NC m-mers from base g0 on (lane j of chunk c has m-mer 32 c + j), and
// the minimum over each w of them that follow one another: h[i] <- min of h[i .. i + 2^s), then
// of the two windows of 2^s that cover w.  Lanes past the last m-mer repeat it: no window asks
// for theirs.
template <int NC>
__device__ __forceinline__ void run_minima(const uint32_t* __restrict__ d32, uint32_t g0, uint32_t n_mers, uint32_t msh, uint32_t mmask,
                                           uint32_t w, uint32_t (&out)[RUN_CHUNKS + 1]) {
    const uint32_t lane = threadIdx.x & 31;
    uint32_t h[NC];
#pragma unroll
    for (int c = 0; c < NC; ++c) {
        const uint32_t i = g0 + (c + 1 < NC ? 32 * c + lane : min(32 * c + lane, n_mers - 1));
        const uint32_t x = __funnelshift_r(d32[i >> 4], d32[(i >> 4) + 1], (i & 15) << 1);
        const uint32_t c0 = min(rev2_32(x) >> msh, ~x & mmask);
        uint32_t z = (c0 ^ 0x3C6EF372u) * 0x9E3779B1u;
        z ^= z >> 15;
        h[c] = z * 0x85EBCA77u;
    }
    auto step = [&](uint32_t by) {
        const uint32_t from = (lane + by) & 31;
        const bool next = lane < by;
#pragma unroll
        for (int c = 0; c < NC; ++c) {
            const uint32_t nx = c + 1 < NC ? h[c + 1 < NC ? c + 1 : c] : 0xFFFFFFFFu;
            h[c] = min(h[c], __shfl_sync(0xffffffffu, next ? nx : h[c], from));
        }
    };
    uint32_t span = 1;
    for (; 2 * span <= w; span *= 2) step(span);
    if (w > span) step(w - span);
#pragma unroll
    for (int c = 0; c < NC; ++c) out[c] = h[c];
}

// One warp per read, lane = window; a sliding minimum over the w m-mers of a window takes
// log2(w) steps of one shuffle each, with the read's hashes in registers.  Runs that end wait
// in shared memory until there are 32, which are binned, counted and logged together: 2 runs
// end in 32 windows at k of 46 and more.  Bound by instruction issue: about 25 instructions
// per 32 m-mers for their hashes, 4 per step of the minimum, 40 for the ends of runs.
// 5 Mbp at 100x, 500 M bases: k = 31 2.66 ms with a run binned by the lane that ends it and the
// chunks counted at run time, 2.09 so, 1.98 with the next read's length and place loaded ahead;
// k = 77 2.18, 1.73, 1.64.
__global__ void __launch_bounds__(256) k_bin_runs(BankDev b, uint32_t k, MinPlan mp, uint32_t n_bins, uint64_t* __restrict__ log,
                                                  uint32_t* __restrict__ log_n, uint32_t cap_w, unsigned long long* __restrict__ hist,
                                                  unsigned long long* __restrict__ need) {
    __shared__ uint4 s_queue[8][RUN_QUEUE];  // first base, windows | left << 12 | right << 13, minimizer
    const uint32_t lane = threadIdx.x & 31;
    const uint64_t gw = ((uint64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const uint64_t nwarps = ((uint64_t)gridDim.x * blockDim.x) >> 5;
    const uint32_t* __restrict__ d32 = reinterpret_cast<const uint32_t*>(b.data);
    const uint32_t msh = 32 - 2 * mp.m, mmask = 0xFFFFFFFFu >> msh;
    uint4* queue = s_queue[threadIdx.x >> 5];
    uint64_t* out = log + gw * cap_w;
    uint32_t n_out = 0, n_in = 0;  // warp-uniform: runs logged, runs ended
    auto flush = [&](uint32_t n) {  // the n oldest of the queue
        __syncwarp();
        if (lane < n) {
            const uint4 e = queue[(n_out + lane) % RUN_QUEUE];
            const uint32_t windows = e.y & 0xFFFu;
            const uint32_t z = e.z ^ (e.z >> 16);
            const uint32_t bin = __umulhi(z * 0xC2B2AE3Du, n_bins);
            if (n_out + lane < cap_w) out[n_out + lane] = run_pack(e.x, windows, (e.y >> 12) & 1u, (e.y >> 13) & 1u, bin);
            atomicAdd(&hist[bin], (1ull << 32) | windows);
        }
        n_out += n;
        __syncwarp();
    };
    uint32_t len_next = 0, off_next = 0;  // of the warp's next read, loaded ahead (the bank holds fewer than 2^32 bases)
    if (b.r_begin + gw < b.r_end) len_next = b.len[b.r_begin + gw], off_next = (uint32_t)b.off[b.r_begin + gw];
    for (uint64_t r = b.r_begin + gw; r < b.r_end; r += nwarps) {
        const uint32_t len = len_next, off = off_next;
        if (r + nwarps < b.r_end) len_next = b.len[r + nwarps], off_next = (uint32_t)b.off[r + nwarps];
        if (len < k || !bank_keep(b, r)) continue;
        const uint32_t nk = len - k + 1;
        uint32_t start = 0, prev_min = 0;  // first window of the open run; minimizer of the last window seen
        for (uint32_t q0 = 0; q0 <= nk; q0 += 32 * RUN_CHUNKS) {
            const uint32_t n_mers = min(nk - q0, 32u * RUN_CHUNKS) + mp.w - 1;  // q0 == nk: no window left, only the end
            const uint32_t g0 = off + q0 + mp.skip;
            uint32_t h[RUN_CHUNKS + 1];
            const uint32_t nc = (n_mers + 31) / 32;
            switch (nc) {
                case 1: run_minima<1>(d32, g0, n_mers, msh, mmask, mp.w, h); break;
                case 2: run_minima<2>(d32, g0, n_mers, msh, mmask, mp.w, h); break;
                case 3: run_minima<3>(d32, g0, n_mers, msh, mmask, mp.w, h); break;
                case 4: run_minima<4>(d32, g0, n_mers, msh, mmask, mp.w, h); break;
                case 5: run_minima<5>(d32, g0, n_mers, msh, mmask, mp.w, h); break;
                case 6: run_minima<6>(d32, g0, n_mers, msh, mmask, mp.w, h); break;
                default: run_minima<7>(d32, g0, n_mers, msh, mmask, mp.w, h); break;
            }
#pragma unroll
            for (int c = 0; c < RUN_CHUNKS; ++c) {
                const uint32_t qc = q0 + 32 * c;
                if (qc > nk) break;
                const uint32_t q = qc + lane;
                uint32_t before = __shfl_up_sync(0xffffffffu, h[c], 1);
                if (lane == 0) before = prev_min;
                // a run ends before window q (or at the read's end)
                const bool cut = q <= nk && q > 0 && (q == nk || h[c] != before || q % RUN_SPLIT == 0);
                const uint32_t mask = __ballot_sync(0xffffffffu, cut);
                if (cut) {
                    const uint32_t below = mask & ((1u << lane) - 1);
                    const uint32_t s = below ? qc + 31 - __clz(below) : start;
                    queue[(n_in + __popc(below)) % RUN_QUEUE] =
                        make_uint4(off + s, (q - s) | (s > 0 ? 1u << 12 : 0u) | (q < nk ? 1u << 13 : 0u), before, 0);
                }
                n_in += __popc(mask);
                if (mask) start = qc + 31 - __clz(mask);
                prev_min = __shfl_sync(0xffffffffu, h[c], 31);
                if (n_in - n_out >= 32) flush(32);
            }
        }
    }
    flush(n_in - n_out);
    if (lane == 0) {
        log_n[gw] = min(n_out, cap_w);
        if (n_out > cap_w) atomicMax(need, (unsigned long long)n_out);
    }
}

// Exclusive prefix of the bins' (runs << 32 | windows); both totals stay below 2^32, so one
// 64-bit sum carries the two.  Blocks of 1024 bins: their sums, then the bins' prefixes.
constexpr uint32_t SCAN_TILE = 1024;
__global__ void __launch_bounds__(256) k_bin_scan_sums(const unsigned long long* __restrict__ hist, uint32_t n,
                                                       unsigned long long* __restrict__ part) {
    __shared__ unsigned long long s[8];
    unsigned long long v = 0;
    for (uint32_t j = 0; j < 4; ++j) {
        const uint32_t i = blockIdx.x * SCAN_TILE + j * 256 + threadIdx.x;
        if (i < n) v += hist[i];
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
    if ((threadIdx.x & 31) == 0) s[threadIdx.x >> 5] = v;
    __syncthreads();
    if (threadIdx.x == 0) {
        for (int j = 1; j < 8; ++j) v += s[j];
        part[blockIdx.x] = v;
    }
}
// big (not null): the windows in bins of more than 2^13, 2^15 and 2^17 of them.
__global__ void __launch_bounds__(256) k_bin_scan(const unsigned long long* __restrict__ hist, uint32_t n,
                                                  const unsigned long long* __restrict__ part, unsigned long long* __restrict__ pre,
                                                  uint32_t* __restrict__ cursor, unsigned long long* __restrict__ big) {
    __shared__ unsigned long long s[8], s_base;
    const uint32_t lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    unsigned long long v = 0;
    for (uint32_t j = threadIdx.x; j < blockIdx.x; j += 256) v += part[j];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
    if (lane == 0) s[w] = v;
    __syncthreads();
    if (threadIdx.x == 0) {
        for (int j = 1; j < 8; ++j) v += s[j];
        s_base = v;
    }
    __syncthreads();
    const uint32_t i0 = blockIdx.x * SCAN_TILE + threadIdx.x * 4;
    unsigned long long x[4], t = 0;
    for (int j = 0; j < 4; ++j) {
        x[j] = i0 + j < n ? hist[i0 + j] : 0;
        t += x[j];
    }
    unsigned long long inc = t;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const unsigned long long y = __shfl_up_sync(0xffffffffu, inc, o);
        if (lane >= (uint32_t)o) inc += y;
    }
    if (lane == 31) s[w] = inc;
    __syncthreads();
    unsigned long long p = s_base + inc - t;
    for (uint32_t j = 0; j < w; ++j) p += s[j];
    for (int j = 0; j < 4; ++j) {
        if (i0 + j < n) {
            pre[i0 + j] = p;
            cursor[i0 + j] = (uint32_t)(p >> 32);
        }
        p += x[j];
        if (i0 + j == n - 1) pre[n] = p;
        const uint32_t windows = (uint32_t)x[j];
        if (big && windows > 1u << 13) {  // rare (HEAVY_FROM)
            for (int c = 0; c < 3; ++c)
                if (windows > 1u << (13 + 2 * c)) atomicAdd(&big[c], (unsigned long long)windows);
        }
    }
}

// Moves every logged run to its bin's range.  One returning atomic and one 8-byte store per
// run; the bins' open ends (8 MB of sectors at most) stay in L2 until full.  Bound by the L2
// (59% of its peak, DRAM 19%, issue 15%): 5 Mbp at 100x, 64 M runs of k = 21 1.4 ms, 14 M of
// k = 77 0.27.  Eight runs a lane, or half and a quarter of the bins, took as long.
__global__ void __launch_bounds__(256) k_bin_scatter(const uint64_t* __restrict__ log, const uint32_t* __restrict__ log_n, uint32_t cap_w,
                                                     uint32_t* __restrict__ cursor, uint64_t* __restrict__ runs, uint64_t cap) {
    const uint32_t lane = threadIdx.x & 31;
    const uint64_t gw = ((uint64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const uint64_t* in = log + gw * cap_w;
    const uint32_t n = log_n[gw];
    // four runs a lane: their atomics are in flight together
    for (uint32_t i0 = lane; i0 < n; i0 += 128) {
        uint64_t e[4];
        uint32_t p[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) e[j] = i0 + 32 * j < n ? __ldcs(in + i0 + 32 * j) : 0;
#pragma unroll
        for (int j = 0; j < 4; ++j)
            if (i0 + 32 * j < n) p[j] = atomicAdd(&cursor[e[j] >> 46], 1u);
#pragma unroll
        for (int j = 0; j < 4; ++j)
            if (i0 + 32 * j < n && p[j] < cap) runs[p[j]] = e[j];
    }
}

// Groups of consecutive bins of about `target` windows: bin i belongs to group
// floor(windows before it / target), and one of 2 target windows and more, which reaches past
// the next group, to that one alone.  (A frequent k-mer's bin with ordinary ones before it: its
// group has wide counts and so fewer entries, and where the keys did not fit, all of its windows
// were counted twice.  Poly-G in 5% of 1.2 M reads, k = 21: 14.5 or 27.6 ms a build before.)
// start[g] = the prefix (runs << 32 | windows) at the first bin of group g, start[n_groups] =
// the totals.
__global__ void k_bin_groups(const unsigned long long* __restrict__ pre, uint32_t n, uint32_t target, uint32_t n_groups,
                             unsigned long long* __restrict__ start) {
    auto group = [&](uint32_t i) {
        const uint32_t before = (uint32_t)pre[i], windows = (uint32_t)pre[i + 1] - before;
        return before / target + (windows / 2 >= target);
    };
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i <= n; i += gridDim.x * blockDim.x) {
        const uint32_t lo = i ? group(i - 1) + 1 : 0;
        const uint32_t hi = i < n ? group(i) : n_groups;
        for (uint32_t g = lo; g <= hi && g <= n_groups; ++g) start[g] = pre[i];
    }
}

// A window cut from the packed bank in 32-bit words (16 bases each): one funnel shift a
// word and direction, where 64-bit shifts by a lane's own amount take four instructions.
// Canonical key as NK significant big-endian words, its strand (rc iff rc < fwd), and the
// bases before and after the window (read only where the caller knows that they exist).
template <int NK>
__device__ __forceinline__ void window_at(const uint32_t* __restrict__ d, uint32_t g, uint32_t k, uint64_t (&can)[NK], bool& is_rc,
                                          uint32_t& before, uint32_t& after) {
    constexpr int N = 2 * NK;
    const uint32_t wi = g >> 4, sh = (g & 15) << 1;
    uint32_t w[N + 1], u[N];
#pragma unroll
    for (int i = 0; i <= N; ++i) w[i] = d[wi + i];
#pragma unroll
    for (int i = 0; i < N; ++i) u[i] = __funnelshift_r(w[i], w[i + 1], sh);
    before = __funnelshift_r(d[wi ? wi - 1 : 0], w[0], sh) >> 30;
    // base k of the stream: in the last two words of the field, or the next one for k = 32 NK
    const uint32_t ka = k >> 4;
    after = ka == N - 1 ? u[N - 1] : ka == N - 2 ? u[N - 2] : __funnelshift_r(w[N], d[wi + N + 1], sh);
    after = (after >> ((k & 15) << 1)) & 3u;
    // fwd: the 2-bit groups reversed, then shifted right by 64 NK - 2k bits (0 .. 62)
    const uint32_t bs = 64u * NK - 2u * k, b5 = bs & 31;
    uint32_t f[N], r[N];
#pragma unroll
    for (int i = 0; i < N; ++i) f[i] = rev2_32(u[i]);
    if (bs >= 32) {
#pragma unroll
        for (int i = N - 1; i >= 0; --i) f[i] = i >= 1 ? __funnelshift_r(f[i >= 1 ? i - 1 : 0], i >= 2 ? f[i >= 2 ? i - 2 : 0] : 0u, b5) : 0u;
    } else {
#pragma unroll
        for (int i = N - 1; i >= 0; --i) f[i] = __funnelshift_r(f[i], i >= 1 ? f[i >= 1 ? i - 1 : 0] : 0u, b5);
    }
    // rc: the complement of the field; LSB-first word i is big-endian word N - 1 - i, and
    // only the top two can reach past 2k bits
#pragma unroll
    for (int i = 0; i < N; ++i) {
        r[N - 1 - i] = ~u[i];
        if (i >= N - 2) {
            const int bits = (int)(2 * k) - 32 * i;
            r[N - 1 - i] &= bits >= 32 ? 0xFFFFFFFFu : bits <= 0 ? 0u : (1u << bits) - 1;
        }
    }
    bool lt = false, eq = true;
    uint64_t F[NK], R[NK];
#pragma unroll
    for (int i = 0; i < NK; ++i) {
        F[i] = ((uint64_t)f[2 * i] << 32) | f[2 * i + 1];
        R[i] = ((uint64_t)r[2 * i] << 32) | r[2 * i + 1];
        lt = lt || (eq && R[i] < F[i]);
        eq = eq && R[i] == F[i];
    }
    is_rc = lt;
#pragma unroll
    for (int i = 0; i < NK; ++i) can[i] = lt ? R[i] : F[i];
}
template <int NK>
struct Window {  // a window as k_bin_agg counts it
    uint64_t key[NK], fold;
    uint32_t left, right;   // the bases before and after it
    uint32_t bucket, tag;   // where its key's slot is looked for, and the slot's high half
    bool rc;
};
template <int NK>
__device__ __forceinline__ uint64_t fold_of(const uint64_t (&w)[NK]) {
    uint64_t f = 0;
#pragma unroll
    for (int i = 0; i < NK; ++i) f ^= w[i];
    return f;
}

// Heavy bins.  A minimizer that is frequent in the genome (poly-A, the short words of an AT-rich
// one) brings many keys into one bin, which is one block's: it took them in parts as large as its
// table, each over all of the bin's windows.  So the windows of a bin of more than three
// target groups are scattered again, most as runs of one window, over sub-bins of about `target`
// windows by a hash of the key, and these are groups of their own.  Reads of 150 bases at 60x, the
// whole build over records / with heavy bins taken in parts / so, in ms:
//   5 Mbp, GC 0.15, k = 21                       12.9 / 45.2 / 10.2
//   5 Mbp, GC 0.2, a tract of A or T every 500   17.1 / 53.2 /  9.6   (k = 77 13.3 / 27.3 / 7.7)
//   12 Mbp, GC 0.2, a tract every 1000           41.4 / 116  / 24.8   (k = 31 33.7 / 56.8 / 17.5)
// Bins of 2^13 windows and fewer stay whole (0.03 ms of a block's time a part).  Pieces of such a
// bin's runs:
struct HeavyPiece {
    uint32_t begin, end;  // runs
    uint32_t sub, parts;  // sub-bins [sub, sub + parts)
};
constexpr uint32_t HEAVY_PIECE = 1024;  // runs
constexpr uint32_t HEAVY_FROM = 1u << 13;  // not less: k_bin_scan counts the windows of bins above it
// counts: pieces, sub-bins.
__global__ void k_heavy_pieces(const unsigned long long* __restrict__ pre, uint32_t n, uint32_t target, uint32_t from,
                               HeavyPiece* __restrict__ pieces, uint32_t cap, uint32_t* __restrict__ counts) {
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const unsigned long long a = pre[i], b = pre[i + 1];
        const uint32_t windows = (uint32_t)b - (uint32_t)a;
        if (windows <= from) continue;
        const uint32_t r0 = (uint32_t)(a >> 32), r1 = (uint32_t)(b >> 32), np = (r1 - r0 + HEAVY_PIECE - 1) / HEAVY_PIECE;
        const uint32_t parts = windows / target + 1, sub = atomicAdd(counts + 1, parts), p = atomicAdd(counts, np);
        for (uint32_t q = 0; q < np && p + q < cap; ++q)
            pieces[p + q] = {r0 + q * HEAVY_PIECE, min(r1, r0 + (q + 1) * HEAVY_PIECE), sub, parts};
    }
}

// Counts the windows of the pieces by sub-bin (PUT: moves them there), a block per piece, a warp
// per 32 runs, a lane per window.  Windows of one sub-bin that meet in a warp share an atomic.
// Bound by latency and issue: 5 Mbp of GC 0.15 at 25x, k = 21, 0.27 ms to count and 0.36 to move,
// half of the issue slots, L2 12 and 23%, DRAM 4 and 12%.
template <int NK, bool PUT>
__global__ void __launch_bounds__(256) k_heavy_split(const uint64_t* __restrict__ data, const uint64_t* __restrict__ runs,
                                                     const HeavyPiece* __restrict__ pieces, const uint32_t* __restrict__ counts, uint32_t cap,
                                                     uint32_t k, unsigned long long* __restrict__ hist, uint32_t* __restrict__ cursor,
                                                     uint64_t* __restrict__ out, uint64_t cap_out) {
    const uint32_t lane = threadIdx.x & 31;
    const uint32_t* __restrict__ d32 = reinterpret_cast<const uint32_t*>(data);
    const uint32_t n_pieces = min(counts[0], cap);
    for (uint32_t p = blockIdx.x; p < n_pieces; p += gridDim.x) {
        const HeavyPiece piece = pieces[p];
        for (uint32_t r = piece.begin + (threadIdx.x & ~31u); r < piece.end; r += 256) {
            const uint64_t e = r + lane < piece.end ? runs[r + lane] : 0;
            const uint32_t n = (uint32_t)(e >> 32) & 0xFFFu;
            uint32_t inc = n;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const uint32_t y = __shfl_up_sync(0xffffffffu, inc, o);
                if (lane >= (uint32_t)o) inc += y;
            }
            // (the windows of the runs one after another, as in k_bin_agg)
            const uint32_t total = __shfl_sync(0xffffffffu, inc, 31), first = inc - n, shift = (uint32_t)e - first;
            const uint32_t edge_l = (e >> 44) & 1u ? 0xFFFFFFFFu : first, edge_r = (e >> 45) & 1u ? 0xFFFFFFFFu : inc - 1;
            for (uint32_t base = 0, before = 0; base < total; base += 32) {
                const uint32_t rel = first - base;
                const uint32_t starts = __reduce_or_sync(0xffffffffu, n && rel < 32 ? 1u << rel : 0u);
                const int run = (int)(before + __popc(starts & ((2u << lane) - 1))) - 1;
                before += __popc(starts);
                const bool live = base + lane < total;
                const uint32_t x = min(base + lane, total - 1);
                const uint32_t g = __shfl_sync(0xffffffffu, shift, run) + x;
                const bool has_l = __shfl_sync(0xffffffffu, edge_l, run) != x, has_r = __shfl_sync(0xffffffffu, edge_r, run) != x;
                uint64_t key[NK];
                bool rc;
                uint32_t bl, br;
                window_at<NK>(d32, g, k, key, rc, bl, br);
                // (not the hash that places a key in a block's table or that takes a group in parts)
                const uint64_t f = fold_of<NK>(key);
                const uint32_t sub = live ? piece.sub + __umulhi((uint32_t)(((f ^ (f >> 29)) * 0xD6E8FEB86659FD93ULL) >> 32), piece.parts) : 0xFFFFFFFFu;
                // windows of a run that follow one another into the same sub-bin (poly-G) stay a run
                const uint32_t sub_before = __shfl_up_sync(0xffffffffu, sub, 1);
                const int run_before = __shfl_up_sync(0xffffffffu, run, 1);
                const bool head = live && (lane == 0 || run != run_before || sub != sub_before);
                const uint32_t heads = __ballot_sync(0xffffffffu, head), lives = __ballot_sync(0xffffffffu, live);
                const uint32_t same = __match_any_sync(0xffffffffu, sub);  // its first lane is a head
                const int leader = __ffs(same) - 1;
                const uint32_t n_same = __popc(same & heads);
                if constexpr (PUT) {
                    uint32_t at = 0;
                    if (live && (int)lane == leader) at = atomicAdd(&cursor[sub], n_same);
                    at = __shfl_sync(0xffffffffu, at, leader) + __popc(same & heads & ((1u << lane) - 1));
                    const uint32_t above = heads & ~((2u << lane) - 1);
                    const uint32_t len = (above ? __ffs(above) - 1 : __popc(lives)) - lane;
                    const bool last_r = __shfl_sync(0xffffffffu, has_r, min(lane + (head ? len : 1u) - 1, 31u));
                    if (head && at < cap_out) out[at] = run_pack(g, len, has_l, last_r, 0);
                } else if (live && (int)lane == leader) {
                    atomicAdd(&hist[sub], ((unsigned long long)n_same << 32) | (uint32_t)__popc(same));
                }
            }
        }
    }
}

// Counters of a build (u64): rows, low rows, keys seen once, adjacent solid windows, reads of one
// window; of the sample: distinct keys, those seen twice, those that can become solid, windows;
// log words a warp needed; groups handed out (aggregate, sample); windows in large bins
// (k_bin_scan).
enum { BC_ROWS, BC_LOW, BC_SINGLES, BC_PAIRS, BC_LONE, BC_DISTINCT, BC_MULTI, BC_KEPT, BC_WINDOWS, BC_NEED, BC_WORK, BC_WORK_S,
       BC_BIG, BC_N = BC_BIG + 3 };

struct FirstKey {
    uint64_t raw;        // canonical ntHash
    uint32_t at, again;  // the first two places in the bank (0xFFFFFFFF: none)
};
struct AggArgs {
    const uint64_t* data;
    const uint64_t* runs;
    const unsigned long long* start;  // group g: runs and windows [start[g], start[g + stride])
    uint32_t stride;                  // 1; in a sample group g is bin g * stride of the bins' prefixes
    uint32_t n_groups;
    const uint64_t* heavy_runs;               // the first n_heavy groups: sub-bins of the heavy bins (HeavyBins)
    const unsigned long long* heavy_start;
    uint32_t n_heavy, heavy_from;             // a group of more windows than that is a heavy bin, and passed over
    uint32_t k;
    uint32_t mtc;                // 0: every key seen twice is a row; else those with an edge count of mtc, the rest are low
    uint32_t* single;            // bit g: the window at base g holds a key seen once
    uint64_t* keys;
    uint64_t* tags;
    uint32_t tag_stride;
    uint32_t* cnt;
    uint64_t cap_rows;
    uint64_t* low_keys;          // NK words each
    uint64_t cap_low;
    uint64_t* later;             // two lists of later_cap runs a block (see k_bin_agg)
    uint32_t later_cap, max_blocks;
    unsigned long long* counters;
    uint32_t* status;
    FirstKey* firsts;            // AGG_FIRST: the keys (cap_rows of them)
    uint32_t* first;             // and the estimator's first touches, 4 rows of 2^log2w
    uint32_t log2w;
    uint32_t* counts;            // AGG_COUNT: the sketch's counters, 4 rows of 2^log2w
    uint32_t* hll12;             // and its p = 12 registers
};

// What a launch of k_bin_agg is for: the accumulator rows; the same, and the occurrences of the
// keys seen twice or more into a sketch that the caller keeps; the counts of a part of the
// bins, for the sizes; or the first two places of every key (the estimator's).
enum { AGG_BUILD, AGG_COUNT, AGG_SAMPLE, AGG_FIRST };

constexpr int AGG_THREADS = 512;
constexpr uint32_t AGG_SMEM = 113000;  // two blocks an SM (228 KB, 1 KB reserved a block)
constexpr uint32_t AGG_NARROW_MAX = 65535;  // windows of a group whose u16 counts cannot overflow
constexpr uint32_t AGG_QUEUE = 64 * 8;      // bytes of a warp's queue
constexpr uint32_t AGG_LATER = 16384;       // windows a block can put off, at most
constexpr uint32_t SAMPLE_WINDOWS = 4096;   // windows of a sampled bin whose keys are all counted
constexpr uint32_t AGG_TURNS = 1u << 16;    // a turn is repeated only when another lane has entered a key
constexpr uint32_t NO_PLACE = 0xFFFFFFFFu;  // AGG_FIRST; the bank holds fewer than 2^32 - 1 bases
constexpr uint32_t POS_TWICE = 0xFFFFFFFFu; // place + 1 of the key's first window otherwise, 0: no key

// A group's keys in shared memory: entries, filled one after another, of NK key words, the
// edge counts (4 words of u16 pairs, or 8 words in a group of more than 65535 windows) and
// the place of the first window; and an index of two slots an entry, a slot being 0 or the
// key's 16-bit fingerprint and entry + 1.  A free slot costs 4 bytes, not an entry, and the
// entries can be read without gaps.
__host__ __device__ constexpr uint32_t agg_entries(int nk, bool wide) {
    return (AGG_SMEM - AGG_QUEUE * (AGG_THREADS / 32)) / (8u * nk + (wide ? 36u : 20u) + 8u) & ~127u;
}

// AGG_COUNT: one word more, the windows that add nothing to the key's first side.
__host__ __device__ constexpr uint32_t count_entries(int nk, bool wide) {
    return (AGG_SMEM - AGG_QUEUE * (AGG_THREADS / 32)) / (8u * nk + (wide ? 40u : 24u) + 8u) & ~127u;
}
// AGG_FIRST: the key words, its two places and the two slots.
__host__ __device__ constexpr uint32_t first_entries(int nk) {
    return (AGG_SMEM - AGG_QUEUE * (AGG_THREADS / 32)) / (8u * nk + 16u) & ~127u;
}

// Shared memory by its 32-bit address: the parts of the table start at offsets that depend on
// the group.
__device__ __forceinline__ uint32_t sh_addr(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ uint32_t sh_ld(uint32_t a) {
    uint32_t v;
    asm volatile("ld.shared.u32 %0, [%1];" : "=r"(v) : "r"(a) : "memory");
    return v;
}
__device__ __forceinline__ uint64_t sh_ld64(uint32_t a) {
    uint64_t v;
    asm volatile("ld.shared.u64 %0, [%1];" : "=l"(v) : "r"(a) : "memory");
    return v;
}
__device__ __forceinline__ uint4 sh_ld128(uint32_t a) {
    uint4 v;
    asm volatile("ld.volatile.shared.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(a) : "memory");
    return v;
}
__device__ __forceinline__ void sh_st(uint32_t a, uint32_t v) { asm volatile("st.shared.u32 [%0], %1;" ::"r"(a), "r"(v) : "memory"); }
__device__ __forceinline__ void sh_st64(uint32_t a, uint64_t v) { asm volatile("st.shared.u64 [%0], %1;" ::"r"(a), "l"(v) : "memory"); }
__device__ __forceinline__ void sh_zero128(uint32_t a) { asm volatile("st.shared.v4.u32 [%0], {%1, %1, %1, %1};" ::"r"(a), "r"(0u) : "memory"); }
// The same under a predicate: a branch around one instruction costs six.
__device__ __forceinline__ void sh_add_if(bool on, uint32_t a, uint32_t v) {
    asm volatile("{.reg .pred p; setp.ne.u32 p, %2, 0; @p red.shared.add.u32 [%0], %1;}" ::"r"(a), "r"(v), "r"((uint32_t)on) : "memory");
}
__device__ __forceinline__ void sh_st_if(bool on, uint32_t a, uint32_t v) {
    asm volatile("{.reg .pred p; setp.ne.u32 p, %2, 0; @p st.shared.u32 [%0], %1;}" ::"r"(a), "r"(v), "r"((uint32_t)on) : "memory");
}
__device__ __forceinline__ void sh_st64_if(bool on, uint32_t a, uint64_t v) {
    asm volatile("{.reg .pred p; setp.ne.u32 p, %2, 0; @p st.shared.u64 [%0], %1;}" ::"r"(a), "l"(v), "r"((uint32_t)on) : "memory");
}
// An entry is published by the CAS of its slot (release) and read after the slot (acquire).
__device__ __forceinline__ uint32_t slot_acquire(uint32_t a) {
    uint32_t v;
    asm volatile("ld.acquire.cta.shared.u32 %0, [%1];" : "=r"(v) : "r"(a) : "memory");
    return v;
}
__device__ __forceinline__ uint32_t slot_publish(uint32_t a, uint32_t v) {
    uint32_t old;
    asm volatile("atom.release.cta.shared.cas.b32 %0, [%1], 0, %2;" : "=r"(old) : "r"(a), "r"(v) : "memory");
    return old;
}
__device__ __forceinline__ uint32_t sh_min(uint32_t a, uint32_t v) {
    uint32_t old;
    asm volatile("atom.shared.min.u32 %0, [%1], %2;" : "=r"(old) : "r"(a), "r"(v) : "memory");
    return old;
}
__device__ __forceinline__ uint32_t first_of(bool a, bool b, bool c, bool d) { return a ? 0u : b ? 1u : c ? 2u : d ? 3u : 4u; }

// n occurrences of a key into a sketch that the caller keeps, as its pass 1 adds them (the
// counters are sums, so a key's occurrences may come at once; the registers see the same keys).
// 1 Mbp at 50x, k = 31, 2^22 columns: the build with its sketch 2.7 ms over occurrences and
// records, 1.5 so.
__device__ __forceinline__ void count_key(uint32_t* counts, uint32_t log2w, uint32_t* hll12, uint64_t fold, uint32_t n) {
#pragma unroll
    for (int row = 0; row < 4; ++row) atomicAdd(counts + cms_index(fold, row, log2w), n);
    const uint64_t h = smix(fold ^ cms_seed(0));
    if (h & (PASS1_HLL_SAMPLE - 1)) return;
    uint32_t idx, rho;
    hll_idx_rho(h, 12, idx, rho);
    if (__ldca(hll12 + idx) < rho) atomicMax(hll12 + idx, rho);
}

// A block barrier that every lane of a warp reaches together (loops whose lanes leave at
// different turns come right before it).
__device__ __forceinline__ void block_sync() {
    __syncwarp();
    __syncthreads();
}

// One block per group of bins.  A warp takes up to 32 runs at a time and walks the
// concatenation of their windows, one per lane.  When the entries run out, the keys that have
// one are counted to the end, and the windows of the others are put off, as runs of one
// window, for a turn of their own after the entries have been written out: a group may hold
// more keys than expected at the price of those windows alone.  A block whose list of such
// windows overflows takes the group again in parts by a hash of the key (half the range each
// time), so any group fits in the end.
//
// A window adds 1 on its key's right side (canonical orientation) and 1 on its left side,
// unless the read ends there.  A key was seen twice iff a side adds up to 2, or a window
// without both sides found the key already there (POS_TWICE: two one-sided windows can leave
// 1 and 1), or a window without any side entered it (s_alone) and a side is not 0.
//
// Bound by instruction issue.  Slots come in buckets of four, compared at once.  Most windows
// find their key in its first bucket; the others (1 in 10 at k = 21, 1 in 3 at k = 77) go to a
// queue of the warp and are resolved 32 at a time, so that the longer searches and the
// entering of new keys run on full warps.  No lane waits for another: a new key's entry is
// complete before its slot is.
// 5 Mbp at 100x: 418 M windows of k = 21 5.2 ms, 232 M of k = 77 6.3 ms, where the records' emit,
// count and upsert took 12.7 and 15.8.  Slots probed one at a time 6.1 and 11.4 ms, four at once
// with keys in the slots 5.3 and 7.7, with entries of their own 6.5 and 6.3, and with the queue
// as it is; 1, 3 or 4 blocks an SM and other fills within 5%.
template <int NW, int WS, int MODE>
__global__ void __launch_bounds__(AGG_THREADS, 2) k_bin_agg(AggArgs A) {
    constexpr int NK = NW - WS;
    constexpr bool SAMPLE = MODE == AGG_SAMPLE, FIRST = MODE == AGG_FIRST, COUNT = MODE == AGG_COUNT;
    extern __shared__ __align__(16) uint64_t agg_smem[];
    __shared__ uint32_t s_full, s_runs, s_entries, s_later, s_warp[AGG_THREADS / 32], s_alone[agg_entries(1, false) / 32];
    __shared__ unsigned long long s_base, s_low_base, s_next[3];  // next group, its bounds
    const uint32_t lane = threadIdx.x & 31;
    const uint32_t k = A.k;
    const uint32_t queue = sh_addr(agg_smem) + (threadIdx.x >> 5) * AGG_QUEUE;
    const uint32_t* __restrict__ d32 = reinterpret_cast<const uint32_t*>(A.data);
    // A sample is launched before the host has looked whether every run was logged.  One that
    // was not leaves a hole in its bin's range, and a hole is no run: nothing of it is read.
    if (SAMPLE && A.counters[BC_NEED]) return;
    unsigned long long tot_single = 0, tot_multi = 0, tot_kept = 0;
    auto fetch = [&]() {  // thread 0: the block's next group
        const unsigned long long g = atomicAdd(&A.counters[SAMPLE ? BC_WORK_S : BC_WORK], 1ULL);
        s_next[0] = g;
        if (g < A.n_heavy) {
            s_next[1] = A.heavy_start[g];
            s_next[2] = A.heavy_start[g + 1];
        } else if (g < A.n_heavy + A.n_groups) {
            s_next[1] = A.start[(g - A.n_heavy) * A.stride];
            s_next[2] = A.start[(g - A.n_heavy) * A.stride + 1];
        }
    };
    if (threadIdx.x == 0) fetch();
    block_sync();
    while (s_next[0] < A.n_heavy + A.n_groups) {
        const unsigned long long p0 = s_next[1], p1 = s_next[2];
        const bool sub = s_next[0] < A.n_heavy;
        const uint64_t* runs = (sub ? A.heavy_runs : A.runs) + (uint32_t)(p0 >> 32);
        const uint32_t n_runs = (uint32_t)(p1 >> 32) - (uint32_t)(p0 >> 32);
        const uint32_t windows = (uint32_t)p1 - (uint32_t)p0;
        const bool wide = !FIRST && windows > AGG_NARROW_MAX;
        block_sync();  // everyone has read s_next
        if (n_runs == 0 || (!sub && windows > A.heavy_from)) {
            if (threadIdx.x == 0) fetch();
            block_sync();
            continue;
        }
        if (SAMPLE && threadIdx.x == 0) atomicAdd(&A.counters[BC_WINDOWS], (unsigned long long)windows);
        const uint32_t cap = FIRST ? first_entries(NK) : COUNT ? (wide ? count_entries(NK, true) : count_entries(NK, false))
                                                     : wide ? agg_entries(NK, true) : agg_entries(NK, false);
        const uint32_t cl = FIRST ? 0u : wide ? 3u : 2u;  // log2(words of counts per entry)
        const uint32_t n_buckets = cap / 2;
        const uint32_t ekey = sh_addr(agg_smem) + AGG_QUEUE * (AGG_THREADS / 32), ecnt = ekey + 8 * NK * cap;
        const uint32_t epos = ecnt + ((4 * cap) << cl), elack = epos + 4 * cap, slots = elack + (COUNT ? 4 * cap : 0);
        auto window_hash = [&](Window<NK>& w, uint32_t g) {
            window_at<NK>(d32, g, k, w.key, w.rc, w.left, w.right);
            w.fold = fold_of<NK>(w.key);
            const uint64_t hx = (w.fold ^ (w.fold >> 31)) * 0x9E3779B97F4A7C15ULL;
            w.bucket = __umulhi((uint32_t)(hx >> 32), n_buckets);
            w.tag = (uint32_t)hx & 0xFFFF0000u;
        };
        const uint32_t nr = wide ? 0u : 1u;
        auto count_window = [&](const Window<NK>& w, uint32_t g, uint32_t entry, bool on, bool has_l, bool has_r, bool again) {
            if constexpr (FIRST) {
                // the smaller of two places that meet stays the first, the other one is a
                // candidate for the second; one beyond the second so far is neither
                if (on && g < sh_ld(ecnt + 4 * entry)) {
                    const uint32_t other = max(g, sh_min(epos + 4 * entry, g));
                    if (other != NO_PLACE) sh_min(ecnt + 4 * entry, other);
                }
                return;
            }
            sh_st_if(on && again && !(has_l && has_r), epos + 4 * entry, POS_TWICE);
            // pushes as u (base after the window) and as v (base before it)
            const uint32_t c = ecnt + ((4 * entry) << cl);
            const uint32_t r4 = w.rc ? 4u : 0u, eu = w.right + r4, ev = (w.left ^ 3u) + (r4 ^ 4u);
            sh_add_if(on && has_r, c + 4 * (eu >> nr), 1u << ((eu & nr) << 4));
            sh_add_if(on && has_l, c + 4 * (ev >> nr), 1u << ((ev & nr) << 4));
            if constexpr (COUNT) sh_add_if(on && !(w.rc ? has_l : has_r), elack + 4 * entry, 1);
        };
        uint64_t lo = 0, width = 1ULL << 32;  // the part of the hash range being counted
        // of a sampled bin a part of the keys that fits, each for as many as there are parts
        if (SAMPLE && windows > SAMPLE_WINDOWS) width >>= 32 - __clz((windows - 1) / SAMPLE_WINDOWS);
        const uint64_t* src = runs;           // the group's runs, or the windows put off
        uint32_t n_src = n_runs;
        uint64_t* later = A.later + (uint64_t)blockIdx.x * 2 * A.later_cap;
        bool fetched = false;
        while (lo < (1ULL << 32)) {
            for (uint32_t i = threadIdx.x; i < n_buckets; i += blockDim.x) sh_zero128(slots + 16 * i);
            if (!FIRST && threadIdx.x < cap / 32) s_alone[threadIdx.x] = 0;
            if (threadIdx.x == 0) s_full = s_runs = s_entries = s_later = 0;
            block_sync();
            if (threadIdx.x == 0 && !fetched) fetch();  // in flight while the group is counted
            fetched = true;
            const bool part = width < (1ULL << 32);
            // Windows put off are looked up once more when every key of this turn has its slot:
            // a key may have been on its way in when one of its windows found no entry left.
            bool enter = true;
          again:
            // Runs are handed out as the warps get to them, up to 32 at a time and fewer towards
            // the end; the next ones are being loaded while these are counted.
            uint32_t take;
            auto grab = [&]() {
                uint32_t c = 0, t = 0;
                if (lane == 0) {
                    c = *(volatile uint32_t*)&s_runs;
                    t = min(32u, max(8u, (n_src - min(c, n_src)) / (AGG_THREADS / 32)));
                    c = *(volatile uint32_t*)&s_full ? n_src : atomicAdd(&s_runs, t);
                }
                take = __shfl_sync(0xffffffffu, t, 0);
                return __shfl_sync(0xffffffffu, c, 0);
            };
            auto load = [&](uint32_t c) { return lane < take && c + lane < n_src ? __ldcs(src + c + lane) : 0ull; };
            uint32_t c0 = grab();
            uint64_t ahead = load(c0);
            uint32_t n = 0, first = 0, shift = 0, edge_l = 0, edge_r = 0;  // this lane's run
            uint32_t total = 0, base = 0, before = 0;  // windows of the runs taken, windows done, runs that start before those
            uint32_t qn = 0;                           // windows in the warp's queue, below 32 between steps
            for (;;) {
                if (base >= total) {
                    if (c0 < n_src) {
                        const uint64_t e = ahead;
                        c0 = grab();
                        ahead = load(c0);
                        n = (uint32_t)(e >> 32) & 0xFFFu;
                        uint32_t inc = n;
#pragma unroll
                        for (int o = 1; o < 32; o <<= 1) {
                            const uint32_t y = __shfl_up_sync(0xffffffffu, inc, o);
                            if (lane >= (uint32_t)o) inc += y;
                        }
                        total = __shfl_sync(0xffffffffu, inc, 31);
                        first = inc - n;
                        // window x of the concatenation is base off + (x - first) of its run; the
                        // first and last windows of a run have a neighbour where the flags say so
                        shift = (uint32_t)e - first;
                        edge_l = (e >> 44) & 1u ? 0xFFFFFFFFu : first;
                        edge_r = (e >> 45) & 1u ? 0xFFFFFFFFu : inc - 1;
                        base = before = 0;
                    } else if (!qn) {
                        break;
                    }
                }
                if (base < total) {
                    const uint32_t rel = first - base;
                    const uint32_t starts = __reduce_or_sync(0xffffffffu, n && rel < 32 ? 1u << rel : 0u);
                    const int run = (int)(before + __popc(starts & ((2u << lane) - 1))) - 1;
                    before += __popc(starts);
                    // lanes past the last window repeat it and count nothing
                    const bool live = base + lane < total;
                    const uint32_t x = min(base + lane, total - 1);
                    base += 32;
                    const uint32_t g = __shfl_sync(0xffffffffu, shift, run) + x;
                    const bool has_l = __shfl_sync(0xffffffffu, edge_l, run) != x, has_r = __shfl_sync(0xffffffffu, edge_r, run) != x;
                    Window<NK> w;
                    window_hash(w, g);
                    const uint32_t at = slots + 16 * w.bucket;
                    const uint4 v = sh_ld128(at);
                    const uint32_t s = first_of(v.x - w.tag - 1u < 0xFFFFu, v.y - w.tag - 1u < 0xFFFFu, v.z - w.tag - 1u < 0xFFFFu,
                                                v.w - w.tag - 1u < 0xFFFFu);
                    const uint32_t named = slot_acquire(at + 4 * (s & 3u));
                    const uint32_t e = s < 4 ? (named & 0xFFFFu) - 1 : 0;
                    bool eq = s < 4;
#pragma unroll
                    for (int i = 0; i < NK; ++i) eq &= sh_ld64(ekey + 8 * (e * NK + i)) == w.key[i];
                    bool mine = live;
                    if (part) mine &= (smix(w.fold) >> 32) - lo < width;
                    count_window(w, g, e, mine && eq, has_l, has_r, true);
                    const bool miss = mine && !eq;
                    const uint32_t m = __ballot_sync(0xffffffffu, miss);
                    sh_st64_if(miss, queue + 8 * (qn + __popc(m & ((1u << lane) - 1))), run_pack(g, 1, has_l, has_r, 0));
                    qn += __popc(m);
                    __syncwarp();
                }
                if (qn >= 32 || (qn && base >= total && c0 >= n_src)) {
                    // up to 32 windows whose key was not in its first bucket: found further on,
                    // or entered
                    const uint32_t q0 = qn >= 32 ? qn - 32 : 0;
                    bool live = q0 + lane < qn, claimed = false, put_off = false;
                    const uint64_t item = sh_ld64(queue + 8 * min(q0 + lane, qn - 1));
                    const uint32_t g = (uint32_t)item;
                    const bool has_l = (item >> 44) & 1u, has_r = (item >> 45) & 1u;
                    qn = q0;
                    Window<NK> w;
                    window_hash(w, g);
                    bool open = live;
                    uint32_t from = 0, entry = 0xFFFFFFFFu, turns = 0;
                    while (__any_sync(0xffffffffu, open)) {
                        // to the key's fingerprint (from: slots of the bucket already ruled
                        // out) or to a free slot; half of the slots are free at any time
                        uint32_t slot = 0;
                        bool match = false, go = open;
                        while (go) {
                            const uint4 v = sh_ld128(slots + 16 * w.bucket);
                            const uint32_t c[4] = {v.x, v.y, v.z, v.w};
                            bool m[4];
#pragma unroll
                            for (int q = 0; q < 4; ++q) m[q] = c[q] - w.tag - 1u < 0xFFFFu && from <= (uint32_t)q;  // same high half, entry not 0
                            slot = first_of(m[0], m[1], m[2], m[3]);
                            match = slot < 4;
                            if (!match) slot = first_of(c[0] == 0, c[1] == 0, c[2] == 0, c[3] == 0);
                            go = slot == 4;
                            slot += 4 * w.bucket;
                            if (go) {
                                w.bucket = w.bucket + 1 == n_buckets ? 0 : w.bucket + 1;
                                from = 0;
                            }
                        }
                        if (open && match) {
                            const uint32_t e = (slot_acquire(slots + 4 * slot) & 0xFFFFu) - 1;
                            bool eq = true;
#pragma unroll
                            for (int i = 0; i < NK; ++i) eq &= sh_ld64(ekey + 8 * (e * NK + i)) == w.key[i];
                            if (eq) {
                                if (!FIRST && entry != 0xFFFFFFFFu) sh_st(epos + 4 * entry, 0);  // an entry made for nothing
                                entry = e;
                                open = false;
                            }
                            from = (slot & 3u) + 1;
                        }
                        // the others enter their key there
                        const bool want = open && !match && entry == 0xFFFFFFFFu;
                        const uint32_t m_want = __ballot_sync(0xffffffffu, want);
                        if (m_want && !enter) {
                            if (want) put_off = true, open = live = false;
                        } else if (m_want) {
                            uint32_t at = 0;
                            if (lane == 0) at = atomicAdd(&s_entries, (uint32_t)__popc(m_want));
                            at = __shfl_sync(0xffffffffu, at, 0) + __popc(m_want & ((1u << lane) - 1));
                            if (want) {
                                if (at < cap) {
                                    entry = at;
#pragma unroll
                                    for (int i = 0; i < NK; ++i) sh_st64(ekey + 8 * (at * NK + i), w.key[i]);
                                    if constexpr (FIRST) {
                                        sh_st(ecnt + 4 * at, NO_PLACE);
                                        sh_st(epos + 4 * at, NO_PLACE);
                                    } else {
                                        sh_zero128(ecnt + ((4 * at) << cl));
                                        if (wide) sh_zero128(ecnt + 32 * at + 16);
                                        sh_st(epos + 4 * at, g + 1);
                                        if constexpr (COUNT) sh_st(elack + 4 * at, 0);
                                    }
                                } else {
                                    put_off = true;
                                    open = live = false;
                                }
                            }
                        }
                        if (open && !match) {
                            claimed = slot_publish(slots + 4 * slot, w.tag | (entry + 1)) == 0;
                            open = !claimed;  // taken meanwhile: the bucket is looked at again
                            if (!FIRST && claimed && !has_l && !has_r) atomicOr(&s_alone[entry >> 5], 1u << (entry & 31));
                            from = 0;
                        }
                        if (++turns >= AGG_TURNS && open) {
                            atomicOr(A.status, ST_SPIN_TIMEOUT);
                            open = live = false;
                        }
                    }
                    const uint32_t m_off = __ballot_sync(0xffffffffu, put_off);
                    if (m_off) {
                        uint32_t at = 0;
                        if (lane == 0) at = atomicAdd(&s_later, (uint32_t)__popc(m_off));
                        at = __shfl_sync(0xffffffffu, at, 0) + __popc(m_off & ((1u << lane) - 1));
                        if (put_off) {
                            // (the windows of such a list fit the other one)
                            if (at < A.later_cap) later[at] = run_pack(g, 1, has_l, has_r, 0);
                            else s_full = 1;
                        }
                    }
                    count_window(w, g, entry, live, has_l, has_r, !claimed);
                    __syncwarp();
                }
            }
            block_sync();
            if (s_full) {
                block_sync();
                // from the start of this part of the group, in halves
                src = runs;
                n_src = n_runs;
                if (width == 1) {
                    // more keys of one hash value than a table holds
                    if (threadIdx.x == 0) atomicOr(A.status, ST_TABLE_FULL);
                    lo = 1ULL << 32;
                } else {
                    width >>= 1;
                }
                continue;
            }
            if (enter && s_later) {
                uint64_t* lists = A.later + (uint64_t)blockIdx.x * 2 * A.later_cap;
                src = lists;
                n_src = s_later;
                later = lists + A.later_cap;
                enter = false;
                block_sync();
                if (threadIdx.x == 0) s_runs = s_later = 0;
                block_sync();
                goto again;
            }
            const uint32_t n_entries = min(s_entries, cap), n_later = s_later;
            const unsigned long long weight = SAMPLE ? (1ULL << 32) / width : 1;
            // What becomes of entry i: 1 seen once, 2 low row, 3 row; its counts in e.
            auto counts = [&](uint32_t i, uint32_t (&e)[8]) {
                const uint4 a = sh_ld128(ecnt + ((4 * i) << cl));
                if (wide) {
                    const uint4 b = sh_ld128(ecnt + 32 * i + 16);
                    e[0] = a.x, e[1] = a.y, e[2] = a.z, e[3] = a.w, e[4] = b.x, e[5] = b.y, e[6] = b.z, e[7] = b.w;
                } else {
                    const uint32_t v[4] = {a.x, a.y, a.z, a.w};
#pragma unroll
                    for (int q = 0; q < 4; ++q) {
                        e[2 * q] = v[q] & 0xFFFFu;
                        e[2 * q + 1] = v[q] >> 16;
                    }
                }
            };
            uint32_t n_row = 0, n_low = 0, codes = 0;  // 2 bits per entry of this thread
            static_assert(agg_entries(1, false) <= 16 * AGG_THREADS, "codes hold 16 entries a thread");
            uint32_t turn = 0;
            if constexpr (FIRST) {
                if (threadIdx.x == 0) s_base = atomicAdd(&A.counters[BC_ROWS], (unsigned long long)n_entries);
                block_sync();
                for (uint32_t i = threadIdx.x; i < n_entries; i += blockDim.x) {
                    FirstKey f{0, sh_ld(epos + 4 * i), sh_ld(ecnt + 4 * i)};
                    if (f.at != NO_PLACE) {
                        f.raw = nthash_canonical_at(A.data, f.at, k);
#pragma unroll
                        for (int row = 0; row < 4; ++row) atomicMin(A.first + cms_index(f.raw, row, A.log2w), f.at);
                    }
                    if (s_base + i < A.cap_rows) A.firsts[s_base + i] = f;
                }
                block_sync();
            }
            for (uint32_t i = threadIdx.x; !FIRST && i < n_entries; i += blockDim.x, turn += 2) {
                const uint32_t pos = sh_ld(epos + 4 * i);
                if (!pos) continue;
                uint32_t e[8];
                counts(i, e);
                const uint32_t a = e[0] + e[1] + e[2] + e[3], b = e[4] + e[5] + e[6] + e[7];
                if (a < 2 && b < 2 && pos != POS_TWICE && !((a | b) && (s_alone[i >> 5] >> (i & 31) & 1u))) {
                    tot_single += weight;
                    if (!SAMPLE) atomicOr(&A.single[(pos - 1) >> 5], 1u << ((pos - 1) & 31));
                    continue;
                }
                if constexpr (COUNT) {
                    // the windows of the key: those on its first side and those that are not
                    uint64_t f = 0;
#pragma unroll
                    for (int q = 0; q < NK; ++q) f ^= sh_ld64(ekey + 8 * (i * NK + q));
                    count_key(A.counts, A.log2w, A.hll12, f, a + sh_ld(elack + 4 * i));
                }
                uint32_t m = 0;
#pragma unroll
                for (int q = 0; q < 8; ++q) m = max(m, e[q]);
                const bool low = m < A.mtc;
                n_row += !low;
                n_low += low;
                codes |= (low ? 2u : 3u) << turn;
            }
            if constexpr (SAMPLE) {
                tot_multi += (n_row + n_low) * weight;
                tot_kept += n_row * weight;
                block_sync();
            } else if constexpr (!FIRST) {
                // rows and low rows are counted, reserved once, then written
                n_row = __reduce_add_sync(0xffffffffu, n_row);
                n_low = __reduce_add_sync(0xffffffffu, n_low);
                if (lane == 0) s_warp[threadIdx.x >> 5] = n_row | (n_low << 16);  // n_entries at most in a block: both fit 16 bits
                block_sync();
                uint32_t sum = lane < AGG_THREADS / 32 ? s_warp[lane] : 0u;
                const uint32_t own = sum;
#pragma unroll
                for (int o = 1; o < 32; o <<= 1) {  // neither half overflows
                    const uint32_t y = __shfl_up_sync(0xffffffffu, sum, o);
                    if (lane >= (uint32_t)o) sum += y;
                }
                const uint32_t total = __shfl_sync(0xffffffffu, sum, 31);
                const uint32_t before = __shfl_sync(0xffffffffu, sum - own, threadIdx.x >> 5);
                if (threadIdx.x == 0) {
                    s_base = total & 0xFFFFu ? atomicAdd(&A.counters[BC_ROWS], (unsigned long long)(total & 0xFFFFu)) : 0;
                    s_low_base = total >> 16 ? atomicAdd(&A.counters[BC_LOW], (unsigned long long)(total >> 16)) : 0;
                }
                block_sync();
                uint64_t row0 = s_base + (before & 0xFFFFu), low0 = s_low_base + (before >> 16);
                for (uint32_t i = threadIdx.x; __any_sync(0xffffffffu, codes != 0); i += blockDim.x, codes >>= 2) {
                    const uint32_t what = codes & 3u;
                    const uint32_t m_row = __ballot_sync(0xffffffffu, what == 3), m_low = __ballot_sync(0xffffffffu, what == 2);
                    if (what == 3) {
                        const uint64_t o = row0 + __popc(m_row & ((1u << lane) - 1));
                        if (o < A.cap_rows) {
#pragma unroll
                            for (int q = 0; q < NW; ++q) A.keys[o * NW + q] = q < WS ? 0 : sh_ld64(ekey + 8 * (i * NK + (q >= WS ? q - WS : 0)));
                            if (NW > 2) A.tags[o * A.tag_stride] = 1;
                            uint32_t e[8];
                            counts(i, e);
                            uint4* c4 = reinterpret_cast<uint4*>(A.cnt + o * 8);
                            c4[0] = make_uint4(e[0], e[1], e[2], e[3]);
                            c4[1] = make_uint4(e[4], e[5], e[6], e[7]);
                        }
                    } else if (what == 2) {
                        const uint64_t o = low0 + __popc(m_low & ((1u << lane) - 1));
                        if (o < A.cap_low)
#pragma unroll
                            for (int q = 0; q < NK; ++q) A.low_keys[o * NK + q] = sh_ld64(ekey + 8 * (i * NK + q));
                    }
                    row0 += __popc(m_row);
                    low0 += __popc(m_low);
                }
                block_sync();
            }
            later = A.later + (uint64_t)blockIdx.x * 2 * A.later_cap;
            if (n_later) {
                src = later + A.later_cap;
                n_src = n_later;
            } else {
                src = runs;
                n_src = n_runs;
                lo = SAMPLE ? 1ULL << 32 : lo + width;
            }
        }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        tot_single += __shfl_down_sync(0xffffffffu, tot_single, o);
        tot_multi += __shfl_down_sync(0xffffffffu, tot_multi, o);
        tot_kept += __shfl_down_sync(0xffffffffu, tot_kept, o);
    }
    if (lane == 0) {
        if constexpr (SAMPLE) {
            if (tot_single + tot_multi) {
                atomicAdd(&A.counters[BC_DISTINCT], tot_single + tot_multi);
                atomicAdd(&A.counters[BC_MULTI], tot_multi);
                atomicAdd(&A.counters[BC_KEPT], tot_kept);
            }
        } else if (tot_single) {
            atomicAdd(&A.counters[BC_SINGLES], tot_single);
        }
    }
}

// ---------------------------------------------------------------------------
// The sketch (a ladder of two levels) and the gate
// ---------------------------------------------------------------------------
// The ladder in one of two layouts.  Planes: a bit per counter for the first level, then one
// for the top level; CLIMB reads the top first, which is small and saves the atomics of the
// counters that are there already.  Pairs: the two levels of a counter side by side, so that
// one atomic answers for both and nothing is read first.
// Or, where the caller keeps the sketch, its counters themselves.
struct LadderDev {
    uint32_t* bits;
    uint32_t log2w, planes;
    uint64_t top_off;  // words from a counter's first level to its top level
    uint32_t* counts;  // not null: the counters, and no ladder
    uint32_t* hll12;
};
LadderDev ladder_layout(uint32_t* bits, uint32_t log2w, bool planes) {
    return {bits, log2w, planes ? 1u : 0u, planes ? (4ULL << log2w) >> 5 : 0ULL, nullptr, nullptr};
}
struct LadderBits {
    uint32_t wd[4], mk[4];  // word and bit of the first level in the four rows
};
__device__ __forceinline__ void ladder_bits(uint64_t fold, const LadderDev& L, LadderBits& b) {
    const uint64_t wmask = (1ULL << L.log2w) - 1;
    uint64_t hr[4];
    cms_row_hashes(fold, hr);
#pragma unroll
    for (int row = 0; row < 4; ++row) {
        const uint32_t i = ((uint32_t)row << L.log2w) + (uint32_t)(hr[row] & wmask);
        b.wd[row] = i >> (4 + L.planes);
        b.mk[row] = L.planes ? 1u << (i & 31) : 1u << (2 * (i & 15));
    }
}
__device__ __forceinline__ uint32_t top_bit(const LadderDev& L, uint32_t mk) { return mk << (1 - L.planes); }
// Whether the key passes the gate: the top level is set in all four rows.
__device__ __forceinline__ bool ladder_solid(const LadderDev& L, uint64_t fold) {
    if (L.counts) {
        uint32_t c[4];
#pragma unroll
        for (int row = 0; row < 4; ++row) c[row] = __ldcg(L.counts + cms_index(fold, row, L.log2w));
        return min(min(c[0], c[1]), min(c[2], c[3])) >= 2;
    }
    LadderBits b;
    ladder_bits(fold, L, b);
    uint32_t w[4];
#pragma unroll
    for (int row = 0; row < 4; ++row) w[row] = __ldcg(L.bits + L.top_off + b.wd[row]);
    bool ok = true;
#pragma unroll
    for (int row = 0; row < 4; ++row) ok &= (w[row] & top_bit(L, b.mk[row])) != 0;
    return ok;
}

// Keys seen twice or more set their counters' top level (at 100x about 11 M of them: 0.33 ms,
// four random loads and as many atomics in L2 a key, where pass 1 went over every window: 6.5 ms
// at k = 21, 4.6 at k = 77).  Keys of STRIDE words, of which the
// last NK are read.
template <int STRIDE, int NK>
__global__ void __launch_bounds__(256) k_bin_sketch(const uint64_t* __restrict__ keys, uint64_t n, LadderDev L) {
    for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (uint64_t)gridDim.x * blockDim.x) {
        uint64_t f = 0;
#pragma unroll
        for (int q = 0; q < NK; ++q) f ^= keys[i * STRIDE + (STRIDE - NK) + q];
        LadderBits b;
        ladder_bits(f, L, b);
        uint32_t* top = L.bits + L.top_off;
        bool open[4];
#pragma unroll
        for (int row = 0; row < 4; ++row) open[row] = !(__ldcg(top + b.wd[row]) & top_bit(L, b.mk[row]));
#pragma unroll
        for (int row = 0; row < 4; ++row)
            if (open[row]) atomicOr(top + b.wd[row], top_bit(L, b.mk[row]));
    }
}

// The windows a read has, as bits over the bases (a window's bit is its first base's).
// Windows of different reads are never adjacent: k - 1 bases without one lie between.
__global__ void __launch_bounds__(256) k_bin_valid(BankDev b, uint32_t k, uint32_t* __restrict__ valid,
                                                   unsigned long long* __restrict__ lone) {
    uint32_t n_lone = 0;
    for (uint64_t r = b.r_begin + (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; r < b.r_end; r += (uint64_t)gridDim.x * blockDim.x) {
        const uint32_t len = b.len[r];
        if (len < k || !bank_keep(b, r)) continue;
        n_lone += len == k;
        uint64_t g = b.off[r];
        const uint64_t end = g + (len - k + 1);
        while (g < end) {
            const uint32_t s = (uint32_t)(g & 31);
            const uint32_t m = (uint32_t)min((uint64_t)(32 - s), end - g);
            atomicOr(&valid[g >> 5], (m == 32 ? 0xFFFFFFFFu : (1u << m) - 1) << s);
            g += m;
        }
    }
    n_lone = __reduce_add_sync(0xffffffffu, n_lone);
    if ((threadIdx.x & 31) == 0 && n_lone) atomicAdd(lone, (unsigned long long)n_lone);
}

// The three bitmaps: the windows there are, those of keys seen once, and of these the ones
// that pass the gate.  A window is solid if it is there and not one of the rest.
struct SingleMaps {
    const uint32_t* valid;
    const uint32_t* single;
    uint32_t* pass;
    uint64_t n;  // words
};
__device__ __forceinline__ uint32_t solid_word(const SingleMaps& m, uint64_t i) {
    return i < m.n ? m.valid[i] & (~m.single[i] | m.pass[i]) : 0u;  // i - 1 of word 0 wraps to a large i
}

enum { SINGLES_CLIMB, SINGLES_GATE, SINGLES_ROWS };

// The keys seen once, in bank order: a warp takes 32 words of the bitmap, lists their set
// bits in shared memory and works on 32 at a time, cutting the keys from the packed bank.
//   CLIMB: one increment of the key's counters; a key that finds all four at the top
//          already passes whatever else comes.
//   GATE:  the others ask again once every key has been counted.
//   ROWS:  those that pass next to a solid window become accumulator rows.
// Bound by lanes into L2, four a key and mode (5 Mbp at 100x: CLIMB 1.2 and GATE 0.5 ms at k = 21,
// 2.0 and 0.7 at k = 77).  Asking two rows of the gate first and the others only if those pass
// took as long.
template <int NW, int WS, int MODE>
__global__ void __launch_bounds__(256) k_singles(const uint64_t* __restrict__ data, SingleMaps M, uint32_t k, LadderDev L,
                                                 TableDev tb, uint64_t cap_rows, unsigned long long* __restrict__ n_rows) {
    __shared__ uint16_t s_list[8][1024];
    __shared__ uint32_t s_pass[8][32];
    __shared__ uint32_t s_sum;
    __shared__ unsigned long long s_base;
    const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const uint32_t* __restrict__ d32 = reinterpret_cast<const uint32_t*>(data);
    for (uint64_t blk = blockIdx.x; blk * 256 < M.n; blk += gridDim.x) {
        const uint64_t w0 = blk * 256 + warp * 32, wi = w0 + lane;
        uint32_t bits = 0;
        if (wi < M.n) {
            if (MODE == SINGLES_CLIMB) bits = M.single[wi];
            else if (MODE == SINGLES_GATE) bits = M.single[wi] & ~M.pass[wi];
            else {
                bits = M.single[wi] & M.pass[wi];
                if (bits) {
                    const uint32_t s = solid_word(M, wi);
                    bits &= (s << 1) | (s >> 1) | (solid_word(M, wi - 1) >> 31) | (solid_word(M, wi + 1) << 31);
                }
            }
        }
        uint32_t inc = __popc(bits);
        const uint32_t mine = inc;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t y = __shfl_up_sync(0xffffffffu, inc, o);
            if (lane >= (uint32_t)o) inc += y;
        }
        const uint32_t total = __shfl_sync(0xffffffffu, inc, 31);
        uint64_t row0 = 0;
        if (MODE == SINGLES_ROWS) {  // one reservation per block step
            if (threadIdx.x == 0) s_sum = 0;
            __syncthreads();
            uint32_t at = 0;
            if (lane == 0 && total) at = atomicAdd(&s_sum, total);
            __syncthreads();
            if (threadIdx.x == 0) s_base = s_sum ? atomicAdd(n_rows, (unsigned long long)s_sum) : 0;
            __syncthreads();
            row0 = s_base + __shfl_sync(0xffffffffu, at, 0);
        }
        s_pass[warp][lane] = 0;
        uint32_t o = inc - mine;
        while (bits) {
            const uint32_t b = __ffs(bits) - 1;
            bits &= bits - 1;
            s_list[warp][o++] = (uint16_t)(lane * 32 + b);
        }
        __syncwarp();
        for (uint32_t x = lane; x < total; x += 32) {
            const uint32_t at = s_list[warp][x];
            const uint32_t g = (uint32_t)(w0 * 32) + at;
            uint64_t key[NW - WS];
            bool rc;
            uint32_t bl, br;
            window_at<NW - WS>(d32, g, k, key, rc, bl, br);
            if (MODE == SINGLES_ROWS) {
                const uint64_t row = row0 + x;
                const bool sl = g > 0 && ((solid_word(M, (g - 1) >> 5) >> ((g - 1) & 31)) & 1u);
                const bool sr = (solid_word(M, (g + 1) >> 5) >> ((g + 1) & 31)) & 1u;
                const uint32_t eu = sr ? br + (rc ? 4u : 0u) : 8u, ev = sl ? (bl ^ 3u) + (rc ? 0u : 4u) : 8u;
                if (row < cap_rows) {
#pragma unroll
                    for (int q = 0; q < NW; ++q) tb.keys[row * NW + q] = q < WS ? 0 : key[q >= WS ? q - WS : 0];
                    if (NW > 2) tb.tags[row * tb.tag_stride] = 1;
                    uint32_t e[8];
#pragma unroll
                    for (int q = 0; q < 8; ++q) e[q] = (uint32_t)(eu == (uint32_t)q) + (uint32_t)(ev == (uint32_t)q);
                    uint4* c4 = reinterpret_cast<uint4*>(tb.cnt + row * 8);
                    c4[0] = make_uint4(e[0], e[1], e[2], e[3]);
                    c4[1] = make_uint4(e[4], e[5], e[6], e[7]);
                }
            } else if (MODE == SINGLES_GATE) {
                if (ladder_solid(L, fold_of<NW - WS>(key))) atomicOr(&s_pass[warp][at >> 5], 1u << (at & 31));
            } else if (L.counts) {
                count_key(L.counts, L.log2w, L.hll12, fold_of<NW - WS>(key), 1);
            } else {
                LadderBits b;
                ladder_bits(fold_of<NW - WS>(key), L, b);
                uint32_t* top = L.bits + L.top_off;
                uint32_t w[4] = {0, 0, 0, 0}, old[4];
                if (L.planes) {
#pragma unroll
                    for (int row = 0; row < 4; ++row) w[row] = __ldcg(top + b.wd[row]);
                }
#pragma unroll
                for (int row = 0; row < 4; ++row) old[row] = w[row] & b.mk[row] ? 0u : atomicOr(L.bits + b.wd[row], b.mk[row]);
                bool pass = true;
#pragma unroll
                for (int row = 0; row < 4; ++row) {
                    const bool at_top = L.planes ? (w[row] & b.mk[row]) != 0 : (old[row] & (b.mk[row] << 1)) != 0;
                    if (!at_top && (old[row] & b.mk[row])) atomicOr(top + b.wd[row], top_bit(L, b.mk[row]));
                    pass &= at_top;
                }
                if (pass) atomicOr(&s_pass[warp][at >> 5], 1u << (at & 31));
            }
        }
        __syncwarp();
        if (MODE != SINGLES_ROWS && wi < M.n) {
            const uint32_t p = s_pass[warp][lane];
            if (MODE == SINGLES_CLIMB) M.pass[wi] = p;
            else if (p) M.pass[wi] |= p;
        }
        __syncwarp();
    }
}

// Adjacent solid windows: every pair is two pushes.
__global__ void __launch_bounds__(256) k_bin_pairs(SingleMaps M, unsigned long long* __restrict__ pairs) {
    unsigned long long sum = 0;
    for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < M.n; i += (uint64_t)gridDim.x * blockDim.x) {
        const uint32_t s = solid_word(M, i);
        if (s) sum += __popc(s & ((s >> 1) | (s >> 31 ? solid_word(M, i + 1) << 31 : 0u)));
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) sum += __shfl_down_sync(0xffffffffu, sum, o);
    if ((threadIdx.x & 31) == 0 && sum) atomicAdd(pairs, sum);
}

// Rows: an edge crossed once asks the sketch for the key it leads to; a row that keeps no
// edge is dropped (its slot reads as empty).
template <int NW, int WS>
__global__ void __launch_bounds__(256) k_bin_gate(LadderDev L, uint32_t k, TableDev tb, uint64_t n) {
    constexpr int NK = NW - WS;
    const uint32_t bs = (64u * NW - 2u * k) & 63;
    const uint32_t topb = 2u * k - 2u - 64u * (NK - 1);
    const uint64_t tmask = (topb + 2 >= 64) ? ~0ULL : ((1ULL << (topb + 2)) - 1);
    for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (uint64_t)gridDim.x * blockDim.x) {
        uint4* c4 = reinterpret_cast<uint4*>(tb.cnt + i * 8);
        const uint4 a = c4[0], b = c4[1];
        const uint32_t e[8] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w};
        uint32_t once = 0, more = 0;
#pragma unroll
        for (int q = 0; q < 8; ++q) {
            once |= (uint32_t)(e[q] == 1) << q;
            more |= (uint32_t)(e[q] > 1) << q;
        }
        uint32_t left = once;
        if (once) {
            uint64_t w[NK], r[NK];
#pragma unroll
            for (int q = 0; q < NK; ++q) w[q] = tb.keys[i * NW + WS + q];
            // reverse complement of the key
#pragma unroll
            for (int q = 0; q < NK; ++q) {
                const uint64_t x = (w[q] << bs) | (bs && q + 1 < NK ? w[q + 1 < NK ? q + 1 : q] >> (64 - bs) : 0ULL);
                r[NK - 1 - q] = ~rev2(x) & field_mask(k, q);
            }
            for (uint32_t todo = once; todo; todo &= todo - 1) {
                const uint32_t q0 = __ffs(todo) - 1;
                uint64_t F[NK], R[NK];
#pragma unroll
                for (int q = 0; q < NK; ++q) {
                    F[q] = q0 < 4 ? w[q] : r[q];
                    R[q] = q0 < 4 ? r[q] : w[q];
                }
                roll_strands<NK>(F, R, q0 & 3u, topb, tmask);
                Key<NW> can;
                bool rc;
                strands_canonical<NW, WS>(F, R, can, rc);
                if (!ladder_solid(L, key_fold<NW>(can))) left &= ~(1u << q0);
            }
        }
        if (!(left | more)) {
            if (NW <= 2) tb.keys[i * NW] = tb.keys[i * NW + NW - 1] = KEY_EMPTY;
            else tb.tags[i * tb.tag_stride] = 0;
        } else if (left != once) {
            const uint32_t gone = once & ~left;
#pragma unroll
            for (uint32_t q = 0; q < 8; ++q)
                if ((gone >> q) & 1u) tb.cnt[i * 8 + q] = 0;
        }
    }
}

// The estimator's registers from its distinct keys (see bins_first).  The segment of a place:
// the last one whose first read begins there or before.
__global__ void __launch_bounds__(256) k_first_regs(const FirstKey* __restrict__ keys, uint64_t n, const uint64_t* __restrict__ off,
                                                    const uint32_t* __restrict__ first, uint32_t log2w, uint32_t p, uint32_t n_segs,
                                                    uint32_t* regs_total, uint32_t* regs_solid) {
    const uint64_t m = 1ULL << p;
    auto segment = [&](uint32_t place) {
        uint32_t lo = 0, hi = n_segs;
        while (hi - lo > 1) {
            const uint32_t mid = (lo + hi) / 2;
            if (off[2 * (6000 + 2000 * (uint64_t)(mid - 1))] <= place) lo = mid;
            else hi = mid;
        }
        return lo;
    };
    for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (uint64_t)gridDim.x * blockDim.x) {
        const FirstKey f = keys[i];
        if (f.at == NO_PLACE) continue;
        bool solid = true;
#pragma unroll
        for (int row = 0; row < 4; ++row) solid &= __ldcg(first + cms_index(f.raw, row, log2w)) < f.at;
        uint32_t idx, rho;
        hll_idx_rho(smix(f.raw), p, idx, rho);
        const uint32_t s1 = segment(f.at);
        uint32_t* rt = regs_total + s1 * m + idx;
        if (__ldca(rt) < rho) atomicMax(rt, rho);
        if (!solid && f.again == NO_PLACE) continue;
        uint32_t* rs = regs_solid + (solid ? s1 : segment(f.again)) * m + idx;
        if (__ldca(rs) < rho) atomicMax(rs, rho);
    }
}

// ---------------------------------------------------------------------------
// launchers
// ---------------------------------------------------------------------------
template <class K>
int resident_grid(K kernel, int block, size_t smem, int sms) {
    int per_sm = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, block, smem) != cudaSuccess || per_sm < 1) per_sm = 1;
    return per_sm * sms;
}

template <int NW, int WS, int MODE>
cudaError_t agg_launch(cudaStream_t st, const AggArgs& A) {
    auto kern = k_bin_agg<NW, WS, MODE>;
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)AGG_SMEM);
    if (e != cudaSuccess) return e;
    const int grid = (int)std::min<uint64_t>(A.max_blocks, std::max<uint64_t>(1, (uint64_t)A.n_heavy + A.n_groups));
    kern<<<grid, AGG_THREADS, AGG_SMEM, st>>>(A);
    return cudaGetLastError();
}
// The modes that write no rows know a key by its significant words alone.
template <int MODE>
cudaError_t agg_launch_nk(int nk, cudaStream_t st, const AggArgs& A) {
    return nk == 1 ? agg_launch<1, 0, MODE>(st, A) : nk == 2 ? agg_launch<2, 0, MODE>(st, A)
           : nk == 3 ? agg_launch<3, 0, MODE>(st, A) : agg_launch<4, 0, MODE>(st, A);
}
template <class Kern, class... Args>
cudaError_t stream_launch(cudaStream_t st, int sms, uint64_t n_threads, Kern kern, Args... args) {
    if (!n_threads) return cudaSuccess;
    const int grid = (int)std::min<uint64_t>(resident_grid(kern, 256, 0, sms), (n_threads + 255) / 256);
    kern<<<grid, 256, 0, st>>>(args...);
    return cudaGetLastError();
}
// f(NW, WS) for the key width and word shift of a launch
template <class Fn>
cudaError_t by_width(int nw, uint32_t k, Fn&& f) {
    const uint32_t ws = (64u * (uint32_t)nw - 2u * k) >> 6;
    using std::integral_constant;
#define FBK_W(A, B) f(integral_constant<int, A>{}, integral_constant<int, B>{})
    if (nw == 1) return FBK_W(1, 0);
    if (nw == 2) return ws == 0 ? FBK_W(2, 0) : FBK_W(2, 1);
    if (ws == 0) return FBK_W(4, 0);
    if (ws == 1) return FBK_W(4, 1);
    if (ws == 2) return FBK_W(4, 2);
    return FBK_W(4, 3);
#undef FBK_W
}

struct Scratch {  // device buffers of one build, freed when it ends
    fbk_ctx* c;
    std::vector<void*> p;
    char *at = nullptr, *end = nullptr;  // what is left of a block that buffers share
    // A block for buffers of `bytes` in all, rounded: a context without a pool pays for every
    // allocation (0.02 ms and more with its release).
    static uint64_t rounded(uint64_t bytes) { return (bytes + 255) & ~255ULL; }
    void share(uint64_t bytes) {
        at = (char*)dev_alloc(c, 256 + bytes);
        if (!at) return;
        p.push_back(at);
        end = at + 256 + bytes;
        at += 256;  // none of them begins where the block does
    }
    void* get(uint64_t bytes) {
        if (bytes && rounded(bytes) <= (uint64_t)(end - at)) {
            at += rounded(bytes);
            return at - rounded(bytes);
        }
        void* q = dev_alloc(c, bytes);
        if (q) p.push_back(q);
        return q;
    }
    void drop(void* q) {
        const auto it = std::find(p.begin(), p.end(), q);
        if (it == p.end()) return;  // the block's: it goes with the block
        p.erase(it);
        cudaStreamSynchronize(c->stream);
        dev_free(c, q);
    }
    ~Scratch() {
        cudaStreamSynchronize(c->stream);
        for (void* q : p) dev_free(c, q);
    }
};

}  // namespace

// Where the record buckets stay: t_solid other than 2 (the two-level ladder and the bitmap of
// keys seen once are built on it), k below 17 (runs of one or two windows), reads that
// overlap in the packed words, banks of 2^32 bases and more, and keys of four words with a
// sketch beyond 2^24 columns: with 1% errors nearly every k-mer of such a k is new, and the
// sketch updates leave the L2 (6 Mbp at 60x, 2^26 columns, 1% errors: k = 127 5.5 ms there,
// 6.5 here; at 2^24 columns 6.4 both; k = 77 14.5 there, 13.7 here).
bool bins_applicable(const fbk_ctx* ctx, const fbk_bank* b, const fbk_build_params* p, uint32_t log2w) {
    return ctx->build_form == 1 && !ctx->records_tuned && log2w <= 29 && !p->table_log2_cap && p->t_solid == 2 && p->k >= BINS_MIN_K &&
           (p->k <= 96 || log2w <= 24) && b->n_reads && b->disjoint && b->n_words * 32 < (1ULL << 32);
}

// Up to this many windows no sample is taken: rows are allocated for every window.
constexpr uint64_t BINS_SAMPLE_FROM = 4u << 20;
// Windows of a group then: as many groups as blocks are resident, of 512 to 3000 windows.  (6000
// for all: 100 reads of distinct k-mers, k = 55, 0.29 ms, 0.20 so, 0.35 over records; 3000 reads
// of 3 Mbp, k = 77, 0.36, 0.21 and 0.32; 35,000 of them 0.70, 0.51 and 0.58.)
uint64_t small_group(uint64_t windows, int sms) { return std::max<uint64_t>(512, std::min<uint64_t>(3000, windows / (2 * (uint64_t)sms))); }

namespace {

// The reads' runs by bin.
struct BinRuns {
    MinPlan mp;
    uint32_t F = 64;                              // bins, about 1500 windows each
    unsigned long long *hist = nullptr, *counters = nullptr;  // the caller's, cleared with it
    unsigned long long* pre = nullptr;            // (runs << 32 | windows) before each bin
    uint64_t* runs = nullptr;
    uint64_t n_windows = 0;
    bool est = false;  // of an estimate: timed under its names
    // The warps of k_bin_runs and the runs a warp's log holds.
    uint64_t n_blocks = 0, cap_w = 0;
    BinRuns(uint32_t k, uint64_t windows, uint64_t n_reads, uint32_t max_len, int sms) : mp(min_plan(k)) {
        while (F < RUN_MAX_BINS && (uint64_t)F * 1500 < windows) F <<= 1;
        const uint64_t max_warps = (uint64_t)resident_grid(k_bin_runs, 256, 0, sms) * 8;
        n_blocks = std::max<uint64_t>(1, std::min<uint64_t>(max_warps, n_reads) / 8);
        // a run holds about (w + 1) / 2 windows, and one more ends with every read
        cap_w = (uint64_t)(1.3 * ((2.0 * windows) / (mp.w + 1) + n_reads) / (8 * n_blocks)) + 128 + std::min<uint64_t>(max_len / 4, 2048);
        // and at most one with every window of the longest reads
        cap_w = std::min<uint64_t>(cap_w, (n_reads / (8 * n_blocks) + 1) * (max_len >= k ? max_len - k + 1 : 1));
    }
    // What bin_runs needs, but for the two logs and with them.
    uint64_t bytes(bool logs) const {
        return Scratch::rounded(8ULL * (F + 1 + (F + SCAN_TILE - 1) / SCAN_TILE)) + Scratch::rounded(4ULL * F) + Scratch::rounded(32 * n_blocks) +
               (logs ? 2 * Scratch::rounded(64 * n_blocks * cap_w) : 0);
    }
};

// Cuts the reads of bv into runs (windows: no fewer than they hold) and scatters them by bin;
// with a sample, counts the keys of some bins.  The counters and n_windows are on the host
// then, in ctx->h_pinned.  Clears the caller's block and the context's status first.
fbk_status bin_runs(fbk_ctx* ctx, Scratch& B, BinRuns& R, const BankDev& bv, uint32_t k, uint64_t windows, char* cleared, uint64_t clear_bytes,
                    AggArgs* sample, bool* declined) {
    const MinPlan mp = R.mp;
    const uint32_t F = R.F;
    const int sms = ctx->num_sms;
    const cudaStream_t stream = ctx->stream;
    R.pre = (unsigned long long*)B.get(8ULL * (F + 1 + (F + SCAN_TILE - 1) / SCAN_TILE));
    uint32_t* cursor = (uint32_t*)B.get(4ULL * F);
    if (!R.pre || !cursor) return set_err(ctx, FBK_ERR_OOM, "minimizer bins");
    unsigned long long* part = R.pre + F + 1;
    const uint64_t n_blocks = R.n_blocks, n_warps = 8 * n_blocks;
    uint64_t cap_w = R.cap_w;
    uint32_t* log_n = (uint32_t*)B.get(4 * n_warps);
    if (!log_n) return set_err(ctx, FBK_ERR_OOM, "minimizer bins");
    unsigned long long* h = (unsigned long long*)ctx->h_pinned;
    uint64_t* log = nullptr;
    for (int attempt = 0;; ++attempt) {
        log = (uint64_t*)B.get(8 * n_warps * cap_w);
        R.runs = (uint64_t*)B.get(8 * n_warps * cap_w);
        if (!log || !R.runs) return set_err(ctx, FBK_ERR_OOM, "minimizer bins: runs");
        CK(ctx, cudaMemsetAsync(cleared, 0, clear_bytes, stream));
        CK(ctx, cudaMemsetAsync(ctx->d_status, 0, 4, stream));
        TIMED(ctx, R.est ? "est_runs" : "bins_runs",
              (k_bin_runs<<<(unsigned)n_blocks, 256, 0, stream>>>(bv, k, mp, F, log, log_n, (uint32_t)cap_w, R.hist, R.counters + BC_NEED),
               cudaGetLastError()));
        const unsigned tiles = (F + SCAN_TILE - 1) / SCAN_TILE;
        TIMED(ctx, R.est ? "est_scan" : "bins_scan", (k_bin_scan_sums<<<tiles, 256, 0, stream>>>(R.hist, F, part), cudaGetLastError()));
        TIMED(ctx, R.est ? "est_scan" : "bins_scan", (k_bin_scan<<<tiles, 256, 0, stream>>>(R.hist, F, part, R.pre, cursor, R.counters + BC_BIG), cudaGetLastError()));
        TIMED(ctx, R.est ? "est_scatter" : "bins_scatter",
              (k_bin_scatter<<<(unsigned)n_blocks, 256, 0, stream>>>(log, log_n, (uint32_t)cap_w, cursor, R.runs, n_warps * cap_w),
               cudaGetLastError()));
        if (sample) {
            sample->runs = R.runs;
            sample->n_groups = std::min<uint32_t>(F, 1024);
            sample->stride = F / sample->n_groups;
            sample->start = R.pre;
            sample->heavy_from = 1u << 18;  // (1 ms of a block's time)
            TIMED(ctx, R.est ? "est_sample" : "bins_sample", agg_launch_nk<AGG_SAMPLE>((int)((k + 31) / 32), stream, *sample));
        }
        CK(ctx, cudaMemcpyAsync(h, R.counters, 8 * BC_N, cudaMemcpyDeviceToHost, stream));
        CK(ctx, cudaMemcpyAsync(h + BC_N, R.pre + F, 8, cudaMemcpyDeviceToHost, stream));
        CK(ctx, cudaStreamSynchronize(stream));
        R.n_windows = h[BC_N] & 0xFFFFFFFFull;
        if (!h[BC_NEED]) break;
        // a warp's log was too short: once more with room for the longest, unless a few reads
        // are so much longer than the rest that the logs of all warps would take gigabytes
        if (attempt == 1 || h[BC_NEED] * n_warps > 4 * windows + (64ULL << 20)) {
            *declined = true;
            return FBK_OK;
        }
        cap_w = h[BC_NEED];
        B.drop(log);
        B.drop(R.runs);
    }
    B.drop(log);
    return FBK_OK;
}

// Windows of a group of bins whose keys about fill 0.7 of the entries; no more than 20,000, as
// very deep banks (a key in many of the windows that are in flight is entered many times) need
// more room than that: 30 kb at 2000x, k = 21, with up to 60,000 2.3 ms, so 1.5 (12,000 1.5, 8000
// 1.5; 5 Mbp at 100x 10.8, 10.8, 11.1, 11.5).
uint64_t group_windows(uint32_t entries, uint64_t n_windows, uint64_t distinct) {
    const uint64_t t = (uint64_t)(0.7 * (double)entries * (double)std::max<uint64_t>(n_windows, 1) / (double)std::max<uint64_t>(distinct, 1));
    return std::max<uint64_t>(512, std::min<uint64_t>(t, 20000));
}

// The heavy bins' windows by sub-bin, for groups of `target` windows; A then takes them first and
// passes their bins over.  h: the counters on the host.  Where there is no memory for it, A
// keeps the bins as they are.
fbk_status split_heavy(fbk_ctx* ctx, Scratch& B, const BinRuns& R, const unsigned long long* h, uint64_t target, uint64_t at_least,
                       AggArgs& A) {
    A.n_heavy = 0;
    A.heavy_from = 0xFFFFFFFFu;
    // a group of ordinary bins stays below three targets (k_bin_groups)
    const uint32_t from = (uint32_t)std::max<uint64_t>(3 * target, at_least);
    // the windows in bins above 2^13, 2^15 or 2^17: no fewer than the heavy bins', as `from` is no less
    const uint64_t windows = h[BC_BIG + (from >= 1u << 17 ? 2 : from >= 1u << 15 ? 1 : 0)];
    if (!windows) return FBK_OK;
    const cudaStream_t stream = ctx->stream;
    const uint32_t cap = (uint32_t)(windows / HEAVY_PIECE + windows / from + 1), n_sub = (uint32_t)(windows / target + windows / from + 1);
    const uint32_t tiles = (n_sub + SCAN_TILE - 1) / SCAN_TILE;
    HeavyPiece* pieces = (HeavyPiece*)B.get(sizeof(HeavyPiece) * cap);
    unsigned long long* hist = (unsigned long long*)B.get(8ULL * (n_sub + 1));  // and the two counts
    unsigned long long* pre = (unsigned long long*)B.get(8ULL * (n_sub + 1 + tiles));
    uint32_t* cursor = (uint32_t*)B.get(4ULL * n_sub);
    uint64_t* runs = (uint64_t*)B.get(8 * windows);
    if (!pieces || !hist || !pre || !cursor || !runs) return FBK_OK;
    uint32_t* counts = (uint32_t*)(hist + n_sub);
    CK(ctx, cudaMemsetAsync(hist, 0, 8ULL * (n_sub + 1), stream));
    auto split = [&](auto put) {
        constexpr bool PUT = decltype(put)::value;
        auto launch = [&](auto nk) {
            auto kern = k_heavy_split<decltype(nk)::value, PUT>;
            kern<<<(unsigned)std::min<uint64_t>(resident_grid(kern, 256, 0, ctx->num_sms), cap), 256, 0, stream>>>(
                A.data, R.runs, pieces, counts, cap, A.k, hist, cursor, runs, windows);
            return cudaGetLastError();
        };
        using std::integral_constant;
        const uint32_t nk = (A.k + 31) / 32;
        return nk == 1 ? launch(integral_constant<int, 1>{}) : nk == 2 ? launch(integral_constant<int, 2>{})
               : nk == 3 ? launch(integral_constant<int, 3>{}) : launch(integral_constant<int, 4>{});
    };
    TIMED(ctx, R.est ? "est_heavy" : "bins_heavy",
          (k_heavy_pieces<<<std::min<unsigned>(1024, (R.F + 255) / 256), 256, 0, stream>>>(R.pre, R.F, (uint32_t)target, from, pieces, cap, counts),
           cudaGetLastError()));
    TIMED(ctx, R.est ? "est_heavy" : "bins_heavy", split(std::false_type{}));
    TIMED(ctx, R.est ? "est_heavy" : "bins_heavy", (k_bin_scan_sums<<<tiles, 256, 0, stream>>>(hist, n_sub, pre + n_sub + 1), cudaGetLastError()));
    TIMED(ctx, R.est ? "est_heavy" : "bins_heavy",
          (k_bin_scan<<<tiles, 256, 0, stream>>>(hist, n_sub, pre + n_sub + 1, pre, cursor, nullptr), cudaGetLastError()));
    TIMED(ctx, R.est ? "est_heavy" : "bins_heavy", split(std::true_type{}));
    A.heavy_runs = runs;
    A.heavy_start = pre;
    A.n_heavy = n_sub;
    A.heavy_from = from;
    return FBK_OK;
}

}  // namespace

fbk_status bins_build(fbk_ctx* ctx, const fbk_bank* b, const fbk_build_params* p, const uint64_t* keep_bits, uint32_t log2w, fbk_cms* cms,
                      fbk_table** out, bool* declined, uint64_t* kmers) {
    *declined = false;
    if (p->min_trans_cov > 0xFFFF) return set_err(ctx, FBK_ERR_INVALID, "thresholds must fit u16");
    const int nw = key_words(p->key_bits);
    const uint32_t k = p->k;
    const int nk = nw - (int)((64u * (uint32_t)nw - 2u * k) >> 6);
    const uint64_t windows = b->windows(k, k);  // upper bound (subsampling keeps fewer)
    const bool sampled = windows > BINS_SAMPLE_FROM;
    const int sms = ctx->num_sms;
    const cudaStream_t stream = ctx->stream;
    Scratch B{ctx, {}};
    BinRuns R(k, windows, b->n_reads, b->max_len, sms);
    const uint32_t F = R.F;
    // one cleared block: the ladder, the bin and build counters, the windows' bitmaps
    const uint64_t bm_words = (b->n_words + 63) & ~63ULL;
    const uint64_t lad_bytes = cms ? 0 : (2 * (4ULL << log2w) / 8 + 255) & ~255ULL;
    const uint64_t clear_bytes = lad_bytes + 8ULL * F + 8 * 16 + 2 * 4 * bm_words;
    static_assert(BC_N <= 16, "build counters");
    const uint64_t small = small_group(windows, sms);
    AggArgs A{};
    A.later_cap = sampled ? AGG_LATER : (uint32_t)std::min<uint64_t>(4096, 2 * small);
    A.max_blocks = (uint32_t)(sampled ? 2 * sms : std::min<uint64_t>(2 * sms, windows / small + 1));
    const uint64_t later_bytes = 16ULL * A.later_cap * A.max_blocks;
    // (a sampled build's logs go before its rows come)
    B.share(Scratch::rounded(clear_bytes) + Scratch::rounded(4 * bm_words) + Scratch::rounded(later_bytes) + R.bytes(!sampled) +
            (sampled ? 0 : Scratch::rounded(8 * (windows / small + 2))));
    char* cleared = (char*)B.get(clear_bytes);
    uint32_t* pass = (uint32_t*)B.get(4 * bm_words);
    if (!cleared || !pass) return set_err(ctx, FBK_ERR_OOM, "minimizer bins");
    uint32_t* lad = (uint32_t*)cleared;
    R.hist = (unsigned long long*)(cleared + lad_bytes);
    unsigned long long* counters = R.counters = R.hist + F;
    uint32_t* single = (uint32_t*)(counters + 16);
    uint32_t* valid = single + bm_words;
    const BankDev bv = bank_view(b, 0, b->n_reads, keep_bits);
    A.data = b->data;
    A.k = k;
    A.single = single;
    A.counters = counters;
    A.status = ctx->d_status;
    A.later = (uint64_t*)B.get(later_bytes);
    if (!A.later) return set_err(ctx, FBK_ERR_OOM, "minimizer bins");
    unsigned long long* h = (unsigned long long*)ctx->h_pinned;
    const bool may_filter = p->min_trans_cov >= 2 && ctx->acc_filter != 0;
    A.mtc = may_filter ? p->min_trans_cov : 0;
    fbk_status rs = bin_runs(ctx, B, R, bv, k, windows, cleared, clear_bytes, sampled ? &A : nullptr, declined);
    if (rs || *declined) return rs;
    const uint64_t n_windows = R.n_windows;
    uint64_t* runs = R.runs;
    unsigned long long* pre = R.pre;
    uint64_t distinct = n_windows, multi = n_windows, kept = n_windows;  // upper bounds without a sample
    bool filter = may_filter && (ctx->acc_filter == 2 || nw == 4);
    if (sampled && h[BC_WINDOWS]) {
        // Where most k-mers are new a key of three words and more costs here, entered, sketched
        // and asked for once, what it costs over records or more.  Records / here by the share of
        // distinct windows, 2 and 20 Mbp, 0.1-5% errors: k = 127 0.50 1.25, 0.61 1.10, 0.73 0.95,
        // 0.83 0.87, 0.92 0.74, 1.0 0.61-0.69; k = 101 0.64 1.07, 0.74 1.02, 0.83 0.94-1.01, 0.93
        // 0.76-0.82; k = 91 0.69 1.14, 0.79 1.01-1.14, 0.87 0.96, 0.91 0.81, 1.0 0.67-1.09.  (What is
        // done by here is a tenth to a quarter of the build over records.)
        const double share = (double)h[BC_DISTINCT] / (double)h[BC_WINDOWS];
        *declined = nk >= 3 && share > (k > 96 ? 0.75 : 0.85);
        if (*declined) return FBK_OK;
        const double scale = (double)n_windows / (double)h[BC_WINDOWS];
        auto est = [&](int c) { return std::min<uint64_t>(n_windows, (uint64_t)(1.1 * scale * (double)h[c]) + 65536); };
        distinct = est(BC_DISTINCT);
        multi = est(BC_MULTI);
        kept = est(BC_KEPT);
        filter = may_filter && acc_filter_on(ctx->acc_filter, nw, distinct, n_windows);
    }
    const uint64_t target =
        sampled ? group_windows(cms ? count_entries(nk, false) : agg_entries(nk, false), n_windows, distinct) : small;
    const uint32_t n_groups = (uint32_t)(n_windows / target + 1);
    unsigned long long* start = (unsigned long long*)B.get(8ULL * (n_groups + 1));
    if (!start) return set_err(ctx, FBK_ERR_OOM, "minimizer bins: groups");
    A.runs = runs;
    rs = split_heavy(ctx, B, R, h, target, sampled ? HEAVY_FROM : 2 * HEAVY_FROM, A);
    if (rs) return rs;
    fbk_table* tb = new fbk_table();
    tb->ctx = ctx;
    tb->nw = (uint32_t)nw;
    tb->k = k;
    tb->min_trans_cov = p->min_trans_cov;
    tb->filtered = filter;
    struct TableGuard {
        fbk_table* t;
        ~TableGuard() {
            if (!t) return;
            cudaStreamSynchronize(t->ctx->stream);
            tbl_free_storage(t);
            tbl_free_out(t);
            delete t;
        }
    } guard{tb};
    // (a sketch that the caller keeps takes the low keys where they are counted)
    uint64_t rows = (filter ? kept : distinct) + 1, lows = filter && !cms ? multi + 1 : 0;
    if (cms) {
        A.counts = cms->cnt;
        A.hll12 = cms->hll12;
        A.log2w = log2w;
    }
    uint64_t* low = nullptr;
    for (int attempt = 0;; ++attempt) {
        // a table of the rows alone: every slot that is read is one, no probing
        tb->cap = rows;
        const uint64_t key_bytes = Scratch::rounded(rows * 8 * nw), tag_bytes = nw > 2 && !tag_in_key((uint32_t)nw, k) ? Scratch::rounded(rows * 8) : 0;
        tb->keys = (uint64_t*)dev_alloc(ctx, key_bytes + tag_bytes + rows * 32);
        tb->one_block = true;
        if (tb->keys) {
            if (nw > 2) tb->tags = tb->keys + (tag_bytes ? key_bytes / 8 : 0);
            tb->cnt = (uint32_t*)((char*)tb->keys + key_bytes + tag_bytes);
        }
        if (lows) low = (uint64_t*)B.get(lows * 8 * nk);
        if (!tb->keys || (lows && !low)) return set_err(ctx, FBK_ERR_OOM, "solid table rows");
        const TableDev td = tbl_dev(tb);
        A.start = start;
        A.stride = 1;
        A.n_groups = n_groups;
        A.mtc = filter ? p->min_trans_cov : 0;
        A.keys = td.keys;
        A.tags = td.tags;
        A.tag_stride = td.tag_stride;
        A.cnt = td.cnt;
        A.cap_rows = rows;
        A.low_keys = low;
        A.cap_low = lows;
        TIMED(ctx, "bins_groups",
              (k_bin_groups<<<std::min<unsigned>(1024, (F + 256) / 256), 256, 0, stream>>>(pre, F, (uint32_t)target, n_groups, start),
               cudaGetLastError()));
        TIMED(ctx, "bins_aggregate", by_width(nw, k, [&](auto a, auto w) {
                  constexpr int NW = decltype(a)::value, WS = decltype(w)::value;
                  return cms ? agg_launch<NW, WS, AGG_COUNT>(stream, A) : agg_launch<NW, WS, AGG_BUILD>(stream, A);
              }));
        CK(ctx, cudaMemcpyAsync(h, counters, 8 * BC_N, cudaMemcpyDeviceToHost, stream));
        CK(ctx, cudaMemcpyAsync(h + BC_N, ctx->d_status, 4, cudaMemcpyDeviceToHost, stream));
        CK(ctx, cudaStreamSynchronize(stream));
        // Keys that no hash tells apart (more of one fold and one minimizer than a block holds and
        // puts off), a bounded search that gave up: the record buckets' table takes them.
        *declined = (uint32_t)h[BC_N] != 0;
        if (*declined) return FBK_OK;
        const uint64_t need = h[BC_ROWS] + (filter ? 0 : h[BC_SINGLES]);
        if (need <= rows && (cms || h[BC_LOW] <= lows)) break;
        // the sample's estimate was low: again with the counted sizes
        *declined = attempt == 1;
        if (*declined) return FBK_OK;
        tbl_free_storage(tb);
        if (low) B.drop(low);
        rows = need + 1;
        lows = filter && !cms ? h[BC_LOW] + 1 : 0;
        if (cms) {
            fbk_status st = fbk_cms_clear(cms);
            if (st) return st;
        }
        CK(ctx, cudaMemsetAsync(counters, 0, 8 * BC_N, stream));
        CK(ctx, cudaMemsetAsync(single, 0, 4 * bm_words, stream));
    }
    const uint64_t n_rows = h[BC_ROWS], n_low = cms ? 0 : h[BC_LOW], n_singles = h[BC_SINGLES];
    // Without a sample the distinct keys are known only now: the filter then leaves out the keys
    // seen once, which are no rows yet (20,000 reads of 3 Mbp, k = 31: 0.50 ms with them, 0.46
    // without, as over records)
    if (!sampled && !filter && may_filter) filter = tb->filtered = acc_filter_on(ctx->acc_filter, nw, n_rows + n_singles, n_windows);
    const TableDev td = tbl_dev(tb);
    const SingleMaps maps{valid, single, pass, b->n_words};
    LadderDev ladder = ladder_layout(lad, log2w, n_singles > 2ULL << log2w);
    if (cms) ladder.counts = cms->cnt, ladder.hll12 = cms->hll12;
    auto singles = [&](int mode) {
        return by_width(nw, k, [&](auto a, auto w) {
            constexpr int NW = decltype(a)::value, WS = decltype(w)::value;
            auto kern = mode == SINGLES_CLIMB ? k_singles<NW, WS, SINGLES_CLIMB>
                        : mode == SINGLES_GATE ? k_singles<NW, WS, SINGLES_GATE> : k_singles<NW, WS, SINGLES_ROWS>;
            return stream_launch(stream, sms, b->n_words, kern, (const uint64_t*)b->data, maps, k, ladder, td, rows, counters + BC_ROWS);
        });
    };
    TIMED(ctx, "bins_valid", stream_launch(stream, sms, b->n_reads, k_bin_valid, bv, k, valid, counters + BC_LONE));
    if (!cms) {
        TIMED(ctx, "bins_sketch", by_width(nw, k, [&](auto a, auto w) {
                  constexpr int NW = decltype(a)::value, NK = NW - decltype(w)::value;
                  return stream_launch(stream, sms, n_rows, k_bin_sketch<NW, NK>, (const uint64_t*)td.keys, n_rows, ladder);
              }));
        TIMED(ctx, "bins_sketch", by_width(nw, k, [&](auto a, auto w) {
                  constexpr int NK = decltype(a)::value - decltype(w)::value;
                  return stream_launch(stream, sms, n_low, k_bin_sketch<NK, NK>, (const uint64_t*)low, n_low, ladder);
              }));
    }
    TIMED(ctx, "bins_singles", singles(SINGLES_CLIMB));
    TIMED(ctx, "bins_singles_gate", singles(SINGLES_GATE));
    TIMED(ctx, "bins_gate", by_width(nw, k, [&](auto a, auto w) {
              return stream_launch(stream, sms, n_rows, k_bin_gate<decltype(a)::value, decltype(w)::value>, ladder, k, td,
                                   n_rows);
          }));
    if (!filter && n_singles) TIMED(ctx, "bins_single_rows", singles(SINGLES_ROWS));
    TIMED(ctx, "bins_pairs", stream_launch(stream, sms, b->n_words, k_bin_pairs, maps, counters + BC_PAIRS));
    CK(ctx, cudaMemcpyAsync(h, counters, 8 * BC_N, cudaMemcpyDeviceToHost, stream));
    CK(ctx, cudaStreamSynchronize(stream));
    const uint64_t pushes = 2 * h[BC_PAIRS];
    if (kmers) *kmers = 2 * n_windows - h[BC_LONE];  // pass 2 leaves out the reads of one window
    tb->cap = h[BC_ROWS];
    // rows of the conversion: a subset of those with an edge count of min_trans_cov
    const uint64_t oc = std::min<uint64_t>(tb->cap, kept) + 16;
    tb->out_keys = (uint64_t*)dev_alloc(ctx, oc * (8 * nw + 2 + 1));
    tb->out_one_block = true;
    if (!tb->out_keys) return set_err(ctx, FBK_ERR_OOM, "solid table output");
    tb->out_cov = (uint16_t*)(tb->out_keys + oc * nw);
    tb->out_mask = (uint8_t*)(tb->out_cov + oc);
    tb->out_cap = oc;
    if (cms) TIMED(ctx, "cms_clamp", launch_clamp_counters(launch_cfg(ctx, 256, 0), cms->cnt, cms->n));
    fbk_status st = tbl_convert(tb);
    if (st) return st;
    // the pushes of the keys that the filter left out
    tb->skipped_pushes = pushes - tb->pushes;
    tb->pushes = pushes;
    guard.t = nullptr;
    *out = tb;
    return FBK_OK;
}

// The estimator's sample loop over distinct k-mers.  Of a k-mer's occurrences only the first
// two say anything: the first touches its four counters earliest and is solid iff each was
// touched before (by another k-mer), and every later one is solid, as the first has touched
// them; a register takes the k-mer's hash from its first occurrence and its solid one from the
// first that is solid.  So the bins give each key's first two places, the first touches are
// the minimum over the keys, and the registers follow from the keys.
//
// Adds the reads [0, n_reads) to first and to the segments' registers (not yet prefixed),
// which may hold what earlier rounds put there: minima and maxima of a part of the same
// values.  Declined, with nothing spoilt, where memory is short or more than 0.4 of the windows
// (0.3 for keys of several words) are distinct: a distinct key costs four random atomics and four random loads here and a
// window about as much in the loop over occurrences (39 M windows of a 5 Mbp genome, k = 21,
// 0.23 distinct: 2.0 ms here, 3.15 there; 36 M, k = 31, 0.41: 2.7 and 2.9; 30 M, k = 51, 0.39:
// 2.8 and 2.4).
fbk_status bins_first(fbk_ctx* ctx, const fbk_bank* b, uint64_t n_reads, uint64_t windows, uint32_t k, uint32_t* first, uint32_t log2w,
                      uint32_t p, uint32_t n_segs, uint32_t* regs_total, uint32_t* regs_solid, bool* declined) {
    *declined = true;
    const int nk = (int)((k + 31) / 32), sms = ctx->num_sms;
    const cudaStream_t stream = ctx->stream;
    Scratch B{ctx, {}};
    BinRuns R(k, windows, n_reads, b->max_len, sms);
    R.est = true;
    const uint64_t clear_bytes = 8ULL * R.F + 8 * 16;
    char* cleared = (char*)B.get(clear_bytes);
    AggArgs A{};
    A.data = b->data;
    A.k = k;
    A.status = ctx->d_status;
    A.later_cap = AGG_LATER;
    A.max_blocks = 2 * (uint32_t)sms;
    A.later = (uint64_t*)B.get(16ULL * A.later_cap * A.max_blocks);
    if (!cleared || !A.later) return FBK_OK;
    R.hist = (unsigned long long*)cleared;
    A.counters = R.counters = R.hist + R.F;
    unsigned long long* h = (unsigned long long*)ctx->h_pinned;
    bool no = false;
    fbk_status st = bin_runs(ctx, B, R, bank_view(b, 0, n_reads, nullptr), k, windows, cleared, clear_bytes, &A, &no);
    if (st == FBK_ERR_OOM || no) return FBK_OK;
    if (st) return st;
    const uint64_t n_windows = R.n_windows;
    const double share = h[BC_WINDOWS] ? (double)h[BC_DISTINCT] / (double)h[BC_WINDOWS] : 1.0;
    if (share > (nk == 1 ? 0.4 : 0.3)) return FBK_OK;
    const uint64_t distinct = std::min<uint64_t>(n_windows, (uint64_t)(1.1 * share * (double)n_windows) + 65536);
    const uint64_t target = group_windows(first_entries(nk), n_windows, distinct);
    A.runs = R.runs;
    A.stride = 1;
    A.n_groups = (uint32_t)(n_windows / target + 1);
    unsigned long long* start = (unsigned long long*)B.get(8ULL * (A.n_groups + 1));
    A.first = first;
    A.log2w = log2w;
    // Entries made for nothing come on top: a key is entered once for every warp that meets it
    // before the first one's slot is published (1400 reads of 7.5 kb, k = 21: a third of the keys;
    // 300,000 reads of 150: a fifth).  The groups' fill leaves them 1 / 0.7 of the keys' room.
    A.cap_rows = distinct + distinct / 2;
    A.firsts = (FirstKey*)B.get(A.cap_rows * sizeof(FirstKey));
    if (!start || !A.firsts) return FBK_OK;
    A.start = start;
    st = split_heavy(ctx, B, R, h, target, HEAVY_FROM, A);
    if (st) return st;
    TIMED(ctx, "est_groups", (k_bin_groups<<<std::min<unsigned>(1024, (R.F + 256) / 256), 256, 0, stream>>>(R.pre, R.F, (uint32_t)target,
                                                                                                          A.n_groups, start),
                               cudaGetLastError()));
    TIMED(ctx, "est_first_keys", agg_launch_nk<AGG_FIRST>(nk, stream, A));
    CK(ctx, cudaMemcpyAsync(h, A.counters, 8 * BC_N, cudaMemcpyDeviceToHost, stream));
    CK(ctx, cudaMemcpyAsync(h + BC_N, ctx->d_status, 4, cudaMemcpyDeviceToHost, stream));
    CK(ctx, cudaStreamSynchronize(stream));
    if ((uint32_t)h[BC_N] || h[BC_ROWS] > A.cap_rows) return FBK_OK;
    TIMED(ctx, "est_first_regs", stream_launch(stream, sms, h[BC_ROWS], k_first_regs, (const FirstKey*)A.firsts, (uint64_t)h[BC_ROWS],
                                               (const uint64_t*)b->off, (const uint32_t*)first, log2w, p, n_segs, regs_total, regs_solid));
    *declined = false;
    return FBK_OK;
}

}  // namespace fbk
