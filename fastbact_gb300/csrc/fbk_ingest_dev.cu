// fbk_ingest_dev.cu — ingest_reads_ext_with_seed (src/ingest/trim_merge.rs:307-417) on
// the device: the two FASTQ files' bytes in, a device ReadBank out.
//
//   1. line index: a thread counts the newlines of 16 bytes, a block those of a 4 KiB
//      chunk; after a prefix over the chunks each block writes its newlines' positions;
//   2. records: line 4r is the header of record r, 4r+1 its sequence, 4r+3 its
//      qualities (plain 4-line FASTQ, the form the host reader and the generator use;
//      a trailing '\r' is dropped from every line);
//   3. one warp per pair applies the subsampler, adapter and quality trimming and
//      the overlap merge (trim_merge.rs:17-238) and records what the pair becomes;
//   4. after a prefix over tiles of pairs, one warp per pair writes its reads' 2-bit
//      codes (ASCII_TO_2BIT, bitseq.rs:67-81) into the arenas (merged, pe_forward,
//      pe_reverse), concatenated as a device bank.
// The result equals the host ingest byte for byte (tests compare the banks).
#include <algorithm>
#include <cerrno>
#include <cstring>
#include <vector>

#include <sys/stat.h>
#include <unistd.h>

#include "fbk_device.cuh"
#include "fbk_internal.h"

using namespace fbk;

namespace {

constexpr uint32_t CHUNK = 4096;

// The 16 bytes at i, newline beyond the end of the text masked off: one bit each.  The text's
// allocation reaches past its end to the next 16 bytes.
__device__ __forceinline__ uint32_t nl_bits(const uint8_t* __restrict__ t, uint64_t n, uint64_t i) {
    if (i >= n) return 0;
    const uint4 v = *reinterpret_cast<const uint4*>(t + i);
    const uint32_t w[4] = {v.x, v.y, v.z, v.w};
    uint32_t m = 0;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        const uint32_t e = __vcmpeq4(w[j], 0x0A0A0A0Au);  // 0xFF per newline
        m |= (((e & 0x08040201u) * 0x01010101u) >> 24) << (4 * j);
    }
    return n - i < 16 ? m & ((1u << (n - i)) - 1) : m;
}

__global__ void __launch_bounds__(256) k_nl_count(const uint8_t* __restrict__ t, uint64_t n, uint32_t* cnt) {
    __shared__ uint32_t s_warp[8];
    const uint32_t m = __reduce_add_sync(0xffffffffu, (uint32_t)__popc(nl_bits(t, n, (uint64_t)blockIdx.x * CHUNK + threadIdx.x * 16)));
    if ((threadIdx.x & 31) == 0) s_warp[threadIdx.x >> 5] = m;
    __syncthreads();
    if (threadIdx.x == 0) {
        uint32_t x = 0;
        for (int j = 0; j < 8; ++j) x += s_warp[j];
        cnt[blockIdx.x] = x;
    }
}

// Inclusive block scan of v over the 1024 threads of a block; the block's total in `total`.
__device__ __forceinline__ unsigned long long block_scan_1024(unsigned long long v, unsigned long long* s_warp, unsigned long long& total) {
    const uint32_t lane = threadIdx.x & 31, w = threadIdx.x >> 5;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const unsigned long long y = __shfl_up_sync(0xffffffffu, v, o);
        if (lane >= (uint32_t)o) v += y;
    }
    if (lane == 31) s_warp[w] = v;
    __syncthreads();
    unsigned long long before = 0;
    total = 0;
    for (uint32_t j = 0; j < 32; ++j) {
        const unsigned long long x = s_warp[j];
        before += j < w ? x : 0;
        total += x;
    }
    __syncthreads();
    return v + before;
}

// Exclusive prefix of the chunks' counts and their total, one block (26,000 chunks of a 106 MB
// text: 7 turns).
__global__ void __launch_bounds__(1024) k_nl_scan(const uint32_t* __restrict__ cnt, uint64_t n, uint64_t* __restrict__ pre,
                                                  unsigned long long* __restrict__ total) {
    __shared__ unsigned long long s_warp[32];
    unsigned long long base = 0;
    for (uint64_t i0 = 0; i0 < n; i0 += 4096) {
        const uint64_t i = i0 + threadIdx.x * 4;
        uint32_t c[4];
        unsigned long long t = 0, all;
#pragma unroll
        for (int j = 0; j < 4; ++j) t += c[j] = i + j < n ? cnt[i + j] : 0;
        unsigned long long x = base + block_scan_1024(t, s_warp, all) - t;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            if (i + j < n) pre[i + j] = x;
            x += c[j];
        }
        base += all;
    }
    if (threadIdx.x == 0) *total = base;
}

// Positions of the newlines of each chunk, in order: thread j has the bytes
// [c0 + 16 j, c0 + 16 j + 16); a block scan of the per-thread counts orders them.
__global__ void __launch_bounds__(256) k_nl_pos(const uint8_t* __restrict__ t, uint64_t n, const uint64_t* __restrict__ pre,
                                                uint64_t* pos) {
    __shared__ uint32_t s_warp[8];
    const uint64_t c0 = (uint64_t)blockIdx.x * CHUNK + (uint64_t)threadIdx.x * 16;
    uint32_t bits = nl_bits(t, n, c0);
    const uint32_t m = __popc(bits);
    const uint32_t lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    uint32_t x = m;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t y = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= (uint32_t)o) x += y;
    }
    if (lane == 31) s_warp[w] = x;
    __syncthreads();
    uint32_t before = 0;
    for (uint32_t j = 0; j < w; ++j) before += s_warp[j];
    for (uint64_t o = pre[blockIdx.x] + before + x - m; bits; bits &= bits - 1) pos[o++] = c0 + __ffs(bits) - 1;
}

struct Fq {
    const uint8_t* t;
    const uint64_t* nl;  // newline positions
    uint64_t n_lines;
};

// Line j: [start, end) without the newline and a trailing '\r'.
__device__ __forceinline__ void line_span(const Fq& f, uint64_t j, uint64_t& a, uint64_t& e) {
    a = j == 0 ? 0 : f.nl[j - 1] + 1;
    e = f.nl[j];
    if (e > a && f.t[e - 1] == '\r') --e;
}

__device__ __forceinline__ uint8_t up(uint8_t c) { return (c >= 'a' && c <= 'z') ? (uint8_t)(c - 32) : c; }
__device__ __forceinline__ uint32_t code_of(uint8_t c) {  // ASCII_TO_2BIT
    c = up(c);
    return c == 'C' ? 1u : c == 'G' ? 2u : c == 'T' ? 3u : 0u;
}
// Complement for the merge's reverse complement of R2: a base other than ACGT becomes
// 'A' when R2 has at most 512 bases (trim_merge.rs:152-162) and 'T' when it is longer
// (reverse_complement_ascii, bitseq.rs:90-98, reads it as A and complements it).
__device__ __forceinline__ uint8_t rc_char(uint8_t c, uint64_t l2) {
    return (c == 'A' || c == 'a')   ? 'T'
           : (c == 'C' || c == 'c') ? 'G'
           : (c == 'G' || c == 'g') ? 'C'
           : (c == 'T' || c == 't') ? 'A'
                                    : (l2 <= 512 ? 'A' : 'T');
}

// ---- a pair by one warp -----------------------------------------------------------------
// A read as three bit planes over its bases (bit of base i at bit i of the plane): the two
// bits of its code and whether it is one of ACGTacgt; a base that is not equals none.  One
// word of zeros before the first and after the last, so that 32 bits can be taken from any
// place.  Reads of up to PLANE_BASES bases; longer ones are compared byte by byte.
constexpr uint32_t PLANE_BASES = 512, PLANE_WORDS = PLANE_BASES / 32 + 2;
struct Planes {
    uint32_t lo[PLANE_WORDS], hi[PLANE_WORDS], ok[PLANE_WORDS];
};
__device__ __forceinline__ uint32_t bits_at(const uint32_t* p, int pos) {  // -32 <= pos <= PLANE_BASES - 1
    const uint32_t q = (uint32_t)(pos + 32);
    return __funnelshift_r(p[q >> 5], p[(q >> 5) + 1], q & 31);
}
__device__ __forceinline__ bool is_acgt(uint8_t c) {
    c &= 0xDF;
    return c == 'A' || c == 'C' || c == 'G' || c == 'T';
}
__device__ __forceinline__ void load_planes(Planes& P, const uint8_t* s, uint32_t len) {
    const uint32_t lane = threadIdx.x & 31;
    if (lane < 3) (lane == 0 ? P.lo : lane == 1 ? P.hi : P.ok)[0] = 0;
    const uint32_t words = (len + 31) / 32;
    for (uint32_t c = 0; c <= words; ++c) {
        const uint32_t i = 32 * c + lane;
        const uint8_t b = i < len ? s[i] : 0;
        const uint32_t code = code_of(b);
        const uint32_t lo = __ballot_sync(0xffffffffu, code & 1), hi = __ballot_sync(0xffffffffu, code >> 1);
        const uint32_t ok = __ballot_sync(0xffffffffu, is_acgt(b));
        if (lane < 3) (lane == 0 ? P.lo : lane == 1 ? P.hi : P.ok)[c + 1] = lane == 0 ? lo : lane == 1 ? hi : ok;
    }
}

// The first ten bases of the adapters (trim_merge.rs:17-33).
#define FBK_ADAPTERS "AGATCGGAAG", "AGATGTGTAT", "CTGTCTCTTA"
__host__ __device__ constexpr uint32_t adapter_bits(const char* a, int plane) {
    uint32_t m = 0;
    for (int j = 0; j < 10; ++j) {
        const uint32_t c = a[j] == 'C' ? 1u : a[j] == 'G' ? 2u : a[j] == 'T' ? 3u : 0u;
        m |= (c >> plane & 1u) << j;
    }
    return m;
}

// trim_merge.rs:17-76: the first place among the last 100 where ten bases differ from an
// adapter's in one at most.  (The reference looks only where one of the adapter's first two
// bases is right, which one mismatch at most implies.)
__device__ uint64_t w_trim_adapter(const Planes* P, const uint8_t* s, uint64_t len) {
    if (len < 10) return len;
    const uint32_t lane = threadIdx.x & 31;
    for (uint64_t i0 = len > 100 ? len - 100 : 0; i0 + 10 <= len; i0 += 32) {
        const uint64_t i = i0 + lane;
        bool hit = false;
        if (i + 10 <= len) {
            uint32_t lo = 0, hi = 0, ok = 0;
            if (P) {
                lo = bits_at(P->lo, (int)i), hi = bits_at(P->hi, (int)i), ok = bits_at(P->ok, (int)i);
            } else {
                for (int j = 0; j < 10; ++j) {
                    const uint32_t c = code_of(s[i + j]);
                    lo |= (c & 1) << j, hi |= (c >> 1) << j, ok |= (uint32_t)is_acgt(s[i + j]) << j;
                }
            }
            constexpr const char* ads[3] = {FBK_ADAPTERS};
            constexpr uint32_t al[3] = {adapter_bits(ads[0], 0), adapter_bits(ads[1], 0), adapter_bits(ads[2], 0)};
            constexpr uint32_t ah[3] = {adapter_bits(ads[0], 1), adapter_bits(ads[1], 1), adapter_bits(ads[2], 1)};
#pragma unroll
            for (int a = 0; a < 3; ++a) hit |= __popc(((lo ^ al[a]) | (hi ^ ah[a]) | ~ok) & 0x3FFu) <= 1;
        }
        const uint32_t m = __ballot_sync(0xffffffffu, hit);
        if (m) return i0 + __ffs(m) - 1;
    }
    return len;
}

// trim_merge.rs:79-115 (-1 = None): the longest prefix whose last four qualities average
// min_qual, three if there is none.
__device__ int64_t w_trim_quality(const uint8_t* q, uint64_t len, uint32_t min_qual, uint64_t min_len) {
    if (len < min_len) return -1;
    if (len < 4) return (int64_t)len;
    const uint32_t lane = threadIdx.x & 31;
    uint64_t cut = 3;
    for (uint64_t done = 0; done + 4 <= len; done += 32) {
        bool good = false;
        if (done + lane + 4 <= len) {
            const uint8_t* e = q + (len - done - lane);
            uint64_t s = 0;
#pragma unroll
            for (int j = 1; j <= 4; ++j) s += e[-j] > 33 ? e[-j] - 33 : 0;
            good = s >= (uint64_t)min_qual * 4;
        }
        const uint32_t m = __ballot_sync(0xffffffffu, good);
        if (m) {
            cut = len - done - (__ffs(m) - 1);
            break;
        }
    }
    return cut < min_len ? -1 : (int64_t)cut;
}

// trim_merge.rs:135-238, the overlap search: of the overlaps d of 15 bases and more with at
// most d * 0.10 mismatches (= d / 10 rounded down: 0.10 as a double lies above a tenth by less
// than a rounding), the one with the highest d - 2.5 * mismatches, the longest on a tie; 0 =
// none.  Lane = overlap.  (The reference goes from the longest down and stops where no shorter
// one can score more, which changes nothing.)
__device__ uint64_t w_merge_overlap(const Planes* A, Planes* R, const uint8_t* r1, uint64_t l1, const uint8_t* r2, uint64_t l2) {
    constexpr uint64_t MIN_OVERLAP = 15;
    if (l1 < MIN_OVERLAP || l2 < MIN_OVERLAP) return 0;
    const uint32_t lane = threadIdx.x & 31;
    const uint64_t max_d = l1 < l2 ? l1 : l2;
    if (A) {
        // R holds read 2 forward: its reverse complement takes its place (a base that is not
        // ACGT becomes A, as the read has 512 bases at most)
        uint32_t lo = 0, hi = 0;
        if (lane * 32 < l2) {
            const int pos = (int)l2 - 32 * (int)lane - 32;
            const uint32_t ok = bits_at(R->ok, pos);
            lo = __brev(~bits_at(R->lo, pos) & ok);
            hi = __brev(~bits_at(R->hi, pos) & ok);
        }
        __syncwarp();
        if (lane * 32 < l2) R->lo[lane] = lo, R->hi[lane] = hi;
        __syncwarp();
        uint32_t best = 0;  // score << 10 | d, the score doubled
        for (int d = (int)max_d - (int)lane; d >= (int)MIN_OVERLAP; d -= 32) {
            uint32_t mm = 0;
            for (int c = 0; 32 * c < d; ++c) {
                const int pos = (int)l1 - d + 32 * c;
                const uint32_t x = (bits_at(A->lo, pos) ^ R->lo[c]) | (bits_at(A->hi, pos) ^ R->hi[c]) | ~bits_at(A->ok, pos);
                mm += __popc(d - 32 * c < 32 ? x & ((1u << (d - 32 * c)) - 1) : x);
            }
            if (mm <= (uint32_t)d / 10) best = max(best, (2u * d - 5 * mm) << 10 | (uint32_t)d);
        }
        return __reduce_max_sync(0xffffffffu, best) & 1023u;
    }
    uint64_t score = 0, at = 0;
    for (int64_t d = (int64_t)max_d - lane; d >= (int64_t)MIN_OVERLAP; d -= 32) {
        const uint8_t* s1 = r1 + (l1 - d);
        const uint64_t allowed = (uint64_t)d / 10;
        uint64_t mm = 0;
        for (int64_t i = 0; i < d; ++i)
            if (up(s1[i]) != rc_char(r2[l2 - 1 - i], l2) && ++mm > allowed) break;
        if (mm <= allowed && 2 * (uint64_t)d - 5 * mm > score) score = 2 * (uint64_t)d - 5 * mm, at = (uint64_t)d;
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        const uint64_t s2 = __shfl_xor_sync(0xffffffffu, score, o), a2 = __shfl_xor_sync(0xffffffffu, at, o);
        if (s2 > score || (s2 == score && a2 > at)) score = s2, at = a2;
    }
    return at;
}

struct IngestArgs {
    Fq f1, f2;
    uint64_t n_pairs;
    double factor;
    uint64_t keep_threshold;
    int subsample, trim, merge;
    uint64_t min_len, seed;
    uint32_t min_qual;
};

// What a pair becomes: kind 0 dropped (or subsampled out), 1 merged, 2 unmerged; t1, t2
// the trimmed lengths and ov the merge overlap (merged length t1 + t2 - ov); raw = l1 + l2.
// One warp per pair.  Bound by instruction issue: the bytes of a read are loaded once, side by
// side, and become bit planes by ballots; each adapter place is three popcounts, each overlap
// a popcount a word, where one thread per pair compared byte by byte and every load of a warp
// touched 32 lines.  1 Mbp at 50x, 106 MB of text: 1.80 ms before, 0.38 now.
constexpr int PAIR_WARPS = 8;  // pairs a block works on at a time
__global__ void __launch_bounds__(32 * PAIR_WARPS) k_pair_decide(IngestArgs A, uint8_t* kind, uint32_t* ta, uint32_t* tb, uint32_t* ov,
                                                                 uint32_t* raw, uint8_t* err) {
    __shared__ Planes s_a[PAIR_WARPS], s_b[PAIR_WARPS];
    const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    for (uint64_t p = (uint64_t)blockIdx.x * PAIR_WARPS + warp; p < A.n_pairs; p += (uint64_t)gridDim.x * PAIR_WARPS) {
        // lane j < 8: line j & 3 of the pair's record in file j >> 2
        uint64_t la = 0, le = 0;
        bool bad = false;
        if (lane < 8) {
            const Fq& f = lane < 4 ? A.f1 : A.f2;
            line_span(f, 4 * p + (lane & 3), la, le);
            if ((lane & 1) == 0) bad = le == la || f.t[la] != ((lane & 2) ? '+' : '@');
        }
        const uint64_t s1a = __shfl_sync(0xffffffffu, la, 1), s2a = __shfl_sync(0xffffffffu, la, 5);
        const uint64_t q1a = __shfl_sync(0xffffffffu, la, 3), q2a = __shfl_sync(0xffffffffu, la, 7);
        const uint64_t n = le - la;
        const uint64_t l1 = __shfl_sync(0xffffffffu, n, 1), l2 = __shfl_sync(0xffffffffu, n, 5);
        if (lane == 3) bad = n != l1;
        if (lane == 7) bad = n != l2;
        uint64_t t1 = 0, t2 = 0, d = 0;
        uint32_t what = 0;
        if (__any_sync(0xffffffffu, bad)) {
            if (lane == 0) *err = 1;
        } else if (!(A.subsample && smix((p + 1) ^ A.seed) > A.keep_threshold)) {  // 1-based input pair (trim_merge.rs:324-348)
            const uint8_t *s1 = A.f1.t + s1a, *q1 = A.f1.t + q1a, *s2 = A.f2.t + s2a, *q2 = A.f2.t + q2a;
            const bool planes = l1 <= PLANE_BASES && l2 <= PLANE_BASES;
            Planes *pa = planes ? &s_a[warp] : nullptr, *pb = planes ? &s_b[warp] : nullptr;
            if (planes) {
                __syncwarp();
                load_planes(*pa, s1, (uint32_t)l1);
                load_planes(*pb, s2, (uint32_t)l2);
                __syncwarp();
            }
            int64_t x1 = l1 < A.min_len ? -1 : (int64_t)l1, x2 = l2 < A.min_len ? -1 : (int64_t)l2;
            if (A.trim) {
                x1 = w_trim_quality(q1, w_trim_adapter(pa, s1, l1), A.min_qual, A.min_len);
                x2 = w_trim_quality(q2, w_trim_adapter(pb, s2, l2), A.min_qual, A.min_len);
            }
            if (x1 >= 0 && x2 >= 0) {
                t1 = (uint64_t)x1;
                t2 = (uint64_t)x2;
                d = A.merge ? w_merge_overlap(pa, pb, s1, t1, s2, t2) : 0;
                what = d ? 1 : 2;
            }
        }
        if (lane == 0) {
            raw[p] = (uint32_t)(l1 + l2);
            kind[p] = (uint8_t)what;
            ta[p] = (uint32_t)t1;
            tb[p] = (uint32_t)t2;
            ov[p] = (uint32_t)d;
        }
    }
}

// Sums over pairs: reads and bases of the three arenas (pe_reverse has as many reads as
// pe_forward), bases after and before trimming, longest read.
enum { PS_MERGED, PS_MERGED_BASES, PS_UNMERGED, PS_FWD_BASES, PS_REV_BASES, PS_AFTER, PS_BEFORE, PS_MAX_LEN, PS_N };
constexpr uint32_t PAIR_TILE = 64;
struct PairState {
    const uint8_t* kind;
    const uint32_t *ta, *tb, *ov, *raw;
    uint64_t n;
};
__device__ __forceinline__ void pair_sums(const PairState& S, uint64_t p, unsigned long long (&v)[PS_N]) {
#pragma unroll
    for (int q = 0; q < PS_N; ++q) v[q] = 0;
    if (p >= S.n) return;
    const uint32_t kd = S.kind[p];
    v[PS_BEFORE] = S.raw[p];
    if (!kd) return;
    const unsigned long long t1 = S.ta[p], t2 = S.tb[p];
    v[PS_AFTER] = t1 + t2;
    if (kd == 1) {
        v[PS_MERGED] = 1;
        v[PS_MERGED_BASES] = v[PS_MAX_LEN] = t1 + t2 - S.ov[p];
    } else {
        v[PS_UNMERGED] = 1;
        v[PS_FWD_BASES] = t1;
        v[PS_REV_BASES] = t2;
        v[PS_MAX_LEN] = max(t1, t2);
    }
}

// Sums of each tile of pairs, one warp a tile.
__global__ void __launch_bounds__(256) k_pair_sums(PairState S, uint64_t n_tiles, unsigned long long* __restrict__ part) {
    const uint32_t lane = threadIdx.x & 31;
    const uint64_t tile = (uint64_t)blockIdx.x * 8 + (threadIdx.x >> 5);
    if (tile >= n_tiles) return;
    unsigned long long a[PS_N], b[PS_N];
    pair_sums(S, tile * PAIR_TILE + lane, a);
    pair_sums(S, tile * PAIR_TILE + 32 + lane, b);
#pragma unroll
    for (int q = 0; q < PS_N; ++q) {
        unsigned long long x = q == PS_MAX_LEN ? max(a[q], b[q]) : a[q] + b[q];
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            const unsigned long long y = __shfl_xor_sync(0xffffffffu, x, o);
            x = q == PS_MAX_LEN ? max(x, y) : x + y;
        }
        if (lane == q) part[tile * PS_N + q] = x;
    }
}

// The tiles' sums to exclusive prefixes in place, and the totals; one block.
__global__ void __launch_bounds__(1024) k_pair_scan(unsigned long long* __restrict__ part, uint64_t n_tiles,
                                                    unsigned long long* __restrict__ total) {
    __shared__ unsigned long long s_warp[32], s_max;
    if (threadIdx.x == 0) s_max = 0;
    unsigned long long base[PS_MAX_LEN] = {}, longest = 0;
    for (uint64_t i0 = 0; i0 < n_tiles; i0 += 1024) {
        const uint64_t i = i0 + threadIdx.x;
#pragma unroll
        for (int q = 0; q < PS_MAX_LEN; ++q) {
            const unsigned long long v = i < n_tiles ? part[i * PS_N + q] : 0;
            unsigned long long all;
            const unsigned long long x = base[q] + block_scan_1024(v, s_warp, all) - v;
            if (i < n_tiles) part[i * PS_N + q] = x;
            base[q] += all;
        }
        if (i < n_tiles) longest = max(longest, part[i * PS_N + PS_MAX_LEN]);
    }
    __syncthreads();
    atomicMax(&s_max, longest);
    __syncthreads();
    if (threadIdx.x == 0) {
#pragma unroll
        for (int q = 0; q < PS_MAX_LEN; ++q) total[q] = base[q];
        total[PS_MAX_LEN] = s_max;
    }
}

struct WriteArgs {
    uint64_t* data;      // all arenas' words, arena a from word wbase[a]
    uint64_t* off;       // bank-global base offsets
    uint32_t* len;
    uint32_t* pair_idx;
    uint64_t wbase[3];
    uint64_t rbase[3];   // first read of each arena
};

__device__ __forceinline__ uint64_t spread_bits(uint32_t v) {  // bit i to bit 2 i
    uint64_t x = v;
    x = (x | (x << 16)) & 0x0000FFFF0000FFFFull;
    x = (x | (x << 8)) & 0x00FF00FF00FF00FFull;
    x = (x | (x << 4)) & 0x0F0F0F0F0F0F0F0Full;
    x = (x | (x << 2)) & 0x3333333333333333ull;
    return (x | (x << 1)) & 0x5555555555555555ull;
}
// n bases to the packed words from base g on, by a warp: 32 codes a step become one word by
// two ballots; words collect in the lanes and are written 32 at a time (into cleared words,
// whose ends other reads share).
template <class Code>
__device__ __forceinline__ void put_read(uint64_t* data, uint64_t g, uint64_t n, Code&& code) {
    const uint32_t lane = threadIdx.x & 31, sh = (uint32_t)(g & 31) * 2;
    for (uint64_t i0 = 0; i0 < n; i0 += 1024) {
        uint64_t word = 0;
        for (uint32_t c = 0; c < 32 && i0 + 32 * c < n; ++c) {
            const uint64_t i = i0 + 32 * c + lane;
            const uint32_t x = i < n ? code(i) : 0u;
            const uint32_t lo = __ballot_sync(0xffffffffu, x & 1), hi = __ballot_sync(0xffffffffu, x >> 1);
            if (lane == c) word = spread_bits(lo) | (spread_bits(hi) << 1);
        }
        unsigned long long* w = (unsigned long long*)data + (g >> 5) + (i0 >> 5) + lane;
        if (word << sh) atomicOr(w, (unsigned long long)(word << sh));
        if (sh && word >> (64 - sh)) atomicOr(w + 1, (unsigned long long)(word >> (64 - sh)));
    }
}

// A block per tile of pairs: their places in the arenas by a scan, then a warp per pair.  One
// word and two atomics per 32 bases, where each base was an atomic of its own: 0.33 ms before
// at 1 Mbp and 50x, 0.26 now, and the host's pass over the pairs (4 copies, 2 ms) is gone.
__global__ void __launch_bounds__(32 * PAIR_WARPS) k_pair_write(IngestArgs A, WriteArgs W, PairState S,
                                                                const unsigned long long* __restrict__ part) {
    __shared__ uint64_t s_read[PAIR_TILE], s_base[PAIR_TILE], s_base2[PAIR_TILE], s_sum[3];
    const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const unsigned long long* before = part + (uint64_t)blockIdx.x * PS_N;
    unsigned long long v[PS_N], x[PS_MAX_LEN] = {};
    if (threadIdx.x < PAIR_TILE) {
        pair_sums(S, (uint64_t)blockIdx.x * PAIR_TILE + threadIdx.x, v);
#pragma unroll
        for (int q = 0; q <= PS_REV_BASES; ++q) {
            x[q] = v[q];
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const unsigned long long y = __shfl_up_sync(0xffffffffu, x[q], o);
                if (lane >= (uint32_t)o) x[q] += y;
            }
        }
        const bool merged = v[PS_MERGED];
        s_read[threadIdx.x] = merged ? before[PS_MERGED] + x[PS_MERGED] - 1 : before[PS_UNMERGED] + x[PS_UNMERGED] - v[PS_UNMERGED];
        s_base[threadIdx.x] = merged ? before[PS_MERGED_BASES] + x[PS_MERGED_BASES] - v[PS_MERGED_BASES]
                                     : before[PS_FWD_BASES] + x[PS_FWD_BASES] - v[PS_FWD_BASES];
        s_base2[threadIdx.x] = before[PS_REV_BASES] + x[PS_REV_BASES] - v[PS_REV_BASES];
        // the first warp's sums, which the second one's pairs come after
        if (threadIdx.x == 31) s_sum[0] = x[PS_MERGED] | (x[PS_UNMERGED] << 32), s_sum[1] = x[PS_MERGED_BASES], s_sum[2] = x[PS_FWD_BASES];
    }
    __shared__ uint64_t s_rev;
    if (threadIdx.x == 31) s_rev = x[PS_REV_BASES];
    __syncthreads();
    for (uint32_t j = warp; j < PAIR_TILE; j += PAIR_WARPS) {
        const uint64_t p = (uint64_t)blockIdx.x * PAIR_TILE + j;
        if (p >= S.n) break;
        const uint8_t kd = S.kind[p];
        if (!kd) continue;
        uint64_t read = s_read[j], base = s_base[j], base2 = s_base2[j];
        if (j >= 32) {
            read += kd == 1 ? s_sum[0] & 0xFFFFFFFFu : s_sum[0] >> 32;
            base += kd == 1 ? s_sum[1] : s_sum[2];
            base2 += s_rev;
        }
        uint64_t s1a, s1e, q1a, q1e, s2a, s2e, q2a, q2e;
        line_span(A.f1, 4 * p + 1, s1a, s1e);
        line_span(A.f1, 4 * p + 3, q1a, q1e);
        line_span(A.f2, 4 * p + 1, s2a, s2e);
        line_span(A.f2, 4 * p + 3, q2a, q2e);
        const uint8_t *s1 = A.f1.t + s1a, *q1 = A.f1.t + q1a, *s2 = A.f2.t + s2a, *q2 = A.f2.t + q2a;
        const uint64_t t1 = S.ta[p], t2 = S.tb[p];
        auto place = [&](uint64_t r, uint64_t g, uint64_t n) {
            if (lane) return;
            W.off[r] = g;
            W.len[r] = (uint32_t)n;
            W.pair_idx[r] = (uint32_t)p;
        };
        if (kd == 1) {
            // merged read (trim_merge.rs:214-237): r1 prefix, the overlap base by base
            // (agreeing bases, else the higher quality), then rc(r2) past the overlap
            const uint64_t d = S.ov[p], m = t1 + t2 - d, g = W.wbase[0] * 32 + base;
            place(W.rbase[0] + read, g, m);
            put_read(W.data, g, m, [&](uint64_t i) {
                const uint64_t j2 = t2 - 1 - (i - (t1 - d));  // of read 2, from i = t1 - d on
                if (i < t1 - d) return code_of(s1[i]);
                if (i >= t1) return code_of(rc_char(s2[j2], t2));
                const uint8_t b1 = up(s1[i]), b2 = rc_char(s2[j2], t2);
                return code_of(b1 == b2 || q1[i] >= q2[j2] ? b1 : b2);
            });
        } else {
            const uint64_t g1 = W.wbase[1] * 32 + base, g2 = W.wbase[2] * 32 + base2;
            place(W.rbase[1] + read, g1, t1);
            place(W.rbase[2] + read, g2, t2);
            put_read(W.data, g1, t1, [&](uint64_t i) { return code_of(s1[i]); });
            put_read(W.data, g2, t2, [&](uint64_t i) { return code_of(s2[i]); });
        }
    }
}

// Reads per length below bins - 1; hist[bins] the bases of the others.
constexpr uint32_t HIST_SHARED = 2048;
__global__ void __launch_bounds__(256) k_len_hist(const uint32_t* __restrict__ len, uint64_t n, uint64_t bins,
                                                  unsigned long long* __restrict__ hist) {
    __shared__ uint32_t s[HIST_SHARED];  // a block sees fewer than 2^32 reads
    for (uint32_t i = threadIdx.x; i < HIST_SHARED; i += blockDim.x) s[i] = 0;
    __syncthreads();
    for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (uint64_t)gridDim.x * blockDim.x) {
        const uint32_t L = len[i];
        if (L >= bins - 1) atomicAdd(&hist[bins], (unsigned long long)L);
        else if (L < HIST_SHARED) atomicAdd(&s[L], 1u);
        else atomicAdd(&hist[L], 1ULL);
    }
    __syncthreads();
    for (uint32_t i = threadIdx.x; i < HIST_SHARED; i += blockDim.x)
        if (s[i]) atomicAdd(&hist[i], (unsigned long long)s[i]);
}

struct DBufs {
    fbk_ctx* c;
    std::vector<void*> p;
    void* get(uint64_t b) {
        void* q = dev_alloc(c, std::max<uint64_t>(b, 8));
        if (q) p.push_back(q);
        return q;
    }
    ~DBufs() {
        cudaStreamSynchronize(c->stream);
        for (void* q : p) dev_free(c, q);
    }
};

// A FASTQ text in host memory or in an open file.  A file is read straight into the page-locked
// staging slots, in pieces by the worker threads while the other slot's copy runs: 106 MB in
// 1.5 ms, where reading the file into a new array took 10.5 and the copy of that array 4.
struct Text {
    const uint8_t* mem;
    int fd;
    uint64_t len;
    bool read(void* dst, uint64_t off, uint64_t n) const {  // of the file
        while (n) {
            const ssize_t got = pread(fd, dst, n, (off_t)off);
            if (got < 0 && errno == EINTR) continue;
            if (got <= 0) return false;
            dst = (char*)dst + got;
            off += (uint64_t)got;
            n -= (uint64_t)got;
        }
        return true;
    }
};

// One text on the device (with the final newline it may lack) and its newlines per chunk.
struct Lines {
    Fq f{};
    uint64_t n = 0;
    uint64_t* pre = nullptr;
};

fbk_status upload_text(fbk_ctx* ctx, DBufs& B, const Text& T, Lines& ln, unsigned long long* d_total) {
    uint8_t last = 0;
    if (T.len) {
        if (T.mem) last = T.mem[T.len - 1];
        else if (!T.read(&last, T.len - 1, 1)) return set_err(ctx, FBK_ERR_IO, "reading a FASTQ file");
    }
    const bool add_nl = T.len && last != '\n';
    const uint64_t n = T.len + (add_nl ? 1 : 0);
    const uint64_t n_chunks = (n + CHUNK - 1) / CHUNK;
    uint8_t* t = (uint8_t*)B.get((n + 15) & ~15ULL);
    uint32_t* cnt = (uint32_t*)B.get(n_chunks * 4);
    ln.pre = (uint64_t*)B.get(n_chunks * 8);
    if (!t || !cnt || !ln.pre) return set_err(ctx, FBK_ERR_OOM, "FASTQ text on the device");
    ln.f.t = t;
    ln.n = n;
    if (!n) {
        CK(ctx, cudaMemsetAsync(d_total, 0, 8, ctx->stream));
        return FBK_OK;
    }
    if (T.mem) {
        CK(ctx, copy_h2d(ctx, t, T.mem, T.len));
    } else {
        bool ok = true;
        CK(ctx, copy_h2d_from(ctx, t, T.len, [&](void* dst, size_t off, size_t bytes) { return T.read(dst, off, bytes); }, &ok));
        if (!ok) return set_err(ctx, FBK_ERR_IO, "reading a FASTQ file");
    }
    if (add_nl) CK(ctx, cudaMemsetAsync(t + T.len, '\n', 1, ctx->stream));
    TIMED(ctx, "ingest_lines", (k_nl_count<<<(unsigned)n_chunks, 256, 0, ctx->stream>>>(t, n, cnt), cudaGetLastError()));
    TIMED(ctx, "ingest_lines", (k_nl_scan<<<1, 1024, 0, ctx->stream>>>(cnt, n_chunks, ln.pre, d_total), cudaGetLastError()));
    return FBK_OK;
}

fbk_status index_lines(fbk_ctx* ctx, DBufs& B, Lines& ln, uint64_t total) {
    uint64_t* pos = (uint64_t*)B.get(total * 8);
    if (!pos) return set_err(ctx, FBK_ERR_OOM, "FASTQ line index");
    ln.f.nl = pos;
    ln.f.n_lines = total;
    if (ln.n)
        TIMED(ctx, "ingest_lines", (k_nl_pos<<<(unsigned)((ln.n + CHUNK - 1) / CHUNK), 256, 0, ctx->stream>>>(ln.f.t, ln.n, ln.pre, pos),
                                    cudaGetLastError()));
    return FBK_OK;
}

fbk_status ingest_device(fbk_ctx* ctx, const Text& T1, const Text& T2, double subsample_factor, uint64_t min_len, uint32_t min_qual,
                         int enable_trim, int enable_merge, uint64_t seed, fbk_bank** out, fbk_ingest_stats* stats) {
    CK(ctx, cudaSetDevice(ctx->device));
    DBufs B{ctx, {}};
    Lines ln[2];
    // totals of the two line counts, then of the pairs, then the error flag
    unsigned long long* d_tot = (unsigned long long*)B.get(8 * (2 + PS_N + 1));
    if (!d_tot) return set_err(ctx, FBK_ERR_OOM, "device ingest");
    unsigned long long* h = (unsigned long long*)ctx->h_pinned;
    fbk_status st = upload_text(ctx, B, T1, ln[0], d_tot);
    if (st == FBK_OK) st = upload_text(ctx, B, T2, ln[1], d_tot + 1);
    if (st) return st;
    CK(ctx, cudaMemcpyAsync(h, d_tot, 16, cudaMemcpyDeviceToHost, ctx->stream));
    CK(ctx, cudaStreamSynchronize(ctx->stream));
    const uint64_t lines1 = h[0], lines2 = h[1];
    if (lines1 % 4 || lines2 % 4)
        return set_err(ctx, FBK_ERR_FORMAT, "device ingest reads plain 4-line FASTQ records (a record is incomplete or blank lines "
                                            "separate records; the host ingest reads those)");
    if (lines1 != lines2) return set_err(ctx, FBK_ERR_FORMAT, "Mismatched paired-end FASTQ mate counts between R1 and R2");
    const uint64_t n_pairs = lines1 / 4;
    if (n_pairs >= (1ULL << 32)) return set_err(ctx, FBK_ERR_INVALID, "device ingest: 2^32 or more pairs");
    st = index_lines(ctx, B, ln[0], lines1);
    if (st == FBK_OK) st = index_lines(ctx, B, ln[1], lines2);
    if (st) return st;
    IngestArgs A{};
    A.f1 = ln[0].f;
    A.f2 = ln[1].f;
    A.n_pairs = n_pairs;
    A.factor = subsample_factor;
    A.subsample = subsample_factor < 0.999;
    const double x = subsample_factor * 18446744073709551616.0;
    A.keep_threshold = !(x > 0.0) ? 0 : x >= 18446744073709551616.0 ? UINT64_MAX : (uint64_t)x;
    A.trim = enable_trim != 0;
    A.merge = enable_merge != 0;
    A.min_len = min_len;
    A.min_qual = min_qual;
    A.seed = seed;
    const uint64_t n_tiles = (n_pairs + PAIR_TILE - 1) / PAIR_TILE;
    uint8_t* kind = (uint8_t*)B.get(n_pairs);
    uint32_t* ta = (uint32_t*)B.get(n_pairs * 4);
    uint32_t* tb = (uint32_t*)B.get(n_pairs * 4);
    uint32_t* ov = (uint32_t*)B.get(n_pairs * 4);
    uint32_t* raw = (uint32_t*)B.get(n_pairs * 4);
    unsigned long long* part = (unsigned long long*)B.get(n_tiles * PS_N * 8);
    unsigned long long* d_sums = d_tot + 2;
    uint8_t* err = (uint8_t*)(d_sums + PS_N);
    if (!kind || !ta || !tb || !ov || !raw || !part) return set_err(ctx, FBK_ERR_OOM, "device ingest pair state");
    CK(ctx, cudaMemsetAsync(d_sums, 0, 8 * (PS_N + 1), ctx->stream));
    const PairState S{kind, ta, tb, ov, raw, n_pairs};
    if (n_pairs) {
        const unsigned grid = (unsigned)std::min<uint64_t>((n_pairs + PAIR_WARPS - 1) / PAIR_WARPS, (uint64_t)ctx->num_sms * 32);
        TIMED(ctx, "ingest_decide", (k_pair_decide<<<grid, 32 * PAIR_WARPS, 0, ctx->stream>>>(A, kind, ta, tb, ov, raw, err),
                                     cudaGetLastError()));
        TIMED(ctx, "ingest_places", (k_pair_sums<<<(unsigned)((n_tiles + 7) / 8), 256, 0, ctx->stream>>>(S, n_tiles, part),
                                     cudaGetLastError()));
        TIMED(ctx, "ingest_places", (k_pair_scan<<<1, 1024, 0, ctx->stream>>>(part, n_tiles, d_sums), cudaGetLastError()));
    }
    CK(ctx, cudaMemcpyAsync(h, d_sums, 8 * (PS_N + 1), cudaMemcpyDeviceToHost, ctx->stream));
    CK(ctx, cudaStreamSynchronize(ctx->stream));
    if (h[PS_N] & 0xFF) return set_err(ctx, FBK_ERR_FORMAT, "Corrupted FASTQ record (header, '+' line or quality length)");
    // IngestStats (trim_merge.rs:307-417); reads and bases per arena (pair order = push order)
    fbk_ingest_stats R{};
    R.input_read_pairs = n_pairs;
    R.retained_read_pairs = h[PS_MERGED] + h[PS_UNMERGED];
    R.bases_before_trim = h[PS_BEFORE];
    R.bases_after_trim = h[PS_AFTER];
    R.merged_pairs_count = h[PS_MERGED];
    R.merged_bases = h[PS_MERGED_BASES];
    R.unmerged_pairs_count = h[PS_UNMERGED];
    const uint64_t nr[3] = {h[PS_MERGED], h[PS_UNMERGED], h[PS_UNMERGED]};
    const uint64_t nb[3] = {h[PS_MERGED_BASES], h[PS_FWD_BASES], h[PS_REV_BASES]};
    const uint32_t max_len = (uint32_t)h[PS_MAX_LEN];
    const uint64_t n_reads = nr[0] + nr[1] + nr[2];
    if (n_reads == 0)
        return set_err(ctx, FBK_ERR_EMPTY, "No valid reads survived trimming and quality filtering (check input FASTQ files)");
    const uint64_t aw[3] = {(nb[0] + 31) / 32, (nb[1] + 31) / 32, (nb[2] + 31) / 32};
    const uint64_t n_words = aw[0] + aw[1] + aw[2];
    const uint64_t bins = std::min<uint64_t>((uint64_t)max_len + 2, 1ULL << 16);
    fbk_bank* bk = new fbk_bank();
    struct BankGuard {
        fbk_bank* b;
        ~BankGuard() {
            if (b) fbk_bank_release(b);
        }
    } guard{bk};
    bk->ctx = ctx;
    bk->data = (uint64_t*)dev_alloc(ctx, (n_words + 8) * 8);
    bk->off = (uint64_t*)dev_alloc(ctx, n_reads * 8);
    bk->len = (uint32_t*)dev_alloc(ctx, n_reads * 4);
    bk->pair_idx = (uint32_t*)dev_alloc(ctx, n_reads * 4);
    unsigned long long* hist = (unsigned long long*)B.get(8 * (std::max<uint64_t>(bins, HIST_SHARED) + 1));
    if (!bk->data || !bk->off || !bk->len || !bk->pair_idx || !hist) return set_err(ctx, FBK_ERR_OOM, "device memory for the read bank");
    WriteArgs W{};
    W.data = bk->data;
    W.off = bk->off;
    W.len = bk->len;
    W.pair_idx = bk->pair_idx;
    W.wbase[0] = 0;
    W.wbase[1] = aw[0];
    W.wbase[2] = aw[0] + aw[1];
    W.rbase[0] = 0;
    W.rbase[1] = nr[0];
    W.rbase[2] = nr[0] + nr[1];
    CK(ctx, cudaMemsetAsync(bk->data, 0, (n_words + 8) * 8, ctx->stream));
    CK(ctx, cudaMemsetAsync(hist, 0, 8 * (std::max<uint64_t>(bins, HIST_SHARED) + 1), ctx->stream));
    TIMED(ctx, "ingest_write", (k_pair_write<<<(unsigned)n_tiles, 32 * PAIR_WARPS, 0, ctx->stream>>>(A, W, S, part), cudaGetLastError()));
    TIMED(ctx, "ingest_hist", (k_len_hist<<<(unsigned)std::min<uint64_t>((n_reads + 255) / 256, (uint64_t)ctx->num_sms * 2), 256, 0,
                                            ctx->stream>>>(bk->len, n_reads, bins, hist),
                               cudaGetLastError()));
    // bank bookkeeping as bank_upload_impl keeps it
    bk->n_reads = n_reads;
    bk->n_words = n_words;
    bk->n_bases = nb[0] + nb[1] + nb[2];
    bk->n_pairs = n_pairs;
    bk->disjoint = true;
    bk->max_len = max_len;
    bk->arena_reads.assign(nr, nr + 3);
    bk->len_hist.assign(bins, 0);
    std::vector<uint64_t> hh(bins + 1);
    CK(ctx, cudaMemcpyAsync(hh.data(), hist, 8 * (bins + 1), cudaMemcpyDeviceToHost, ctx->stream));
    std::vector<uint32_t> lens;
    if (bk->n_bases >= (1ull << 30)) {  // several chunks: the lengths say where they begin
        lens.resize(n_reads);
        CK(ctx, copy_d2h(ctx, lens.data(), bk->len, n_reads * 4));
    }
    CK(ctx, cudaStreamSynchronize(ctx->stream));
    std::copy(hh.begin(), hh.begin() + bins, bk->len_hist.begin());
    bk->long_bases = hh[bins];
    bk->chunk_starts.push_back(0);
    uint64_t acc = lens.empty() ? bk->n_bases : 0;
    for (uint64_t r = 0; r < lens.size(); ++r) {
        if (acc && acc + lens[r] >= (1ull << 30)) {
            bk->chunk_starts.push_back(r);
            bk->max_chunk = std::max(bk->max_chunk, acc);
            acc = 0;
        }
        acc += lens[r];
    }
    bk->max_chunk = std::max(bk->max_chunk, acc);
    bk->chunk_starts.push_back(n_reads);
    if (stats) *stats = R;
    guard.b = nullptr;
    *out = bk;
    return FBK_OK;
}

}  // namespace

extern "C" {

FBK_API fbk_status fbk_ingest_fastq_device(fbk_ctx* ctx, const uint8_t* r1, uint64_t r1_len, const uint8_t* r2, uint64_t r2_len,
                                           double subsample_factor, uint64_t min_len, uint32_t min_qual, int enable_trim,
                                           int enable_merge, uint64_t seed, fbk_bank** out, fbk_ingest_stats* stats) {
    if (!ctx || !out || (r1_len && !r1) || (r2_len && !r2)) return FBK_ERR_INVALID;
    *out = nullptr;
    static const uint8_t none = 0;
    return ingest_device(ctx, Text{r1 ? r1 : &none, -1, r1_len}, Text{r2 ? r2 : &none, -1, r2_len}, subsample_factor, min_len, min_qual,
                         enable_trim, enable_merge, seed, out, stats);
}

FBK_API fbk_status fbk_ingest_fastq_fd_device(fbk_ctx* ctx, int fd1, int fd2, double subsample_factor, uint64_t min_len,
                                              uint32_t min_qual, int enable_trim, int enable_merge, uint64_t seed, fbk_bank** out,
                                              fbk_ingest_stats* stats) {
    if (!ctx || !out) return FBK_ERR_INVALID;
    *out = nullptr;
    Text T[2] = {{nullptr, fd1, 0}, {nullptr, fd2, 0}};
    for (Text& t : T) {
        struct stat sb;
        if (fstat(t.fd, &sb) != 0 || !S_ISREG(sb.st_mode)) return set_err(ctx, FBK_ERR_IO, "device ingest reads regular files");
        t.len = (uint64_t)sb.st_size;
    }
    return ingest_device(ctx, T[0], T[1], subsample_factor, min_len, min_qual, enable_trim, enable_merge, seed, out, stats);
}

// Copies a device bank back (for checks and hand-off): words (n_words), base offsets
// (bank-global), lengths and pair indices (n_reads each; any may be NULL).
FBK_API fbk_status fbk_bank_export(const fbk_bank* b, uint64_t* words, uint64_t* offsets, uint32_t* lengths, uint32_t* pair_idx) {
    if (!b) return FBK_ERR_INVALID;
    fbk_ctx* ctx = b->ctx;
    CK(ctx, bank_wait(ctx, b));
    if (words && b->n_words) CK(ctx, cudaMemcpyAsync(words, b->data, b->n_words * 8, cudaMemcpyDeviceToHost, ctx->stream));
    if (offsets && b->n_reads) CK(ctx, cudaMemcpyAsync(offsets, b->off, b->n_reads * 8, cudaMemcpyDeviceToHost, ctx->stream));
    if (lengths && b->n_reads) CK(ctx, cudaMemcpyAsync(lengths, b->len, b->n_reads * 4, cudaMemcpyDeviceToHost, ctx->stream));
    if (pair_idx && b->n_reads) {
        if (!b->pair_idx) return set_err(ctx, FBK_ERR_INVALID, "bank has no pair indices");
        CK(ctx, cudaMemcpyAsync(pair_idx, b->pair_idx, b->n_reads * 4, cudaMemcpyDeviceToHost, ctx->stream));
    }
    CK(ctx, cudaStreamSynchronize(ctx->stream));
    return FBK_OK;
}

FBK_API fbk_status fbk_bank_words(const fbk_bank* b, uint64_t* n_words) {
    if (!b || !n_words) return FBK_ERR_INVALID;
    *n_words = b->n_words;
    return FBK_OK;
}

FBK_API fbk_status fbk_bank_arena_counts(const fbk_bank* b, uint64_t* counts3) {
    if (!b || !counts3) return FBK_ERR_INVALID;
    for (int a = 0; a < 3; ++a) counts3[a] = a < (int)b->arena_reads.size() ? b->arena_reads[a] : 0;
    return FBK_OK;
}

}  // extern "C"
