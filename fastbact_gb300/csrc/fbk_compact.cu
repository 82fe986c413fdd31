// fbk_compact.cu — unitig compaction from the device-resident solid table
// (src/graph/build.rs:330-594).
//
// The reference walks, in hash-map order, every out-edge of every boundary directed
// k-mer (in-degree != 1 or out-degree != 1), extending through 1-in-1-out nodes and
// marking the edges it used so the walk from the other end of the same unitig is
// skipped; then it walks the remaining all-1-in-1-out cycles; then it links unitigs
// whose ends overlap by k or k-1 bases.  Here:
//   1. a node index (open addressing over the converted rows) is built on the device;
//   2. the successor of every 1-in-1-out directed node is looked up once, and doubled: table
//      l holds the node 2^l steps on, as long as all of them are 1-in-1-out;
//   3. every (boundary node, direction, out-edge) start finds its path's length and end by
//      descending those tables, one thread per start, with no shared marks: a unitig
//      reachable from both ends is kept from the end whose (row, direction, edge) is smaller
//      — the same set of unitigs, decided without ordering — and one that is its own reverse
//      complement, which has one end, up to its middle;
//   4. the bases of the kept paths are written eight to a thread, each thread jumping to its
//      place, already in the orientation of min(sequence, reverse complement);
//   5. the 1-in-1-out nodes no path visited (isolated cycles, few) and the overlap
//      edges are handled on the host, as build.rs:450-594 does.
// A walk of one thread along a whole unitig is a chain of dependent loads, about 1 us a
// step: 44 ms twice for the 42 k steps of the longest unitig of a 1 Mbp genome (k = 31, 1.0 M
// rows), where the tables take 0.25 ms, the paths 0.05 and their bases 0.04.
// A unitig's coverage is the mean node coverage of its path without the last node
// (build.rs:379-435); which end a path starts from therefore changes its coverage
// when the end nodes differ, exactly as the reference's map order does.
#include <algorithm>
#include <array>
#include <cstring>
#include <string>
#include <unordered_map>
#include <vector>

#include "fbk_device.cuh"
#include "fbk_internal.h"

using namespace fbk;

namespace {

constexpr uint64_t CIDX_SALT = 0x3c6ef372fe94f82bULL;

// ---- multi-word k-mer integers (big-endian words, value = the MSB-first k-mer) ----
template <int NW>
__host__ __device__ __forceinline__ void kshl2_push(Key<NW>& x, uint32_t b, uint32_t k) {
    // ((x << 2) | b) masked to 2k bits (KmerInt::roll_next, forward half)
#pragma unroll
    for (int i = 0; i < NW; ++i) x.w[i] = (x.w[i] << 2) | (i + 1 < NW ? (x.w[i + 1] >> 62) : 0ULL);
    x.w[NW - 1] |= b;
    const uint32_t bits = 2 * k;
#pragma unroll
    for (int i = 0; i < NW; ++i) {
        const int lo = 64 * (NW - 1 - i);  // lowest bit of word i
        if ((int)bits <= lo) x.w[i] = 0;
        else if ((int)bits < lo + 64) x.w[i] &= (1ULL << (bits - lo)) - 1;
    }
}
template <int NW>
__host__ __device__ __forceinline__ void kshr2_put(Key<NW>& x, uint32_t c, uint32_t k) {
    // (x >> 2) | (c << 2(k-1))  (KmerInt::roll_next, reverse half)
#pragma unroll
    for (int i = NW - 1; i >= 0; --i) x.w[i] = (x.w[i] >> 2) | (i > 0 ? (x.w[i - 1] << 62) : 0ULL);
    const uint32_t pos = 2 * (k - 1);
    x.w[NW - 1 - pos / 64] |= (uint64_t)c << (pos % 64);
}
template <int NW>
__host__ __device__ __forceinline__ uint32_t kbase(const Key<NW>& x, uint32_t i, uint32_t k) {
    // base i from the 5' end (i = 0: most significant)
    const uint32_t pos = 2 * (k - 1 - i);
    return (uint32_t)(x.w[NW - 1 - pos / 64] >> (pos % 64)) & 3u;
}
// Base 0 (the 5' end) and the reverse complement, on registers (no word index of its own).
template <int NW>
__device__ __forceinline__ uint32_t kfirst(const Key<NW>& x, uint32_t k) {
    const uint32_t pos = 2 * (k - 1), wd = NW - 1 - pos / 64;
    uint64_t v = 0;
#pragma unroll
    for (int i = 0; i < NW; ++i) v = (uint32_t)i == wd ? x.w[i] : v;
    return (uint32_t)(v >> (pos % 64)) & 3u;
}
template <int NW>
__device__ __forceinline__ Key<NW> krc_dev(const Key<NW>& x, uint32_t k) {
    // all 32 NW groups reversed and complemented, then the 64 NW - 2k bits of padding dropped
    const uint32_t s = 64u * NW - 2u * k, ws = s >> 6, bs = s & 63;
    uint64_t y[NW];
#pragma unroll
    for (int i = 0; i < NW; ++i) y[i] = ~rev2(x.w[NW - 1 - i]);
    Key<NW> r;
#pragma unroll
    for (int i = 0; i < NW; ++i) {
        uint64_t hi = 0, lo = 0;  // words i - ws and i - ws - 1
#pragma unroll
        for (int j = 0; j < NW; ++j) {
            hi = (uint32_t)(i - j) == ws ? y[j] : hi;
            lo = (uint32_t)(i - j - 1) == ws ? y[j] : lo;
        }
        r.w[i] = (hi >> bs) | (bs ? lo << (64 - bs) : 0ULL);
    }
    return r;
}
template <int NW>
__device__ __forceinline__ void kshr2_put_dev(Key<NW>& x, uint32_t c, uint32_t k) {
#pragma unroll
    for (int i = NW - 1; i >= 0; --i) x.w[i] = (x.w[i] >> 2) | (i > 0 ? (x.w[i - 1] << 62) : 0ULL);
    const uint32_t pos = 2 * (k - 1), wd = NW - 1 - pos / 64;
#pragma unroll
    for (int i = 0; i < NW; ++i)
        if ((uint32_t)i == wd) x.w[i] |= (uint64_t)c << (pos % 64);
}
template <int NW>
__host__ __device__ __forceinline__ Key<NW> krc(const Key<NW>& x, uint32_t k) {
    Key<NW> r;
#pragma unroll
    for (int i = 0; i < NW; ++i) r.w[i] = 0;
    for (uint32_t i = 0; i < k; ++i) {
        // base i of rc = complement of base k-1-i of x
        const uint32_t c = 3u - kbase<NW>(x, k - 1 - i, k);
        const uint32_t pos = 2 * (k - 1 - i);
        r.w[NW - 1 - pos / 64] |= (uint64_t)c << (pos % 64);
    }
    return r;
}
template <int NW>
__host__ __device__ __forceinline__ bool kless(const Key<NW>& a, const Key<NW>& b) {
    for (int i = 0; i < NW; ++i)
        if (a.w[i] != b.w[i]) return a.w[i] < b.w[i];
    return false;
}
template <int NW>
__host__ __device__ __forceinline__ bool keq(const Key<NW>& a, const Key<NW>& b) {
    for (int i = 0; i < NW; ++i)
        if (a.w[i] != b.w[i]) return false;
    return true;
}
template <int NW>
__host__ __device__ __forceinline__ uint64_t kfold(const Key<NW>& a) {
    uint64_t f = 0;
    for (int i = 0; i < NW; ++i) f ^= a.w[i];
    return f;
}

struct Rows {
    const uint64_t* keys;
    const uint16_t* cov;
    const uint8_t* mask;
    uint64_t n;
    const uint32_t* idx;  // node index: row + 1, 0 = empty
    uint64_t cap;         // power of two
};

template <int NW>
__device__ __forceinline__ Key<NW> row_key(const Rows& R, uint64_t r) {
    Key<NW> x;
#pragma unroll
    for (int i = 0; i < NW; ++i) x.w[i] = R.keys[r * NW + i];
    return x;
}

template <int NW>
__device__ __forceinline__ int64_t find_row(const Rows& R, const Key<NW>& x) {
    uint64_t s = smix(kfold<NW>(x) ^ CIDX_SALT) & (R.cap - 1);
    for (uint64_t probe = 0; probe < R.cap; ++probe) {
        const uint32_t v = R.idx[s];
        if (v == 0) return -1;
        if (keq<NW>(row_key<NW>(R, v - 1), x)) return (int64_t)(v - 1);
        s = (s + 1) & (R.cap - 1);
    }
    return -1;
}

template <int NW>
__global__ void k_cidx_build(const uint64_t* __restrict__ keys, uint64_t n, uint32_t* idx, uint64_t cap, uint32_t* status) {
    for (uint64_t r = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; r < n; r += (uint64_t)gridDim.x * blockDim.x) {
        Key<NW> x;
#pragma unroll
        for (int i = 0; i < NW; ++i) x.w[i] = keys[r * NW + i];
        uint64_t s = smix(kfold<NW>(x) ^ CIDX_SALT) & (cap - 1);
        bool done = false;
        for (uint64_t probe = 0; probe < cap && !done; ++probe) {
            done = atomicCAS(&idx[s], 0u, (uint32_t)(r + 1)) == 0u;
            s = (s + 1) & (cap - 1);
        }
        if (!done) atomicOr(status, ST_TABLE_FULL);
    }
}

__device__ __forceinline__ uint32_t pc4(uint32_t v) { return __popc(v & 15u); }

__device__ __forceinline__ bool one_in_one_out(uint32_t m) { return pc4(m) == 1 && pc4(m >> 4) == 1; }

// Walk starts of a row: every out-edge of both directions of a boundary row.
__device__ __forceinline__ uint32_t starts_of(uint32_t m) { return one_in_one_out(m) ? 0u : pc4(m) + pc4(m >> 4); }

// Exclusive prefix sums of n values v(i), in tiles of 2048: the tiles' sums, then every tile's
// prefix from the sums before it.  pre[n] is the total.
constexpr uint32_t PRE_TILE = 2048;
template <class Fn>
__global__ void __launch_bounds__(256) k_tile_sums(Fn v, uint64_t n, uint64_t* __restrict__ part) {
    __shared__ uint64_t s[8];
    uint64_t t = 0;
    for (uint32_t j = 0; j < PRE_TILE / 256; ++j) {
        const uint64_t i = (uint64_t)blockIdx.x * PRE_TILE + j * 256 + threadIdx.x;
        if (i < n) t += v(i);
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) t += __shfl_down_sync(0xffffffffu, t, o);
    if ((threadIdx.x & 31) == 0) s[threadIdx.x >> 5] = t;
    __syncthreads();
    if (threadIdx.x == 0) {
        for (int j = 1; j < 8; ++j) t += s[j];
        part[blockIdx.x] = t;
    }
}
template <class Fn>
__global__ void __launch_bounds__(256) k_tile_prefix(Fn v, uint64_t n, const uint64_t* __restrict__ part, uint64_t* __restrict__ pre) {
    __shared__ uint64_t s[8], s_base;
    const uint32_t lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    uint64_t t = 0;
    for (uint32_t j = threadIdx.x; j < blockIdx.x; j += 256) t += part[j];
    __syncwarp();
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) t += __shfl_down_sync(0xffffffffu, t, o);
    if (lane == 0) s[w] = t;
    __syncthreads();
    if (threadIdx.x == 0) {
        for (int j = 1; j < 8; ++j) t += s[j];
        s_base = t;
    }
    __syncthreads();
    const uint64_t i0 = (uint64_t)blockIdx.x * PRE_TILE + threadIdx.x * 8;
    uint64_t x[8], sum = 0;
#pragma unroll
    for (int j = 0; j < 8; ++j) {
        x[j] = i0 + j < n ? v(i0 + j) : 0;
        sum += x[j];
    }
    uint64_t inc = sum;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint64_t y = __shfl_up_sync(0xffffffffu, inc, o);
        if (lane >= (uint32_t)o) inc += y;
    }
    if (lane == 31) s[w] = inc;
    __syncthreads();
    uint64_t p = s_base + inc - sum;
    for (uint32_t j = 0; j < w; ++j) p += s[j];
#pragma unroll
    for (int j = 0; j < 8; ++j) {
        if (i0 + j < n) pre[i0 + j] = p;
        p += x[j];
        if (i0 + j + 1 == n) pre[n] = p;
    }
}
struct StartCount {
    const uint8_t* mask;
    __device__ uint64_t operator()(uint64_t i) const { return starts_of(mask[i]); }
};
struct PathLength {
    const uint32_t* len;
    __device__ uint64_t operator()(uint64_t i) const { return len[i]; }
};

// Start list from the exclusive prefix of the counts: start = row << 4 | dir << 3 | edge.
__global__ void k_walk_starts(const uint8_t* __restrict__ mask, uint64_t n, const uint64_t* __restrict__ pre, uint64_t* starts) {
    for (uint64_t r = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; r < n; r += (uint64_t)gridDim.x * blockDim.x) {
        const uint32_t m = mask[r];
        if (one_in_one_out(m)) continue;
        uint64_t o = pre[r];
        for (uint32_t dir = 0; dir < 2; ++dir) {
            const uint32_t out = dir ? (m >> 4) & 15u : m & 15u;
            for (uint32_t b = 0; b < 4; ++b)
                if ((out >> b) & 1u) starts[o++] = (r << 4) | (dir << 3) | b;
        }
    }
}

// A directed node is row << 1 | direction (1: the reverse complement of the row's key).
constexpr uint32_t NO_NODE = 0xFFFFFFFFu;

// The k-mer of a directed node and its reverse complement, moved one base along edge b: the
// row it leads to (-1: none) and the direction in which that is entered.
template <int NW>
__device__ __forceinline__ int64_t take_edge(const Rows& R, uint32_t k, uint64_t row, uint32_t dir, uint32_t b, Key<NW>& f, Key<NW>& rv,
                                             uint32_t& rc_p, bool& c_rc) {
    const Key<NW> u = row_key<NW>(R, row), ur = krc_dev<NW>(u, k);
    f = dir ? ur : u;
    rv = dir ? u : ur;
    rc_p = 3u - kfirst<NW>(f, k);
    kshl2_push<NW>(f, b, k);
    kshr2_put_dev<NW>(rv, 3u - b, k);
    c_rc = kless<NW>(rv, f);
    return find_row<NW>(R, c_rc ? rv : f);
}
__device__ __forceinline__ uint32_t only_edge(uint32_t m, uint32_t dir) { return __ffs(dir ? (m >> 4) & 15u : m & 15u) - 1; }

// The successor of a directed 1-in-1-out node, where it is one too.
template <int NW>
__device__ __forceinline__ uint32_t next_node(const Rows& R, uint32_t k, uint32_t at) {
    const uint32_t m = R.mask[at >> 1];
    if (!one_in_one_out(m)) return NO_NODE;
    Key<NW> f, rv;
    uint32_t rc_p;
    bool c_rc;
    const int64_t r = take_edge<NW>(R, k, at >> 1, at & 1u, only_edge(m, at & 1u), f, rv, rc_p, c_rc);
    return r >= 0 && one_in_one_out(R.mask[r]) ? (uint32_t)(r << 1) | (c_rc ? 1u : 0u) : NO_NODE;
}
template <int NW>
__global__ void __launch_bounds__(256) k_next(Rows R, uint32_t k, uint32_t* __restrict__ next) {
    for (uint64_t s = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; s < 2 * R.n; s += (uint64_t)gridDim.x * blockDim.x)
        next[s] = next_node<NW>(R, k, (uint32_t)s);
}
// Table l + 1 from table l; any: whether an entry is left.
__global__ void __launch_bounds__(256) k_double(const uint32_t* __restrict__ in, uint32_t* __restrict__ out, uint64_t n, uint32_t* any) {
    bool some = false;
    for (uint64_t s = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; s < n; s += (uint64_t)gridDim.x * blockDim.x) {
        const uint32_t a = in[s], b = a == NO_NODE ? NO_NODE : in[a];
        out[s] = b;
        some |= b != NO_NODE;
    }
    if (__any_sync(0xffffffffu, some) && (threadIdx.x & 31) == 0) atomicOr(any, 1u);
}

// The tables there is memory for, the highest of them taken as often as need be; without any
// the successors are looked up one by one.
constexpr int MAX_TABLES = 33;
struct Jumps {
    const uint32_t* t[MAX_TABLES];  // t[l][s]: 2^l steps on from s
    int n;
};
template <int NW>
__device__ __forceinline__ uint32_t jump(const Rows& R, const Jumps& J, uint32_t k, int l, uint32_t at) {
    return J.n ? J.t[l][at] : next_node<NW>(R, k, at);
}

// The node d steps on from `at`, on a path that has it.
template <int NW>
__device__ __forceinline__ uint32_t steps_on(const Rows& R, const Jumps& J, uint32_t k, uint32_t at, uint32_t d) {
    const int top = J.n ? J.n - 1 : 0;
    for (uint32_t i = d >> top; i; --i) at = jump<NW>(R, J, k, top, at);
    for (int l = 0; l < top; ++l)
        if ((d >> l) & 1u) at = J.t[l][at];
    return at;
}

// A path (build.rs:349-445): its first 1-in-1-out node (NO_NODE: none), how many of them, and
// how it is stored: 0 as walked, 1 reverse complemented, 2 decided once it is written.
struct Path {
    uint32_t first, nodes, flip;
};
template <int NW>
__global__ void __launch_bounds__(256) k_paths(Rows R, Jumps J, uint32_t k, const uint64_t* __restrict__ starts, uint64_t n_starts,
                                               uint32_t* __restrict__ len_out, Path* __restrict__ paths, uint32_t* status) {
    for (uint64_t s = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; s < n_starts; s += (uint64_t)gridDim.x * blockDim.x) {
        const uint64_t start = starts[s];
        const uint64_t r0 = start >> 4;
        const uint32_t dir0 = (uint32_t)(start >> 3) & 1u;
        Key<NW> f, rv;
        uint32_t rc_p;
        bool c_rc;
        Key<NW> head = row_key<NW>(R, r0);
        if (dir0) head = krc_dev<NW>(head, k);
        int64_t r = take_edge<NW>(R, k, r0, dir0, (uint32_t)start & 7u, f, rv, rc_p, c_rc);
        Path p{NO_NODE, 0, 0};
        if (r >= 0 && one_in_one_out(R.mask[r])) {
            p.first = (uint32_t)(r << 1) | (c_rc ? 1u : 0u);
            uint32_t at = p.first;
            uint64_t nodes = 1;
            const int top = J.n ? J.n - 1 : 0;
            for (int l = top; l >= 0;) {
                const uint32_t nx = jump<NW>(R, J, k, l, at);
                if (nx != NO_NODE) {
                    at = nx;
                    nodes += 1ULL << l;
                }
                if (l < top || nx == NO_NODE || nodes > 2 * R.n) --l;
            }
            if (nodes > 2 * R.n) {  // more than there are directed nodes: impossible for valid rows
                atomicOr(status, ST_SPIN_TIMEOUT);
                nodes = 1;
            }
            p.nodes = (uint32_t)nodes;
            r = take_edge<NW>(R, k, at >> 1, at & 1u, only_edge(R.mask[at >> 1], at & 1u), f, rv, rc_p, c_rc);
        }
        bool keep = true;  // a path that ends at a k-mer with no node: no walk comes back
        if (r >= 0) {
            // boundary end: the walk from (r, !c_rc, rc_p) covers the same unitig
            const uint32_t m = R.mask[r], back = c_rc ? m & 15u : (m >> 4) & 15u;
            const uint64_t other = ((uint64_t)r << 4) | ((uint64_t)(c_rc ? 0u : 1u) << 3) | rc_p;
            if ((back >> rc_p) & 1u) keep = start <= other;
            if (start == other && p.nodes) {
                // its own reverse complement: past its middle every edge has been used already,
                // in the other direction, and the walk ends there (build.rs:349-445)
                p.nodes = (p.nodes + 1) / 2;
                const uint32_t at = steps_on<NW>(R, J, k, p.first, p.nodes - 1);
                take_edge<NW>(R, k, at >> 1, at & 1u, only_edge(R.mask[at >> 1], at & 1u), f, rv, rc_p, c_rc);
            }
        }
        // min(sequence, reverse complement) (build.rs:438-439): their first k bases decide
        p.flip = kless<NW>(rv, head) ? 1u : keq<NW>(rv, head) ? 2u : 0u;
        len_out[s] = keep ? k + 1 + p.nodes : 0;
        paths[s] = p;
    }
}

// Writes the kept paths' bases, marks their nodes and sums the coverage of the start and the
// 1-in-1-out nodes.  A thread takes 8 consecutive bases of the concatenated paths: it jumps
// to the node of its first one and steps on from there.
template <int NW>
__global__ void __launch_bounds__(256) k_path_bases(Rows R, Jumps J, uint32_t k, const uint64_t* __restrict__ starts, uint64_t n_starts,
                                                    const uint32_t* __restrict__ len, const uint64_t* __restrict__ off,
                                                    const Path* __restrict__ paths, uint64_t total, uint8_t* __restrict__ seqs,
                                                    uint8_t* __restrict__ visited, unsigned long long* __restrict__ cov) {
    for (uint64_t p0 = ((uint64_t)blockIdx.x * blockDim.x + threadIdx.x) * 8; p0 < total; p0 += (uint64_t)gridDim.x * blockDim.x * 8) {
        // the path of base p0: the last one that starts at or before it (paths not kept have
        // no bases and start where the next one does)
        uint64_t lo = 0, hi = n_starts;
        while (hi - lo > 1) {
            const uint64_t mid = (lo + hi) / 2;
            if (off[mid] <= p0) lo = mid;
            else hi = mid;
        }
        uint64_t s = lo;
        const uint64_t p1 = min(p0 + 8, total);
        uint64_t p = p0;
        while (p < p1) {
            while (!len[s] || off[s] + len[s] <= p) ++s;
            const uint32_t L = len[s];
            const uint64_t start = starts[s];
            const Path path = paths[s];
            const uint64_t end = min(p1, off[s] + L);
            uint32_t j = (uint32_t)(p - off[s]);
            uint32_t at = path.first;
            if (j > k) at = steps_on<NW>(R, J, k, at, j - k - 1);  // node j - k (1-based)
            unsigned long long c = 0;
            Key<NW> head;
            if (j < k) {
                head = row_key<NW>(R, start >> 4);
                if ((start >> 3) & 1u) head = krc_dev<NW>(head, k);
            }
            for (; p < end; ++p, ++j) {
                uint32_t b;
                if (j < k) {
                    const uint32_t pos = 2 * (k - 1 - j), wd = NW - 1 - pos / 64;
                    uint64_t v = 0;
#pragma unroll
                    for (int i = 0; i < NW; ++i) v = (uint32_t)i == wd ? head.w[i] : v;
                    b = (uint32_t)(v >> (pos % 64)) & 3u;
                } else if (j == k) {
                    b = (uint32_t)start & 7u;
                    c += R.cov[start >> 4];
                } else {
                    const uint32_t row = at >> 1;
                    b = only_edge(R.mask[row], at & 1u);
                    c += R.cov[row];
                    visited[row] = 1;
                    at = jump<NW>(R, J, k, 0, at);
                }
                seqs[off[s] + (path.flip == 1 ? L - 1 - j : j)] = "ACGT"[path.flip == 1 ? 3u - b : b];
            }
            if (c) atomicAdd(&cov[s], c);
        }
    }
}

// min(sequence, reverse complement), in place, for the paths whose first k bases left it open.
__global__ void k_canon_seq(uint8_t* seqs, const uint64_t* __restrict__ off, const uint32_t* __restrict__ len,
                            const Path* __restrict__ paths, uint64_t n) {
    for (uint64_t s = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; s < n; s += (uint64_t)gridDim.x * blockDim.x) {
        const uint64_t L = len[s];
        if (!L || paths[s].flip != 2) continue;
        uint8_t* q = seqs + off[s];
        auto comp = [](uint8_t c) -> uint8_t { return c == 'A' ? 'T' : c == 'C' ? 'G' : c == 'G' ? 'C' : 'A'; };
        int cmp = 0;
        for (uint64_t i = 0; i < L && !cmp; ++i) {
            const uint8_t a = comp(q[L - 1 - i]), b = q[i];
            cmp = a < b ? -1 : a > b ? 1 : 0;
        }
        if (cmp < 0) {
            for (uint64_t i = 0; i < L / 2; ++i) {
                const uint8_t a = q[i], b = q[L - 1 - i];
                q[i] = comp(b);
                q[L - 1 - i] = comp(a);
            }
            if (L & 1) q[L / 2] = comp(q[L / 2]);
        }
    }
}

// Rows that are 1-in-1-out and on no path: candidates for isolated cycles, and how many.
__global__ void k_cycle_candidates(const uint8_t* __restrict__ mask, const uint8_t* __restrict__ visited, uint64_t n, uint8_t* flag,
                                   unsigned long long* n_flag) {
    for (uint64_t r = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; r < n; r += (uint64_t)gridDim.x * blockDim.x) {
        const uint32_t m = mask[r];
        const bool f = !visited[r] && one_in_one_out(m);
        flag[r] = f ? 1 : 0;
        if (f) atomicAdd(n_flag, 1ULL);
    }
}

// ---- host side ---------------------------------------------------------------
struct HUnitig {
    std::string seq;
    float cov;
    bool circular;
};

template <int NW>
struct HKeyHash {
    size_t operator()(const std::array<uint64_t, NW>& a) const {
        uint64_t f = 0;
        for (int i = 0; i < NW; ++i) f ^= a[i];
        return (size_t)smix(f);
    }
};

// build.rs:450-555 over the candidate rows (host).
template <int NW>
void host_cycles(uint32_t k, const std::vector<uint64_t>& keys, const std::vector<uint16_t>& cov, const std::vector<uint8_t>& mask,
                 std::vector<HUnitig>& out) {
    using A = std::array<uint64_t, NW>;
    struct N {
        uint16_t cov;
        uint8_t mask, visited;
    };
    std::unordered_map<A, N, HKeyHash<NW>> map;
    std::vector<A> order;
    for (size_t i = 0; i < cov.size(); ++i) {
        A a;
        for (int j = 0; j < NW; ++j) a[j] = keys[i * NW + j];
        map[a] = N{cov[i], mask[i], 0};
        order.push_back(a);
    }
    auto toK = [](const A& a) {
        Key<NW> x;
        for (int j = 0; j < NW; ++j) x.w[j] = a[j];
        return x;
    };
    auto toA = [](const Key<NW>& x) {
        A a;
        for (int j = 0; j < NW; ++j) a[j] = x.w[j];
        return a;
    };
    for (const A& a : order) {
        auto it = map.find(a);
        const N n0 = it->second;
        const uint32_t fo = n0.mask & 15u, fi = (n0.mask >> 4) & 15u;
        if (__builtin_popcount(fo) != 1 || __builtin_popcount(fi) != 1) continue;
        const uint32_t b = __builtin_ctz(fo);
        if ((n0.visited >> b) & 1u) continue;
        it->second.visited |= (uint8_t)(1u << b);
        const Key<NW> start = toK(a);
        std::string path(k, 'A');
        for (uint32_t i = 0; i < k; ++i) path[i] = "ACGT"[kbase<NW>(start, i, k)];
        Key<NW> f = start, rv = krc<NW>(start, k);
        const uint32_t rc_first = 3u - kbase<NW>(f, 0, k);
        kshl2_push<NW>(f, b, k);
        kshr2_put<NW>(rv, 3u - b, k);
        bool c_rc = kless<NW>(rv, f);
        Key<NW> cur = c_rc ? rv : f;
        auto mark = [&](const Key<NW>& x, uint32_t bit) {
            auto m = map.find(toA(x));
            if (m != map.end()) m->second.visited |= (uint8_t)(1u << bit);
        };
        mark(cur, !c_rc ? rc_first + 4 : rc_first);
        path.push_back("ACGT"[b]);
        uint64_t total = n0.cov, points = 1;
        while (!keq<NW>(cur, start)) {
            auto m = map.find(toA(cur));
            if (m == map.end()) break;
            const N nc = m->second;
            const uint32_t c_out = !c_rc ? nc.mask & 15u : (nc.mask >> 4) & 15u;
            const uint32_t c_in = !c_rc ? (nc.mask >> 4) & 15u : nc.mask & 15u;
            if (__builtin_popcount(c_in) != 1 || __builtin_popcount(c_out) != 1) break;
            const uint32_t nb = __builtin_ctz(c_out);
            const uint32_t ebit = !c_rc ? nb : nb + 4;
            if ((nc.visited >> ebit) & 1u) break;
            m->second.visited |= (uint8_t)(1u << ebit);
            const uint32_t rc_p = 3u - kbase<NW>(f, 0, k);
            kshl2_push<NW>(f, nb, k);
            kshr2_put<NW>(rv, 3u - nb, k);
            c_rc = kless<NW>(rv, f);
            cur = c_rc ? rv : f;
            mark(cur, !c_rc ? rc_p + 4 : rc_p);
            path.push_back("ACGT"[nb]);
            total += nc.cov;
            points++;
        }
        if (keq<NW>(cur, start) && path.size() > k) {
            if (path.compare(path.size() - k, k, path, 0, k) == 0) path.resize(path.size() - k);
            else if (path.compare(path.size() - (k - 1), k - 1, path, 0, k - 1) == 0) path.resize(path.size() - (k - 1));
            out.push_back(HUnitig{path, std::max(1.0f, (float)total / (float)points), true});
        }
    }
}

std::string rc_string(const std::string& s) {
    std::string r(s.size(), 'A');
    for (size_t i = 0; i < s.size(); ++i) {
        const char c = s[s.size() - 1 - i];
        r[i] = c == 'A' ? 'T' : c == 'C' ? 'G' : c == 'G' ? 'C' : 'A';
    }
    return r;
}

}  // namespace

struct fbk_unitigs {
    std::vector<HUnitig> u;
    // edges: from id, from side (0 forward, 1 reverse strand), to id, to rc, overlap, support
    std::vector<std::array<uint32_t, 6>> edges;
    uint64_t bases = 0, linear_walks = 0, cycle_candidates = 0;
};

namespace {

// build.rs:557-594: edges by exact k and k-1 overlap; cdbg.rs:113-122 merges repeats.
void link_unitigs(uint32_t k, fbk_unitigs* U) {
    const uint32_t n = (uint32_t)U->u.size();
    std::vector<std::vector<std::array<uint32_t, 4>>> side[2];
    side[0].resize(n);
    side[1].resize(n);
    auto add = [&](uint32_t id, int s, uint32_t t, uint32_t trc, uint32_t ov, uint32_t sup) {
        for (auto& e : side[s][id])
            if (e[0] == t && e[1] == trc && e[2] == ov) {
                e[3] = std::min<uint32_t>(65535, e[3] + sup);
                return;
            }
        side[s][id].push_back({t, trc, ov, sup});
    };
    for (uint32_t id = 0; id < n; ++id)
        if (U->u[id].circular) add(id, 0, id, 0, k - 1, 10);  // build.rs:546-547
    for (uint32_t ov : {k, k - 1}) {
        if (ov == 0) continue;
        // an end of the reverse complement is the complement of the other end: the whole of it
        // is never needed
        std::unordered_map<std::string, std::vector<std::pair<uint32_t, uint32_t>>> prefix;
        prefix.reserve(2 * (size_t)n);
        std::vector<std::string> tail[2];  // last ov bases of both strands
        tail[0].resize(n);
        tail[1].resize(n);
        for (uint32_t id = 0; id < n; ++id) {
            const std::string& f = U->u[id].seq;
            if (f.size() < ov) continue;
            const std::string head = f.substr(0, ov);
            tail[0][id] = f.substr(f.size() - ov);
            tail[1][id] = rc_string(head);
            prefix[head].push_back({id, 0});
            prefix[rc_string(tail[0][id])].push_back({id, 1});
        }
        for (uint32_t id = 0; id < n; ++id) {
            if (U->u[id].seq.size() < ov) continue;
            for (int s = 0; s < 2; ++s) {
                auto a = prefix.find(tail[s][id]);
                if (a == prefix.end()) continue;
                for (auto& t : a->second)
                    if (t.first != id || U->u[id].circular) add(id, s, t.first, t.second, ov, 10);
            }
        }
    }
    for (uint32_t id = 0; id < n; ++id)
        for (int s = 0; s < 2; ++s)
            for (auto& e : side[s][id]) U->edges.push_back({id, (uint32_t)s, e[0], e[1], e[2], e[3]});
}

template <int NW>
fbk_status compact_impl(fbk_table* t, fbk_unitigs* U) {
    fbk_ctx* ctx = t->ctx;
    const uint64_t n = t->n_solid;
    const uint32_t k = t->k;
    if (k < 2) return set_err(ctx, FBK_ERR_INVALID, "compaction needs k >= 2");
    if (n == 0) return FBK_OK;
    if (n >= (1ULL << 31)) return set_err(ctx, FBK_ERR_INVALID, "compaction: more than 2^31 solid rows");
    Launch L = launch_cfg(ctx, 256, 0);
    uint64_t cap = 1;
    while (cap < 2 * n) cap <<= 1;
    Jumps J{};
    struct Bufs {
        fbk_ctx* c;
        Jumps* J;
        std::vector<void*> p;
        // where memory is short the highest tables make room: the paths are found with fewer
        void* get(uint64_t b) {
            void* q = dev_alloc(c, b);
            while (!q && J->n) {
                void* t = (void*)J->t[--J->n];
                p.erase(std::find(p.begin(), p.end(), t));
                cudaStreamSynchronize(c->stream);
                dev_free(c, t);
                q = dev_alloc(c, b);
            }
            if (q) p.push_back(q);
            return q;
        }
        uint32_t* table(uint64_t b) {
            void* q = dev_alloc(c, b);
            if (q) p.push_back(q);
            return (uint32_t*)q;
        }
        ~Bufs() {
            cudaStreamSynchronize(c->stream);
            for (void* q : p) dev_free(c, q);
        }
    } B{ctx, &J, {}};
    uint32_t* idx = (uint32_t*)B.get(cap * 4);
    uint8_t* visited = (uint8_t*)B.get(n);
    uint64_t* pre = (uint64_t*)B.get((n + 1) * 8);
    const uint64_t tiles = (n + PRE_TILE - 1) / PRE_TILE;
    uint64_t* part = (uint64_t*)B.get(tiles * 8);
    uint32_t* any = (uint32_t*)B.get(4 * MAX_TABLES);
    uint8_t* flag = (uint8_t*)B.get(n);
    if (!idx || !visited || !pre || !part || !any || !flag) return set_err(ctx, FBK_ERR_OOM, "compaction index");
    CK(ctx, cudaMemsetAsync(idx, 0, cap * 4, ctx->stream));
    CK(ctx, cudaMemsetAsync(visited, 0, n, ctx->stream));
    CK(ctx, cudaMemsetAsync(any, 0, 4 * MAX_TABLES, ctx->stream));
    CK(ctx, cudaMemsetAsync(ctx->d_status, 0, 4, ctx->stream));
    CK(ctx, cudaMemsetAsync(ctx->d_counts, 0, 8, ctx->stream));
    Rows R{t->out_keys, t->out_cov, t->out_mask, n, idx, cap};
    TIMED(ctx, "compact_index", (k_cidx_build<NW><<<L.grid, L.block, 0, ctx->stream>>>(t->out_keys, n, idx, cap, ctx->d_status),
                                 cudaGetLastError()));
    TIMED(ctx, "compact_count", (k_tile_sums<<<(unsigned)tiles, 256, 0, ctx->stream>>>(StartCount{t->out_mask}, n, part), cudaGetLastError()));
    TIMED(ctx, "compact_count", (k_tile_prefix<<<(unsigned)tiles, 256, 0, ctx->stream>>>(StartCount{t->out_mask}, n, part, pre), cudaGetLastError()));
    uint64_t* h = (uint64_t*)ctx->h_pinned;
    CK(ctx, cudaMemcpyAsync(h, pre + n, 8, cudaMemcpyDeviceToHost, ctx->stream));
    // Tables until none of their entries is left (a path of 2^l nodes needs l + 1 of them; an
    // isolated cycle never runs out, so there are at most as many as the nodes can fill), or
    // there is no path, or no memory for more: 8 bytes a row each, of at most half of what a
    // pool has free, which other contexts may share.  The host looks after every four.
    uint64_t room = ~0ULL, largest = 0;
    if (ctx->pool && ctx->pool->active()) fbk_ctx_pool_free(ctx, &room, &largest), room /= 2;
    for (bool more = true; more;) {
        for (int q = J.n ? 0 : -1; q < 4 && more; ++q) {
            uint32_t* up = nullptr;
            if ((J.n == 0 || (1ULL << (J.n - 1)) <= n) && room >= 8 * n * (J.n + 1ULL)) up = B.table(8 * n);
            more = up != nullptr;
            if (!up) break;
            if (J.n == 0) {
                TIMED(ctx, "compact_next", (k_next<NW><<<L.grid, L.block, 0, ctx->stream>>>(R, k, up), cudaGetLastError()));
            } else {
                TIMED(ctx, "compact_next", (k_double<<<L.grid, L.block, 0, ctx->stream>>>(J.t[J.n - 1], up, 2 * n, any + J.n),
                                            cudaGetLastError()));
            }
            J.t[J.n++] = up;
        }
        if (more) CK(ctx, cudaMemcpyAsync(h + 1, any + J.n - 1, 4, cudaMemcpyDeviceToHost, ctx->stream));
        CK(ctx, cudaStreamSynchronize(ctx->stream));
        more = more && h[0] && *(uint32_t*)(h + 1) != 0;
    }
    const uint64_t n_starts = h[0];
    U->linear_walks = n_starts;
    std::vector<uint32_t> hlen(n_starts);
    std::vector<uint64_t> hoff(n_starts);
    std::vector<unsigned long long> hcs(n_starts);
    std::vector<uint8_t> hseq;
    uint64_t total = 0;
    if (n_starts) {
        const uint64_t st_tiles = (n_starts + PRE_TILE - 1) / PRE_TILE;
        uint64_t* starts = (uint64_t*)B.get(n_starts * 8);
        uint32_t* len = (uint32_t*)B.get(n_starts * 4);
        Path* paths = (Path*)B.get(n_starts * sizeof(Path));
        unsigned long long* cs = (unsigned long long*)B.get(n_starts * 8);
        uint64_t* off = (uint64_t*)B.get((n_starts + 1) * 8);
        uint64_t* st_part = (uint64_t*)B.get(st_tiles * 8);
        if (!starts || !len || !paths || !cs || !off || !st_part) return set_err(ctx, FBK_ERR_OOM, "compaction walks");
        CK(ctx, cudaMemsetAsync(cs, 0, n_starts * 8, ctx->stream));
        TIMED(ctx, "compact_starts", (k_walk_starts<<<L.grid, L.block, 0, ctx->stream>>>(t->out_mask, n, pre, starts), cudaGetLastError()));
        TIMED(ctx, "compact_walk", (k_paths<NW><<<L.grid, L.block, 0, ctx->stream>>>(R, J, k, starts, n_starts, len, paths, ctx->d_status),
                                    cudaGetLastError()));
        TIMED(ctx, "compact_walk", (k_tile_sums<<<(unsigned)st_tiles, 256, 0, ctx->stream>>>(PathLength{len}, n_starts, st_part), cudaGetLastError()));
        TIMED(ctx, "compact_walk", (k_tile_prefix<<<(unsigned)st_tiles, 256, 0, ctx->stream>>>(PathLength{len}, n_starts, st_part, off),
                                    cudaGetLastError()));
        CK(ctx, cudaMemcpyAsync(h, off + n_starts, 8, cudaMemcpyDeviceToHost, ctx->stream));
        CK(ctx, cudaMemcpyAsync(h + 1, ctx->d_status, 4, cudaMemcpyDeviceToHost, ctx->stream));
        CK(ctx, cudaStreamSynchronize(ctx->stream));
        total = h[0];
        if ((uint32_t)h[1]) return set_err(ctx, FBK_ERR_INVALID, "compaction: node index full or a path of more nodes than there are");
        uint8_t* seqs = (uint8_t*)B.get(std::max<uint64_t>(total, 1));
        if (!seqs) return set_err(ctx, FBK_ERR_OOM, "compaction sequences");
        if (total)
            TIMED(ctx, "compact_write", (k_path_bases<NW><<<L.grid, L.block, 0, ctx->stream>>>(R, J, k, starts, n_starts, len, off, paths, total,
                                                                                               seqs, visited, cs),
                                         cudaGetLastError()));
        TIMED(ctx, "compact_canon", (k_canon_seq<<<L.grid, L.block, 0, ctx->stream>>>(seqs, off, len, paths, n_starts), cudaGetLastError()));
        hseq.resize(total);
        CK(ctx, cudaMemcpyAsync(hlen.data(), len, n_starts * 4, cudaMemcpyDeviceToHost, ctx->stream));
        CK(ctx, cudaMemcpyAsync(hoff.data(), off, n_starts * 8, cudaMemcpyDeviceToHost, ctx->stream));
        CK(ctx, cudaMemcpyAsync(hcs.data(), cs, n_starts * 8, cudaMemcpyDeviceToHost, ctx->stream));
        if (total) CK(ctx, copy_d2h(ctx, hseq.data(), seqs, total));
    }
    // isolated cycles: candidate rows to the host, if there are any
    TIMED(ctx, "compact_cycles", (k_cycle_candidates<<<L.grid, L.block, 0, ctx->stream>>>(t->out_mask, visited, n, flag, ctx->d_counts),
                                  cudaGetLastError()));
    CK(ctx, cudaMemcpyAsync(h, ctx->d_counts, 8, cudaMemcpyDeviceToHost, ctx->stream));
    CK(ctx, cudaStreamSynchronize(ctx->stream));
    std::vector<uint8_t> hflag;
    if (h[0]) {
        hflag.resize(n);
        CK(ctx, cudaMemcpyAsync(hflag.data(), flag, n, cudaMemcpyDeviceToHost, ctx->stream));
        CK(ctx, cudaStreamSynchronize(ctx->stream));
    }
    for (uint64_t s = 0; s < n_starts; ++s) {
        if (!hlen[s]) continue;
        HUnitig u;
        u.seq.assign((const char*)hseq.data() + hoff[s], hlen[s]);
        u.cov = std::max(1.0f, (float)hcs[s] / (float)(hlen[s] - k));  // the start and the nodes: k + 1 + nodes bases
        u.circular = false;
        U->bases += hlen[s];
        U->u.push_back(std::move(u));
    }
    std::vector<uint64_t> ck;
    std::vector<uint16_t> cc;
    std::vector<uint8_t> cm;
    std::vector<uint64_t> rows;
    for (uint64_t r = 0; r < hflag.size(); ++r)
        if (hflag[r]) rows.push_back(r);
    U->cycle_candidates = rows.size();
    if (!rows.empty()) {
        // the candidates are gathered from a host copy of the rows (cycles are rare)
        std::vector<uint64_t> all_k(n * NW);
        std::vector<uint16_t> all_c(n);
        std::vector<uint8_t> all_m(n);
        CK(ctx, cudaMemcpyAsync(all_k.data(), t->out_keys, n * 8 * NW, cudaMemcpyDeviceToHost, ctx->stream));
        CK(ctx, cudaMemcpyAsync(all_c.data(), t->out_cov, n * 2, cudaMemcpyDeviceToHost, ctx->stream));
        CK(ctx, cudaMemcpyAsync(all_m.data(), t->out_mask, n, cudaMemcpyDeviceToHost, ctx->stream));
        CK(ctx, cudaStreamSynchronize(ctx->stream));
        ck.resize(rows.size() * NW);
        cc.resize(rows.size());
        cm.resize(rows.size());
        for (size_t i = 0; i < rows.size(); ++i) {
            for (int j = 0; j < NW; ++j) ck[i * NW + j] = all_k[rows[i] * NW + j];
            cc[i] = all_c[rows[i]];
            cm[i] = all_m[rows[i]];
        }
        const size_t before = U->u.size();
        host_cycles<NW>(k, ck, cc, cm, U->u);
        for (size_t i = before; i < U->u.size(); ++i) U->bases += U->u[i].seq.size();
    }
    link_unitigs(k, U);
    return FBK_OK;
}

}  // namespace

extern "C" {

FBK_API fbk_status fbk_compact(fbk_table* t, fbk_unitigs** out) {
    if (!t || !out) return FBK_ERR_INVALID;
    *out = nullptr;
    fbk_ctx* ctx = t->ctx;
    CK(ctx, cudaSetDevice(ctx->device));
    auto* U = new fbk_unitigs();
    fbk_status st = t->nw == 1 ? compact_impl<1>(t, U) : t->nw == 2 ? compact_impl<2>(t, U) : compact_impl<4>(t, U);
    if (st) {
        delete U;
        return st;
    }
    *out = U;
    return FBK_OK;
}

FBK_API fbk_status fbk_unitigs_info(const fbk_unitigs* u, uint64_t* n_unitigs, uint64_t* total_bases, uint64_t* n_edges) {
    if (!u) return FBK_ERR_INVALID;
    if (n_unitigs) *n_unitigs = u->u.size();
    if (total_bases) *total_bases = u->bases;
    if (n_edges) *n_edges = u->edges.size();
    return FBK_OK;
}

FBK_API fbk_status fbk_unitigs_export(const fbk_unitigs* u, uint8_t* ascii, uint64_t* offsets, float* cov, uint8_t* circular) {
    if (!u || !offsets) return FBK_ERR_INVALID;
    uint64_t p = 0;
    offsets[0] = 0;
    for (size_t i = 0; i < u->u.size(); ++i) {
        if (ascii) memcpy(ascii + p, u->u[i].seq.data(), u->u[i].seq.size());
        p += u->u[i].seq.size();
        offsets[i + 1] = p;
        if (cov) cov[i] = u->u[i].cov;
        if (circular) circular[i] = u->u[i].circular;
    }
    return FBK_OK;
}

FBK_API fbk_status fbk_unitigs_edges(const fbk_unitigs* u, uint32_t* edges, uint64_t cap, uint64_t* n_out) {
    if (!u || !n_out) return FBK_ERR_INVALID;
    const uint64_t n = std::min<uint64_t>(cap, u->edges.size());
    if (n && !edges) return FBK_ERR_INVALID;
    for (uint64_t i = 0; i < n; ++i) memcpy(edges + 6 * i, u->edges[i].data(), 24);
    *n_out = u->edges.size();
    return FBK_OK;
}

FBK_API fbk_status fbk_unitigs_release(fbk_unitigs* u) {
    delete u;
    return FBK_OK;
}

}  // extern "C"
