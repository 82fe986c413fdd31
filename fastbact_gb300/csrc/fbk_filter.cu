// fbk_filter.cu — the multi-k upgrade's input filter (src/graph/local_multik.rs:259-333)
// on the device.
//
// filter_active_reads keeps the reads that touch unitig ends, branching junctions
// or unresolved regions: it indexes the canonical ntHash (k' = min(k, 31)) of every
// k'-mer of short (< 2000 bp), circular or branching unitigs and of the first and
// last 350 k'-mers of the other unitigs, then keeps a read when the ntHash at offset
// 0, (len - k') / 2 or len - k' is indexed; a pair is kept when either read is.
// Here the unitigs are packed on the device, the index is an open-addressing set of u64
// hashes that the windows of the packed unitigs are entered into, and one thread tests a
// merged read or a pair of the device bank and writes its keep bytes.
#include <algorithm>
#include <vector>

#include "fbk_device.cuh"
#include "fbk_internal.h"

using namespace fbk;

namespace {

constexpr uint64_t HSET_EMPTY = ~0ULL;

// ASCII to packed words (ASCII_TO_2BIT: A0 C1 G2 T3, anything else 0), one word a thread; words
// past the bases are zero.
__global__ void __launch_bounds__(256) k_pack_ascii(const uint8_t* __restrict__ t, uint64_t n, uint64_t* __restrict__ words, uint64_t n_words) {
    const uint64_t w = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (w >= n_words) return;
    uint64_t x = 0;
    for (uint32_t j = 0; j < 32 && w * 32 + j < n; ++j) {
        const uint8_t c = t[w * 32 + j] & 0xDF;
        x |= (uint64_t)(c == 'C' ? 1 : c == 'G' ? 2 : c == 'T' ? 3 : 0) << (2 * j);
    }
    words[w] = x;
}

constexpr uint64_t FILTER_WINDOW = 350, FILTER_LONG = 2000;
// The indexed windows of a unitig of len bases: [0, left) and [right, len - k + 1).
struct FilterSpan {
    uint64_t left, right, n;
};
__host__ __device__ __forceinline__ FilterSpan filter_span(uint64_t len, uint32_t k, bool circular, uint32_t fwd, uint32_t rev) {
    FilterSpan f{0, 0, 0};
    if (len < k) return f;
    const uint64_t nk = len - k + 1;
    f.n = nk;
    if (len < FILTER_LONG || circular || fwd > 1 || rev > 1) return f;
    f.left = nk < FILTER_WINDOW ? nk : FILTER_WINDOW;
    f.right = len - FILTER_WINDOW < len - k ? len - FILTER_WINDOW : len - k;
    return f;
}

// A thread takes FILTER_RUN places of the packed unitigs, finds the unitig of the first one by
// bisection and rolls the hash along the windows there that are indexed.  Bound by the set's
// CAS (random 8-byte accesses in L2).  The host packed base by base and listed the windows
// (8 bytes each, copied over) before: the whole call took 6.5 ms for a 1 Mbp graph at 50x and
// takes 0.39.
constexpr uint32_t FILTER_RUN = 8;
__global__ void __launch_bounds__(256) k_hset_insert(const uint64_t* __restrict__ data, uint64_t n_bases, const uint64_t* __restrict__ uoff,
                                                     const uint8_t* __restrict__ circular, const uint32_t* __restrict__ fwd,
                                                     const uint32_t* __restrict__ rev, uint64_t n_unitigs, uint32_t k,
                                                     unsigned long long* set, uint64_t cap, uint32_t* flags) {
    for (uint64_t t = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; t * FILTER_RUN < n_bases; t += (uint64_t)gridDim.x * blockDim.x) {
        uint64_t g = t * FILTER_RUN;
        const uint64_t end = min(g + FILTER_RUN, n_bases);
        uint64_t lo = 0, hi = n_unitigs;  // the last unitig that begins at g or before
        while (hi - lo > 1) {
            const uint64_t mid = (lo + hi) / 2;
            if (uoff[mid] - uoff[0] <= g) lo = mid;
            else hi = mid;
        }
        for (uint64_t u = lo; u < n_unitigs && g < end; ++u) {
            const uint64_t a = uoff[u] - uoff[0], e = uoff[u + 1] - uoff[0];
            const FilterSpan f = filter_span(e - a, k, circular[u], fwd[u], rev[u]);
            const uint64_t stop = min(end, e);
            auto enter = [&](uint64_t from, uint64_t to) {  // windows of the unitig
                from = max(from, g - a);
                to = min(to, stop - a);
                if (from >= to) return;
                nthash_run(data, a + from, k, 0, (uint32_t)(to - from), [&](uint32_t, uint64_t h) {
                    if (h == HSET_EMPTY) {  // the one value the set cannot hold is kept as a flag
                        atomicOr(flags, 1u);
                        return;
                    }
                    uint64_t s = smix(h) & (cap - 1);
                    for (uint64_t probe = 0; probe < cap; ++probe) {
                        const unsigned long long old = atomicCAS(&set[s], HSET_EMPTY, (unsigned long long)h);
                        if (old == HSET_EMPTY || old == h) break;
                        s = (s + 1) & (cap - 1);
                    }
                });
            };
            enter(0, f.left);
            enter(max(f.left, f.right), f.n);
            g = max(g, stop);
        }
    }
}

__device__ __forceinline__ bool hset_has(const unsigned long long* set, uint64_t cap, uint32_t flags, uint64_t h) {
    if (h == HSET_EMPTY) return flags & 1u;
    uint64_t s = smix(h) & (cap - 1);
    for (uint64_t probe = 0; probe < cap; ++probe) {
        const uint64_t v = set[s];
        if (v == h) return true;
        if (v == HSET_EMPTY) return false;
        s = (s + 1) & (cap - 1);
    }
    return false;
}

// local_multik.rs:296-307: ntHash at offsets 0, (len - k) / 2 and len - k.
__device__ __forceinline__ bool read_active(const BankDev& b, uint64_t r, uint32_t k, const unsigned long long* set, uint64_t cap, uint32_t fl) {
    const uint32_t len = b.len[r];
    bool a = false;
    if (len >= k) {
        const uint64_t off = b.off[r];
        const uint32_t offs[3] = {0u, (len - k) / 2, len - k};
        for (int j = 0; j < 3 && !a; ++j) a = hset_has(set, cap, fl, nthash_canonical_at(b.data, off + offs[j], k));
    }
    return a;
}
// local_multik.rs:309-329: merged reads (M) on their own, the pairs of the other two arenas (F
// and R reads) together; a read without a mate is not kept.
__global__ void __launch_bounds__(256) k_active_reads(BankDev b, uint64_t M, uint64_t F, uint64_t R, uint32_t k,
                                                      const unsigned long long* __restrict__ set, uint64_t cap,
                                                      const uint32_t* __restrict__ flags, uint8_t* __restrict__ keep,
                                                      unsigned long long* __restrict__ n_kept) {
    const uint32_t fl = *flags;
    uint32_t kept = 0;
    for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < M + max(F, R); i += (uint64_t)gridDim.x * blockDim.x) {
        if (i < M) {
            kept += keep[i] = read_active(b, i, k, set, cap, fl);
            continue;
        }
        const uint64_t j = i - M;
        const bool a = j < min(F, R) && (read_active(b, i, k, set, cap, fl) || read_active(b, i + F, k, set, cap, fl));
        if (j < F) keep[i] = a;
        if (j < R) keep[i + F] = a;
        kept += 2 * a;
    }
    kept = __reduce_add_sync(0xffffffffu, kept);
    if ((threadIdx.x & 31) == 0 && kept) atomicAdd(n_kept, (unsigned long long)kept);
}

struct Bufs {
    fbk_ctx* c;
    std::vector<void*> p;
    void* get(uint64_t b) {
        void* q = dev_alloc(c, std::max<uint64_t>(b, 8));
        if (q) p.push_back(q);
        return q;
    }
    ~Bufs() {
        cudaStreamSynchronize(c->stream);
        for (void* q : p) dev_free(c, q);
    }
};

// The bases of the unitigs back to back in packed words on the device (8 words of zeros after
// them).
fbk_status pack_unitigs(fbk_ctx* ctx, Bufs& B, const uint8_t* ascii, const uint64_t* offsets, uint64_t n_unitigs, uint64_t** words) {
    for (uint64_t u = 0; u < n_unitigs; ++u)
        if (offsets[u + 1] < offsets[u]) return set_err(ctx, FBK_ERR_INVALID, "unitig offsets must not fall");
    const uint64_t n = n_unitigs ? offsets[n_unitigs] - offsets[0] : 0, n_words = (n + 31) / 32 + 8;
    uint8_t* text = (uint8_t*)B.get(n);
    *words = (uint64_t*)B.get(n_words * 8);
    if (!text || !*words) return set_err(ctx, FBK_ERR_OOM, "packed unitigs");
    if (n) CK(ctx, copy_h2d(ctx, text, ascii + offsets[0], n));
    TIMED(ctx, "unitig_pack", (k_pack_ascii<<<(unsigned)((n_words + 255) / 256), 256, 0, ctx->stream>>>(text, n, *words, n_words),
                               cudaGetLastError()));
    return FBK_OK;
}

}  // namespace

extern "C" {

FBK_API fbk_status fbk_filter_active_reads(fbk_ctx* ctx, const fbk_bank* bank, const uint8_t* unitig_ascii,
                                           const uint64_t* unitig_offsets, const uint8_t* circular, const uint32_t* edges_fwd,
                                           const uint32_t* edges_rev, uint64_t n_unitigs, uint32_t graph_k, uint8_t* keep_out,
                                           uint64_t* n_kept) {
    if (!ctx || !bank || !unitig_offsets || !keep_out || (n_unitigs && (!unitig_ascii || !circular || !edges_fwd || !edges_rev)))
        return FBK_ERR_INVALID;
    if (bank->arena_reads.size() != 3) return set_err(ctx, FBK_ERR_INVALID, "filter_active_reads needs a three-arena ReadBank");
    if (graph_k < 1) return set_err(ctx, FBK_ERR_INVALID, "graph k must be >= 1");
    CK(ctx, cudaSetDevice(ctx->device));
    CK(ctx, bank_wait(ctx, bank));
    const uint32_t k = std::min<uint32_t>(graph_k, 31);
    const uint64_t M = bank->arena_reads[0], F = bank->arena_reads[1], R = bank->arena_reads[2], n_reads = M + F + R;
    Bufs B{ctx, {}};
    uint64_t* d_words = nullptr;
    fbk_status st = pack_unitigs(ctx, B, unitig_ascii, unitig_offsets, n_unitigs, &d_words);
    if (st) return st;
    uint64_t n_win = 0;
    for (uint64_t u = 0; u < n_unitigs; ++u) {
        const FilterSpan f = filter_span(unitig_offsets[u + 1] - unitig_offsets[u], k, circular[u], edges_fwd[u], edges_rev[u]);
        n_win += f.left + f.n - std::max(f.left, f.right);
    }
    uint64_t cap = 1024;
    while (cap < 2 * n_win) cap <<= 1;
    uint64_t* d_off = (uint64_t*)B.get((n_unitigs + 1) * 8);
    uint8_t* d_circ = (uint8_t*)B.get(n_unitigs);
    uint32_t* d_fwd = (uint32_t*)B.get(n_unitigs * 4);
    uint32_t* d_rev = (uint32_t*)B.get(n_unitigs * 4);
    unsigned long long* set = (unsigned long long*)B.get(cap * 8);
    unsigned long long* d_kept = (unsigned long long*)B.get(16);
    uint8_t* keep = (uint8_t*)B.get(n_reads);
    if (!d_off || !d_circ || !d_fwd || !d_rev || !set || !d_kept || !keep) return set_err(ctx, FBK_ERR_OOM, "filter_active_reads buffers");
    uint32_t* flags = (uint32_t*)(d_kept + 1);
    CK(ctx, cudaMemsetAsync(d_kept, 0, 16, ctx->stream));
    Launch L = launch_cfg(ctx, 256, 0);
    CK(ctx, cudaMemsetAsync(set, 0xFF, cap * 8, ctx->stream));
    if (n_win) {
        CK(ctx, copy_h2d(ctx, d_off, unitig_offsets, (n_unitigs + 1) * 8));
        CK(ctx, copy_h2d(ctx, d_circ, circular, n_unitigs));
        CK(ctx, copy_h2d(ctx, d_fwd, edges_fwd, n_unitigs * 4));
        CK(ctx, copy_h2d(ctx, d_rev, edges_rev, n_unitigs * 4));
        TIMED(ctx, "filter_index", (k_hset_insert<<<L.grid, L.block, 0, L.stream>>>(d_words, unitig_offsets[n_unitigs] - unitig_offsets[0],
                                                                                   d_off, d_circ, d_fwd, d_rev, n_unitigs, k, set, cap, flags),
                                    cudaGetLastError()));
    }
    uint64_t kept = 0;
    if (n_reads) {
        TIMED(ctx, "filter_reads", (k_active_reads<<<L.grid, L.block, 0, L.stream>>>(bank_view(bank, 0, bank->n_reads, nullptr), M, F, R, k,
                                                                                    set, cap, flags, keep, d_kept),
                                    cudaGetLastError()));
        CK(ctx, cudaMemcpyAsync(ctx->h_pinned, d_kept, 8, cudaMemcpyDeviceToHost, ctx->stream));
        CK(ctx, copy_d2h(ctx, keep_out, keep, n_reads));
        CK(ctx, cudaStreamSynchronize(ctx->stream));
        kept = *(const unsigned long long*)ctx->h_pinned;
    }
    if (n_kept) *n_kept = kept;
    return FBK_OK;
}

}  // extern "C"

// ===========================================================================
// index_terminal_kmers (src/resolve/mapper.rs:89-136): the canonical k-mers (folded to
// u64, KmerInt::to_u64) of the first and last 1000 k-mers of every unitig (all of them
// when it has at most 2000), kept when they occur exactly once, with the unitig strand
// (DirUnitigId(id, is_rc)) and the k-mer's position.  A device map counts every key;
// the value written by a key's only occurrence is the one kept.
// ===========================================================================
namespace {

struct TermWindow {
    uint64_t g;     // first base in the packed unitigs
    uint32_t unitig, pos;
};

template <int NW>
__global__ void k_term_insert(const uint64_t* __restrict__ data, const TermWindow* __restrict__ win, uint64_t n_win, uint32_t k,
                              unsigned long long* keys, uint32_t* cnt, uint64_t* vals, uint64_t cap, unsigned long long* full_fold) {
    for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n_win; i += (uint64_t)gridDim.x * blockDim.x) {
        const TermWindow w = win[i];
        Key<NW> can;
        bool rc;
        window_canonical<NW>(data, w.g, k, can, rc);
        const uint64_t h = key_fold<NW>(can);
        const uint64_t v = ((uint64_t)w.unitig << 33) | ((uint64_t)(rc ? 1 : 0) << 32) | w.pos;
        if (h == HSET_EMPTY) {  // the fold the map cannot hold as a key: counted in slot 0 of full_fold
            atomicAdd(&full_fold[0], 1ULL);
            full_fold[1] = v;
            continue;
        }
        uint64_t s = smix(h) & (cap - 1);
        for (uint64_t probe = 0; probe < cap; ++probe) {
            const unsigned long long old = atomicCAS(&keys[s], HSET_EMPTY, (unsigned long long)h);
            if (old == HSET_EMPTY || old == h) {
                atomicAdd(&cnt[s], 1u);
                vals[s] = v;
                break;
            }
            s = (s + 1) & (cap - 1);
        }
    }
}

}  // namespace

extern "C" {

FBK_API fbk_status fbk_index_terminal_kmers(fbk_ctx* ctx, const uint8_t* unitig_ascii, const uint64_t* unitig_offsets,
                                            uint64_t n_unitigs, uint32_t k, uint32_t key_bits, uint64_t* keys_out,
                                            uint32_t* unitig_out, uint8_t* is_rc_out, uint32_t* pos_out, uint64_t cap_out,
                                            uint64_t* n_out) {
    if (!ctx || !unitig_offsets || !n_out || (n_unitigs && !unitig_ascii)) return FBK_ERR_INVALID;
    const int nw = key_bits == 64 ? 1 : key_bits == 128 ? 2 : key_bits == 256 ? 4 : 0;
    if (!nw || k < 1 || k > (uint32_t)(32 * nw - 1)) return set_err(ctx, FBK_ERR_INVALID, "k out of range for key_bits");
    CK(ctx, cudaSetDevice(ctx->device));
    Bufs B{ctx, {}};
    uint64_t* d_words = nullptr;
    fbk_status st = pack_unitigs(ctx, B, unitig_ascii, unitig_offsets, n_unitigs, &d_words);
    if (st) return st;
    std::vector<TermWindow> win;
    for (uint64_t u = 0; u < n_unitigs; ++u) {
        const uint64_t base = unitig_offsets[u] - unitig_offsets[0], len = unitig_offsets[u + 1] - unitig_offsets[u];
        if (len < k) continue;
        const uint64_t total = len - k + 1;
        if (total <= 2000) {
            for (uint64_t i = 0; i < total; ++i) win.push_back({base + i, (uint32_t)u, (uint32_t)i});
        } else {
            for (uint64_t i = 0; i < 1000; ++i) win.push_back({base + i, (uint32_t)u, (uint32_t)i});
            for (uint64_t i = total - 1000; i < total; ++i) win.push_back({base + i, (uint32_t)u, (uint32_t)i});
        }
    }
    uint64_t cap = 1024;
    while (cap < 2 * win.size()) cap <<= 1;
    TermWindow* d_win = (TermWindow*)B.get(std::max<uint64_t>(win.size(), 1) * sizeof(TermWindow));
    unsigned long long* keys = (unsigned long long*)B.get(cap * 8);
    uint32_t* cnt = (uint32_t*)B.get(cap * 4);
    uint64_t* vals = (uint64_t*)B.get(cap * 8);
    unsigned long long* ff = (unsigned long long*)B.get(64);
    if (!d_win || !keys || !cnt || !vals || !ff) return set_err(ctx, FBK_ERR_OOM, "terminal k-mer index buffers");
    if (!win.empty()) CK(ctx, cudaMemcpyAsync(d_win, win.data(), win.size() * sizeof(TermWindow), cudaMemcpyHostToDevice, ctx->stream));
    CK(ctx, cudaMemsetAsync(keys, 0xFF, cap * 8, ctx->stream));
    CK(ctx, cudaMemsetAsync(cnt, 0, cap * 4, ctx->stream));
    CK(ctx, cudaMemsetAsync(ff, 0, 64, ctx->stream));
    Launch L = launch_cfg(ctx, 256, 0);
    if (!win.empty()) {
        cudaError_t e = cudaSuccess;
        TimedLaunch tl;
        time_begin(ctx, "term_index", tl);
        if (nw == 1) k_term_insert<1><<<L.grid, L.block, 0, L.stream>>>(d_words, d_win, win.size(), k, keys, cnt, vals, cap, ff);
        else if (nw == 2) k_term_insert<2><<<L.grid, L.block, 0, L.stream>>>(d_words, d_win, win.size(), k, keys, cnt, vals, cap, ff);
        else k_term_insert<4><<<L.grid, L.block, 0, L.stream>>>(d_words, d_win, win.size(), k, keys, cnt, vals, cap, ff);
        e = cudaGetLastError();
        time_end(ctx, tl);
        if (e != cudaSuccess) return cuda_err(ctx, e, "term_index");
    }
    std::vector<unsigned long long> hk(cap);
    std::vector<uint32_t> hc(cap);
    std::vector<uint64_t> hv(cap);
    unsigned long long hff[2] = {0, 0};
    CK(ctx, cudaMemcpyAsync(hk.data(), keys, cap * 8, cudaMemcpyDeviceToHost, ctx->stream));
    CK(ctx, cudaMemcpyAsync(hc.data(), cnt, cap * 4, cudaMemcpyDeviceToHost, ctx->stream));
    CK(ctx, cudaMemcpyAsync(hv.data(), vals, cap * 8, cudaMemcpyDeviceToHost, ctx->stream));
    CK(ctx, cudaMemcpyAsync(hff, ff, 16, cudaMemcpyDeviceToHost, ctx->stream));
    CK(ctx, cudaStreamSynchronize(ctx->stream));
    std::vector<std::pair<uint64_t, uint64_t>> uniq;
    for (uint64_t s = 0; s < cap; ++s)
        if (hk[s] != HSET_EMPTY && hc[s] == 1) uniq.push_back({hk[s], hv[s]});
    if (hff[0] == 1) uniq.push_back({HSET_EMPTY, hff[1]});
    std::sort(uniq.begin(), uniq.end());
    const uint64_t n = std::min<uint64_t>(cap_out, uniq.size());
    for (uint64_t i = 0; i < n; ++i) {
        if (keys_out) keys_out[i] = uniq[i].first;
        if (unitig_out) unitig_out[i] = (uint32_t)(uniq[i].second >> 33);
        if (is_rc_out) is_rc_out[i] = (uint8_t)((uniq[i].second >> 32) & 1);
        if (pos_out) pos_out[i] = (uint32_t)uniq[i].second;
    }
    *n_out = uniq.size();
    return FBK_OK;
}

}  // extern "C"
