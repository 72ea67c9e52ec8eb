// CUDA engine for sm_100a: device database, phase kernels, phase executor.
//
// Frontiers are row-major uint32 tables (one column per matched query
// vertex).  An extension or reduction by itself runs as
//   count  (thread per row)            -> per-256-row block totals
//   scan   (one CTA or one cluster)    -> exclusive block offsets + total
//   write  (CTA per block; with long lists per share of the outputs)
//                                      -> rows staged in shared memory,
//                                         outputs balanced across the CTA,
//                                         flushed with coalesced stores
// so the output size is known before it is written (no device-side overflow
// protocol, unlike src/miningPattern.cu:3325-3343).  A query's steps run
// either as a chain of one-pass kernels (graphs without long lists, run_chain)
// or counted, an extension and its reduction fused (ext_red_kernel).  Output
// order is deterministic on every path (input-row order, candidates ascending).
//
// Label segments come from an index (packed records or a dense (vertex, label)
// offset table), one load per lookup, replacing the warp bisection with vLabel
// gathers of the reference (FIND_LABEL_LIMIT, include/common.h:18-66).
#include <cooperative_groups.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <atomic>
#include <cstdio>
#include <cstring>
#include <string>

#include "../../include/geneva.h"
#include "gva_engine.cuh"
#include "gva_kernels.cuh"

namespace gva {

namespace {

#define GVA_CUDA(call)                                                                                  \
    do {                                                                                                \
        cudaError_t e_ = (call);                                                                        \
        if (e_ != cudaSuccess)                                                                          \
            return fail(GVA_ERR_CUDA, std::string(#call) + ": " + cudaGetErrorString(e_));              \
    } while (0)

inline size_t align256(size_t x) { return (x + 255) & ~(size_t)255; }

// ---------------------------------------------------------------- kernels ---
__global__ void __launch_bounds__(kThreads) ext_count_kernel(ExtArgs p, uint64_t* __restrict__ block_sums) {
    const uint64_t r = (uint64_t)blockIdx.x * kRowsPerBlock + threadIdx.x;
    uint64_t c = 0;
    if (r < p.nrows) c = ext_count_row(p, p.in + r * p.k);
    store_block_sum(c, block_sums);
}

__global__ void __launch_bounds__(kThreads) red_count_kernel(RedArgs p, uint64_t* __restrict__ block_sums) {
    const uint64_t r = (uint64_t)blockIdx.x * kRowsPerBlock + threadIdx.x;
    uint64_t c = 0;
    if (r < p.nrows) c = red_keep_row(p, p.in + r * p.k) ? 1 : 0;
    store_block_sum(c, block_sums);
}

// The outputs of an extension are shared out to CTAs by an ordinal that
// counts both the rows read and the rows written: block b (256 input rows)
// takes kBlockWork for its prologue (lookups and a scan) and then one for each
// of its output rows.  A CTA takes `chunk` consecutive ordinals, so that a
// block under a hub is written by as many CTAs as its rows need and a run of
// blocks without output costs one.  (With a CTA per block, 910 blocks wrote
// the 24 million rows of one step on an R-MAT graph of 2^18 vertices in 830
// us, most of them waiting for a few hub blocks.)
constexpr uint64_t kBlockWork = 1024;
constexpr uint64_t kEvenDegree = 256;  // up to this degree a CTA takes a block

__device__ __forceinline__ uint64_t block_key(const uint64_t* __restrict__ block_off, uint64_t b) {
    return __ldg(block_off + b) + b * kBlockWork;
}

// Last block b in [0, nb) with block_key(b) <= x, found by the first warp, 32
// pivots per step.
__device__ __forceinline__ uint64_t find_block(const uint64_t* __restrict__ block_off, uint64_t nb, uint64_t x) {
    __shared__ uint64_t found;
    if (threadIdx.x < 32) {
        uint64_t lo = 0, len = nb;
        while (len > 1) {
            const uint64_t step = (len + 31) / 32, at = threadIdx.x * step;
            const uint32_t m = __ballot_sync(0xffffffffu, at < len && block_key(block_off, lo + at) <= x);
            const uint64_t k = (31 - __clz(m)) * step;  // block 0's key is 0
            lo += k;
            len = len - k < step ? len - k : step;
        }
        if (threadIdx.x == 0) found = lo;
    }
    __syncthreads();
    const uint64_t b = found;
    __syncthreads();
    return b;
}

// The part [first, last) of block b's output rows that ordinals [k0, k1) hold.
__device__ __forceinline__ void block_part(const uint64_t* __restrict__ block_off, uint64_t b, uint64_t k0, uint64_t k1,
                                           uint64_t& first, uint64_t& last) {
    const uint64_t base = block_key(block_off, b) + kBlockWork, n = __ldg(block_off + b + 1) - __ldg(block_off + b);
    first = k0 > base ? k0 - base : 0;
    last = k1 > base ? umin64(k1 - base, n) : 0;
}

// One row of a block: its candidate list and the positions in it of matched
// vertices (ascending, each once); returns its output rows.
__device__ __forceinline__ uint32_t block_row(const ExtArgs& p, const uint32_t* row, uint32_t* coll, uint32_t& lo,
                                              uint32_t& nc) {
    uint32_t hi;
    ext_range(p, row, lo, hi);
    nc = 0;
    if (lo >= hi) return 0;
    for (uint32_t j = 0; j < p.n_eq; ++j) {
        const uint32_t pos = find_in(p.adj, lo, hi, row[p.eq_cols[j]]);
        if (pos == 0xffffffffu) continue;
        bool dup = false;
        for (uint32_t i = 0; i < nc; ++i) dup |= (coll[i] == pos);
        if (dup) continue;
        uint32_t i = nc++;  // insertion sort, ascending
        while (i > 0 && coll[i - 1] > pos) {
            coll[i] = coll[i - 1];
            --i;
        }
        coll[i] = pos;
    }
    return hi - lo - nc;
}

// List position of a row's u-th output row.
__device__ __forceinline__ uint32_t nth_candidate(uint32_t lo, const uint32_t* coll, uint32_t nc, uint32_t u) {
    uint32_t j = lo + u;
    for (uint32_t c = 0; c < nc; ++c) j += (coll[c] <= j) ? 1u : 0u;
    return j;
}

// Largest r in [0, nr) with offs[r] <= o.
__device__ __forceinline__ int row_of(const uint64_t* offs, int nr, uint64_t o) {
    int a = 0, b = nr - 1;
    while (a < b) {
        const int m = (a + b + 1) >> 1;
        if (offs[m] <= o)
            a = m;
        else
            b = m - 1;
    }
    return a;
}

// Every thread produces one output row per tile of 256, so a CTA's work is
// balanced however the candidates are spread over its rows.
__global__ void __launch_bounds__(kThreads) ext_write_kernel(ExtArgs p, const uint64_t* __restrict__ block_off,
                                                             uint64_t nb, uint64_t chunk) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    uint64_t* offs_s = reinterpret_cast<uint64_t*>(smem_raw);           // 257
    uint32_t* rows_s = reinterpret_cast<uint32_t*>(offs_s + kRowsPerBlock + 1);  // 256 * k
    uint32_t* lo_s = rows_s + kRowsPerBlock * p.k;                        // 256
    uint32_t* ncol_s = lo_s + kRowsPerBlock;                              // 256
    uint32_t* coll_s = ncol_s + kRowsPerBlock;                            // 256 * n_eq
    uint32_t* out_s = coll_s + kRowsPerBlock * p.n_eq;                    // 256 * (k + 1)
    const uint32_t k = p.k, k1 = p.k + 1;
    const uint64_t o0 = blockIdx.x * chunk, o1 = o0 + chunk;
    for (uint64_t b = chunk ? find_block(block_off, nb, o0) : blockIdx.x;; ++b) {
        uint64_t first = 0, last = 0;
        if (chunk) {
            if (b >= nb || block_key(block_off, b) >= o1) break;
            block_part(block_off, b, o0, o1, first, last);
            if (first >= last) continue;
        }
        const uint64_t row0 = b * kRowsPerBlock;
        const uint32_t nr = (uint32_t)umin64((uint64_t)kRowsPerBlock, p.nrows - row0);

        // coalesced load of this block's rows
        const uint32_t* gin = p.in + row0 * k;
        for (uint32_t w = threadIdx.x; w < nr * k; w += kThreads) rows_s[w] = gin[w];
        __syncthreads();
        uint64_t cnt = 0;
        if (threadIdx.x < nr)
            cnt = block_row(p, rows_s + threadIdx.x * k, coll_s + threadIdx.x * p.n_eq, lo_s[threadIdx.x],
                            ncol_s[threadIdx.x]);
        uint64_t total;
        offs_s[threadIdx.x] = block_exclusive_scan(cnt, &total);
        if (threadIdx.x == 0) offs_s[nr] = total;
        __syncthreads();
        if (!chunk) last = total;

        const uint64_t out0 = __ldg(block_off + b);
        for (uint64_t base = first; base < last; base += kThreads) {
            const uint64_t o = base + threadIdx.x;
            if (o < last) {
                const int a = row_of(offs_s, (int)nr, o);
                const uint32_t j = nth_candidate(lo_s[a], coll_s + a * p.n_eq, ncol_s[a], (uint32_t)(o - offs_s[a]));
                uint32_t* dst = out_s + threadIdx.x * k1;
                const uint32_t* src = rows_s + a * k;
                for (uint32_t c = 0; c < k; ++c) dst[c] = src[c];
                dst[k] = __ldg(p.adj + j);
            }
            __syncthreads();
            const uint32_t n_tile = (uint32_t)umin64((uint64_t)kThreads, last - base);
            uint32_t* gout = p.out + (out0 + base) * k1;
            for (uint32_t w = threadIdx.x; w < n_tile * k1; w += kThreads) gout[w] = out_s[w];
            __syncthreads();
        }
        if (!chunk) break;
    }
}

// First index >= at in [at, hi) with adj[index] >= x (hi if none), looked for
// from `at` outwards.
__device__ __forceinline__ uint32_t gallop(const uint32_t* __restrict__ adj, uint32_t at, uint32_t hi, uint32_t x) {
    uint32_t step = 1;
    while (hi - at > step && __ldg(adj + at + step) < x) {
        at += step;
        step <<= 1;
    }
    return lower_bound_u32(adj, at, hi - at > step ? at + step : hi, x);
}

// An extension and the reduction after it in one: the extension's output rows
// (counted, and placed in block_off, but never written) are tested as they
// are generated, and only those that pass are written.  A row's candidates
// come from the shorter of its list and the checked vertices' lists, cut to
// the vertices between its first and last candidate of this chunk: the rows
// kept, and their order, are those of the two steps.  A thread tests eight
// consecutive candidates, searching the other list from where it found the
// last one.  The count pass keeps its verdicts (a byte per eight candidates,
// `mask_cap` per CTA) for the write pass.
//
// What bounds it: the loads of those searches.  24 million extension rows,
// 1.2 million of them kept, on an R-MAT graph of 2^18 vertices: written,
// counted and written again in 830 + 474 + 608 us as two steps, counted and
// written in 425 + 71 us here (490 with 48 registers and five CTAs per SM
// instead of 32 and eight: more searches in flight).
constexpr uint32_t kTestRun = 8;
template <bool WRITE>
__global__ void __launch_bounds__(kThreads, 8) ext_red_kernel(ExtArgs p, const uint64_t* __restrict__ block_off,
                                                           uint64_t nb, uint64_t chunk, uint64_t* __restrict__ sums,
                                                           uint8_t* __restrict__ masks, uint32_t mask_cap) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    uint64_t* offs_s = reinterpret_cast<uint64_t*>(smem_raw);                  // 257
    const uint32_t** gadj_s = reinterpret_cast<const uint32_t**>(offs_s + kRowsPerBlock + 1);  // 256
    uint32_t* rows_s = reinterpret_cast<uint32_t*>(gadj_s + kRowsPerBlock);    // 256 * k
    uint32_t* glo_s = rows_s + kRowsPerBlock * p.k;                            // 256: the candidates' list
    uint32_t* ghi_s = glo_s + kRowsPerBlock;                                   // 256
    uint32_t* slo_s = ghi_s + kRowsPerBlock;                                   // 256: the list searched
    uint32_t* shi_s = slo_s + kRowsPerBlock;                                   // 256
    int* which_s = reinterpret_cast<int*>(shi_s + kRowsPerBlock);              // 256: check of the candidates' list
    int* other_s = which_s + kRowsPerBlock;                                    // 256: check of the list searched
    uint32_t* coll_s = reinterpret_cast<uint32_t*>(other_s + kRowsPerBlock);   // 256 * n_eq
    constexpr int kSource = -1, kNone_ = -2;
    const uint32_t k = p.k, k1 = p.k + 1;
    const uint64_t o0 = blockIdx.x * chunk, o1 = o0 + chunk;
    uint8_t* mask = masks + (uint64_t)blockIdx.x * mask_cap;
    uint64_t done = 0;  // rows kept so far: by this thread (count), by the CTA (write)
    for (uint64_t b = find_block(block_off, nb, o0); b < nb && block_key(block_off, b) < o1; ++b) {
        uint64_t first, last;
        block_part(block_off, b, o0, o1, first, last);
        if (first >= last) continue;
        const uint64_t row0 = b * kRowsPerBlock;
        const uint32_t nr = (uint32_t)umin64((uint64_t)kRowsPerBlock, p.nrows - row0);
        const uint32_t* gin = p.in + row0 * k;
        for (uint32_t w = threadIdx.x; w < nr * k; w += kThreads) rows_s[w] = gin[w];
        __syncthreads();
        const uint32_t* row = rows_s + threadIdx.x * k;
        uint32_t* coll = coll_s + threadIdx.x * p.n_eq;
        uint32_t lo = 0, nc = 0;
        uint64_t cnt = 0, total;
        if (threadIdx.x < nr) cnt = block_row(p, row, coll, lo, nc);
        const uint64_t before = block_exclusive_scan(cnt, &total);
        // this row's part of the chunk, as list positions [slo, shi); its
        // candidates are those of the shortest list
        uint32_t slo = 0, shi = 0, glo = 0, ghi = 0;
        int which = kSource, other = kNone_;
        const uint32_t* gadj = p.adj;
        if (cnt && before < last && before + cnt > first) {
            const uint32_t u0 = first > before ? (uint32_t)(first - before) : 0;
            const uint32_t u1 = (uint32_t)umin64(cnt, last - before);
            glo = nth_candidate(lo, coll, nc, u0);
            ghi = nth_candidate(lo, coll, nc, u1 - 1) + 1;
            const uint32_t v0 = __ldg(p.adj + glo);
            const uint64_t v1 = (uint64_t)__ldg(p.adj + ghi - 1) + 1;
            for (uint32_t i = 0; i < p.n_chk; ++i) {
                if (p.chk_dir[i]) continue;
                uint32_t cl, ch;
                seg_of(p.chk_off[i], p.L, row[p.chk_col[i]], p.chk_lab[i], cl, ch);
                cl = lower_bound_u32(p.chk_adj[i], cl, ch, v0);
                ch = lower_bound_u32(p.chk_adj[i], cl, ch, v1);
                if (ch - cl < ghi - glo) {  // the new shortest; the old one is searched
                    slo = glo;
                    shi = ghi;
                    other = which;
                    glo = cl;
                    ghi = ch;
                    gadj = p.chk_adj[i];
                    which = (int)i;
                } else if (other == kNone_) {
                    slo = cl;
                    shi = ch;
                    other = (int)i;
                }
            }
        }
        slo_s[threadIdx.x] = slo;
        shi_s[threadIdx.x] = shi;
        glo_s[threadIdx.x] = glo;
        ghi_s[threadIdx.x] = ghi;
        gadj_s[threadIdx.x] = gadj;
        which_s[threadIdx.x] = which;
        other_s[threadIdx.x] = other;
        offs_s[threadIdx.x] = block_exclusive_scan((ghi - glo + kTestRun - 1) / kTestRun, &total);
        __syncthreads();
        for (uint64_t base = 0; base < total; base += kThreads) {
            const uint64_t o = base + threadIdx.x;
            uint32_t m = 0, x = 0;
            int a = 0;
            if (o < total) {
                a = row_of(offs_s, kRowsPerBlock, o);
                x = glo_s[a] + (uint32_t)(o - offs_s[a]) * kTestRun;
                if (WRITE) m = mask[o];
            }
            if (!WRITE && o < total) {
                const uint32_t* r = rows_s + a * k;
                const uint32_t* g = gadj_s[a];
                const int wh = which_s[a], ot = other_s[a];
                const uint32_t* oadj = ot >= 0 ? p.chk_adj[ot] : p.adj;
                const uint32_t n = min(kTestRun, ghi_s[a] - x), oh = shi_s[a];
                uint32_t at = slo_s[a];
                for (uint32_t i = 0; i < n; ++i) {
                    const uint32_t c = __ldg(g + x + i);
                    bool ok = true;
                    for (uint32_t j = 0; j < p.n_eq && ok; ++j) ok = r[p.eq_cols[j]] != c;
                    if (ok && ot != kNone_) {
                        at = i ? gallop(oadj, at, oh, c) : lower_bound_u32(oadj, at, oh, c);
                        ok = at < oh && __ldg(oadj + at) == c;
                    }
                    for (int j = 0; j < (int)p.n_chk && ok; ++j) {
                        if (j == wh || j == ot) continue;
                        ok = p.chk_dir[j] ? seg_has(p.chk_off[j], p.chk_adj[j], p.L, c, p.chk_lab[j], r[p.chk_col[j]])
                                          : seg_has(p.chk_off[j], p.chk_adj[j], p.L, r[p.chk_col[j]], p.chk_lab[j], c);
                    }
                    // with three lists or more the source's may be neither
                    if (ok && wh != kSource && ot != kSource) {
                        uint32_t sl, sh;
                        ext_range(p, r, sl, sh);
                        ok = find_in(p.adj, sl, sh, c) != 0xffffffffu;
                    }
                    if (ok) m |= 1u << i;
                }
                mask[o] = (uint8_t)m;
                done += __popc(m);
            }
            if (WRITE) {
                uint64_t kept;
                const uint64_t at = block_exclusive_scan(__popc(m), &kept);
                uint32_t* dst = p.out + (sums[blockIdx.x] + done + at) * k1;
                const uint32_t* r = rows_s + a * k;
                while (m) {
                    const uint32_t i = __ffs(m) - 1;
                    m &= m - 1;
                    for (uint32_t j = 0; j < k; ++j) dst[j] = r[j];
                    dst[k] = __ldg(gadj_s[a] + x + i);
                    dst += k1;
                }
                done += kept;
            }
        }
        mask += total;
        __syncthreads();  // every thread done with this block's rows
    }
    if (!WRITE) store_block_sum(done, sums);
}

__global__ void __launch_bounds__(kThreads) red_write_kernel(RedArgs p, const uint64_t* __restrict__ block_off) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    uint32_t* rows_s = reinterpret_cast<uint32_t*>(smem_raw);  // 256 * k (compacted in a second buffer)
    uint32_t* out_s = rows_s + kRowsPerBlock * p.k;
    const uint64_t row0 = (uint64_t)blockIdx.x * kRowsPerBlock;
    const uint32_t nr = (uint32_t)umin64((uint64_t)kRowsPerBlock, p.nrows - row0);
    const uint32_t k = p.k;
    const uint32_t* gin = p.in + row0 * k;
    for (uint32_t w = threadIdx.x; w < nr * k; w += kThreads) rows_s[w] = gin[w];
    __syncthreads();
    bool keep = false;
    if (threadIdx.x < nr) keep = red_keep_row(p, rows_s + threadIdx.x * k);
    uint64_t total;
    const uint64_t before = block_exclusive_scan(keep ? 1 : 0, &total);
    if (keep)
        for (uint32_t c = 0; c < k; ++c) out_s[before * k + c] = rows_s[threadIdx.x * k + c];
    __syncthreads();
    uint32_t* gout = p.out + block_off[blockIdx.x] * k;
    for (uint32_t w = threadIdx.x; w < (uint32_t)total * k; w += kThreads) gout[w] = out_s[w];
}

// ------------------------------------------------------- steps in a chain ---
// On a graph without long lists a query's steps are launched one after another
// without a look at their totals: a step counts, places and writes its rows in
// one pass (tiles of 256 input rows, taken in order from a counter; a tile's
// place is the sum of the tiles before it, looked back for while they run),
// takes its input's length from the step before it, and the host reads all
// totals at the end.  Rows and order are those of the counted steps.
//
// What bounds it: latency.  A query of three steps on a 1,000-graph database
// has 30 us of kernels; the host's look at every total (copy, wait, allocate,
// launch) made it 112 us, the chain takes 48.  (Looking back by the whole CTA,
// 256 tiles at a time, was slower: 18 against 16 us for 1,144 tiles.)
struct Chain {
    const uint64_t* n_in;            // rows of the input (null: p.nrows)
    uint64_t cap_in, cap_out;        // rows that the input / output has room for
    unsigned long long* tiles;       // next tile
    unsigned long long* status;      // per tile: 1 << 62 | rows, then 2 << 62 | rows up to here
    uint64_t* n_out;                 // rows of the output
    uint64_t* host_out;              // the same, in host memory
    uint32_t* failed;                // 1: an output has no room, 2: a wait ran out
    uint32_t* host_failed;
    uint32_t polls;                  // of a tile for the ones before it, then the chain fails
};

__device__ __forceinline__ void chain_fail(const Chain& c, uint32_t why) {
    *(volatile uint32_t*)c.failed = why;
    *(volatile uint32_t*)c.host_failed = why;
    __threadfence_system();
}

// Rows of a step's input: none once a step has failed (its rows were not all
// written).  A CTA that starts late may find its own step's failure; the CTAs
// that found none take all of its tiles, so that the total is known.
// A step's launch may start while the one before it runs and waits for it
// here (its rows and totals are read with plain loads).
__device__ __forceinline__ uint64_t chain_rows(const Chain& c, uint64_t nrows) {
    __shared__ uint64_t n;
    asm volatile("griddepcontrol.wait;" ::: "memory");
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    if (threadIdx.x == 0)
        n = *(volatile uint32_t*)c.failed ? 0 : c.n_in ? umin64(*c.n_in, c.cap_in) : nrows;
    __syncthreads();
    return n;
}

// Whether the CTAs with lower numbers are as many as the tiles: this one need
// take none.
__device__ __forceinline__ bool chain_idle(uint64_t n) { return (uint64_t)blockIdx.x * kRowsPerBlock >= n; }

// The next tile, for every thread of the CTA.
__device__ __forceinline__ uint64_t chain_tile(const Chain& c) {
    __shared__ uint64_t tile;
    __syncthreads();  // the last one was read by every thread
    if (threadIdx.x == 0) tile = atomicAdd(c.tiles, 1ull);
    __syncthreads();
    return tile;
}

// Rows before `tile`, whose own number is `total`; ~0: the wait ran out.
// Tiles are taken in order, so the ones waited for are done or running.
__device__ __forceinline__ uint64_t chain_place(const Chain& c, uint64_t tile, uint64_t total) {
    __shared__ uint64_t place;
    constexpr unsigned long long kHas = 1ull << 62, kDone = 2ull << 62, kMask = kHas - 1;
    if (threadIdx.x < 32) {
        const int lane = threadIdx.x;
        volatile unsigned long long* status = c.status;
        uint64_t sum = 0;
        bool ok = true;
        if (tile > 0) {
            if (lane == 0) status[tile] = kHas | total;
            uint32_t polls = 0;
            for (int64_t at = (int64_t)tile - 1; ok;) {
                const int64_t i = at - lane;
                const unsigned long long w = i >= 0 ? status[i] : kDone;
                const uint32_t done = __ballot_sync(0xffffffffu, (w >> 62) == 2);
                const uint32_t none = __ballot_sync(0xffffffffu, (w >> 62) == 0);
                // lanes up to the nearest finished prefix
                const uint32_t upto = done ? (done & -done) | ((done & -done) - 1) : 0xffffffffu;
                if (none & upto) {
                    ok = ++polls < c.polls;
                    continue;
                }
                sum += __shfl_sync(0xffffffffu, warp_sum((upto >> lane & 1) ? (uint64_t)(w & kMask) : 0), 0);
                if (done) break;
                at -= 32;
            }
        }
        if (lane == 0) {
            if (ok)
                status[tile] = kDone | (sum + total);
            else
                chain_fail(c, 2);
            place = ok ? sum : ~0ull;
        }
    }
    __syncthreads();
    return place;
}

// The tile's rows are placed: the last one tells the total.  Returns whether
// they may be written.
__device__ __forceinline__ bool chain_end(const Chain& c, uint64_t tile, uint64_t n, uint64_t place, uint64_t total) {
    const bool room = place + total <= c.cap_out;
    if (threadIdx.x == 0) {
        if (!room) chain_fail(c, 1);
        if ((tile + 1) * kRowsPerBlock >= n) {
            *c.n_out = place + total;
            *(volatile uint64_t*)c.host_out = place + total;
        }
    }
    return room;
}

__global__ void __launch_bounds__(kThreads) chain_ext_kernel(ExtArgs p, Chain c) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    uint64_t* offs_s = reinterpret_cast<uint64_t*>(smem_raw);           // 257
    uint32_t* rows_s = reinterpret_cast<uint32_t*>(offs_s + kRowsPerBlock + 1);  // 256 * k
    uint32_t* lo_s = rows_s + kRowsPerBlock * p.k;                        // 256
    uint32_t* ncol_s = lo_s + kRowsPerBlock;                              // 256
    uint32_t* coll_s = ncol_s + kRowsPerBlock;                            // 256 * n_eq
    uint32_t* out_s = coll_s + kRowsPerBlock * p.n_eq;                    // 256 * (k + 1)
    const uint32_t k = p.k, k1 = p.k + 1;
    const uint64_t n = chain_rows(c, p.nrows);
    if (chain_idle(n)) return;
    for (;;) {
        const uint64_t tile = chain_tile(c), row0 = tile * kRowsPerBlock;
        if (row0 >= n) return;
        const uint32_t nr = (uint32_t)umin64((uint64_t)kRowsPerBlock, n - row0);
        const uint32_t* gin = p.in + row0 * k;
        for (uint32_t w = threadIdx.x; w < nr * k; w += kThreads) rows_s[w] = gin[w];
        __syncthreads();
        uint64_t cnt = 0, total;
        if (threadIdx.x < nr)
            cnt = block_row(p, rows_s + threadIdx.x * k, coll_s + threadIdx.x * p.n_eq, lo_s[threadIdx.x],
                            ncol_s[threadIdx.x]);
        offs_s[threadIdx.x] = block_exclusive_scan(cnt, &total);
        const uint64_t place = chain_place(c, tile, total);
        if (place == ~0ull) return;
        if (!chain_end(c, tile, n, place, total)) continue;  // counted only
        for (uint64_t base = 0; base < total; base += kThreads) {
            const uint64_t o = base + threadIdx.x;
            if (o < total) {
                const int a = row_of(offs_s, (int)nr, o);
                const uint32_t j = nth_candidate(lo_s[a], coll_s + a * p.n_eq, ncol_s[a], (uint32_t)(o - offs_s[a]));
                uint32_t* dst = out_s + threadIdx.x * k1;
                const uint32_t* src = rows_s + a * k;
                for (uint32_t i = 0; i < k; ++i) dst[i] = src[i];
                dst[k] = __ldg(p.adj + j);
            }
            __syncthreads();
            const uint32_t n_tile = (uint32_t)umin64((uint64_t)kThreads, total - base);
            uint32_t* gout = p.out + (place + base) * k1;
            for (uint32_t w = threadIdx.x; w < n_tile * k1; w += kThreads) gout[w] = out_s[w];
            __syncthreads();
        }
    }
}

__global__ void __launch_bounds__(kThreads) chain_red_kernel(RedArgs p, Chain c) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    uint32_t* rows_s = reinterpret_cast<uint32_t*>(smem_raw);
    uint32_t* out_s = rows_s + kRowsPerBlock * p.k;
    const uint32_t k = p.k;
    const uint64_t n = chain_rows(c, p.nrows);
    if (chain_idle(n)) return;
    for (;;) {
        const uint64_t tile = chain_tile(c), row0 = tile * kRowsPerBlock;
        if (row0 >= n) return;
        const uint32_t nr = (uint32_t)umin64((uint64_t)kRowsPerBlock, n - row0);
        const uint32_t* gin = p.in + row0 * k;
        for (uint32_t w = threadIdx.x; w < nr * k; w += kThreads) rows_s[w] = gin[w];
        __syncthreads();
        const bool keep = threadIdx.x < nr && red_keep_row(p, rows_s + threadIdx.x * k);
        uint64_t total;
        const uint64_t before = block_exclusive_scan(keep ? 1 : 0, &total);
        const uint64_t place = chain_place(c, tile, total);
        if (place == ~0ull) return;
        if (!chain_end(c, tile, n, place, total)) continue;  // counted only
        if (keep)
            for (uint32_t i = 0; i < k; ++i) out_s[before * k + i] = rows_s[threadIdx.x * k + i];
        __syncthreads();
        uint32_t* gout = p.out + place * k;
        for (uint32_t w = threadIdx.x; w < (uint32_t)total * k; w += kThreads) gout[w] = out_s[w];
    }
}

// The last step of a counted query: only its total.  c.status[0] counts the
// CTAs that have added theirs.
template <class Args>
__global__ void __launch_bounds__(kThreads) chain_count_kernel(Args p, Chain c) {
    const uint64_t n = chain_rows(c, p.nrows);
    uint64_t v = 0;
    for (uint64_t r = (uint64_t)blockIdx.x * kThreads + threadIdx.x; r < n; r += (uint64_t)gridDim.x * kThreads) {
        if constexpr (sizeof(Args) == sizeof(ExtArgs))
            v += ext_count_plain(p, p.in + r * p.k);
        else
            v += red_keep_row(p, p.in + r * p.k) ? 1 : 0;
    }
    __shared__ uint64_t ws[kThreads / 32];
    v = warp_sum(v);
    if ((threadIdx.x & 31) == 0) ws[threadIdx.x >> 5] = v;
    __syncthreads();
    if (threadIdx.x == 0) {
        for (int i = 1; i < kThreads / 32; ++i) v += ws[i];
        if (v) atomicAdd((unsigned long long*)c.n_out, (unsigned long long)v);
        __threadfence();
        if (atomicAdd(c.status, 1ull) + 1 == gridDim.x)
            *(volatile uint64_t*)c.host_out = atomicAdd((unsigned long long*)c.n_out, 0ull);
    }
}
static_assert(sizeof(ExtArgs) != sizeof(RedArgs), "told apart by their sizes");

// The same scan as scan_block_sums_kernel by one cluster: every thread takes a
// contiguous share, the CTAs exchange their sums through distributed shared
// memory.  94,578 sums: 93 us with one CTA.
constexpr int kScanCtas = 8;
__global__ void __cluster_dims__(kScanCtas, 1, 1) __launch_bounds__(kScanThreads)
scan_cluster_kernel(uint64_t* __restrict__ sums, uint64_t n) {
    namespace cg = cooperative_groups;
    cg::cluster_group cl = cg::this_cluster();
    __shared__ uint64_t ws[32];
    __shared__ uint64_t mine;
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    const uint64_t all = (uint64_t)kScanCtas * kScanThreads, per = (n + all - 1) / all;
    const uint64_t me = (uint64_t)blockIdx.x * kScanThreads + threadIdx.x;
    const uint64_t b = umin64(n, me * per), e = umin64(n, b + per);
    uint64_t v = 0;
    for (uint64_t i = b; i < e; ++i) v += sums[i];
    uint64_t inc = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint64_t y = __shfl_up_sync(0xffffffffu, inc, o);
        if (lane >= o) inc += y;
    }
    if (lane == 31) ws[wid] = inc;
    __syncthreads();
    if (wid == 0) {
        uint64_t w = ws[lane];
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint64_t y = __shfl_up_sync(0xffffffffu, w, o);
            if (lane >= o) w += y;
        }
        ws[lane] = w;
        if (lane == 31) mine = w;
    }
    cl.sync();
    uint64_t at = (wid > 0 ? ws[wid - 1] : 0) + inc - v, total = 0;
    for (uint32_t r = 0; r < kScanCtas; ++r) {
        const uint64_t x = *cl.map_shared_rank(&mine, r);
        if (r < cl.block_rank()) at += x;
        total += x;
    }
    for (uint64_t i = b; i < e; ++i) {
        const uint64_t x = sums[i];
        sums[i] = at;
        at += x;
    }
    if (me == 0) sums[n] = total;
    cl.sync();  // no CTA leaves while another reads its sum
}

size_t ext_smem_bytes(uint32_t k, uint32_t n_eq) {
    return sizeof(uint64_t) * (kRowsPerBlock + 1) +
           sizeof(uint32_t) * ((size_t)kRowsPerBlock * k + 2 * kRowsPerBlock + (size_t)kRowsPerBlock * n_eq +
                               (size_t)kRowsPerBlock * (k + 1));
}
size_t ext_red_smem_bytes(uint32_t k, uint32_t n_eq) {
    return sizeof(uint64_t) * (2 * kRowsPerBlock + 1) +
           sizeof(uint32_t) * ((size_t)kRowsPerBlock * k + 6 * kRowsPerBlock + (size_t)kRowsPerBlock * n_eq);
}
size_t red_smem_bytes(uint32_t k) { return sizeof(uint32_t) * 2 * (size_t)kRowsPerBlock * k; }

std::atomic<uint64_t> g_launches{0};

int set_smem_limits() {
    static std::atomic<bool> done[64];  // callers may run on several threads
    int dev = 0;
    GVA_CUDA(cudaGetDevice(&dev));
    if (dev < 64 && done[dev].load(std::memory_order_acquire)) return GVA_OK;
    GVA_CUDA(cudaFuncSetAttribute(ext_write_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                  (int)ext_smem_bytes(kMaxCols - 1, kMaxCols)));
    GVA_CUDA(cudaFuncSetAttribute(chain_ext_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                  (int)ext_smem_bytes(kMaxCols - 1, kMaxCols)));
    GVA_CUDA(cudaFuncSetAttribute(chain_red_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                  (int)red_smem_bytes(kMaxCols)));
    for (const void* fn : {(const void*)ext_red_kernel<false>, (const void*)ext_red_kernel<true>})
        GVA_CUDA(cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                      (int)ext_red_smem_bytes(kMaxCols - 1, kMaxCols)));
    GVA_CUDA(cudaFuncSetAttribute(red_write_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                  (int)red_smem_bytes(kMaxCols)));
    if (dev < 64) done[dev].store(true, std::memory_order_release);
    return GVA_OK;
}

void fill_ext(ExtArgs& a, const DevDB& db, const Step& st, const uint32_t* in, uint64_t nrows, uint32_t* out) {
    memset(&a, 0, sizeof a);
    const DevPart& P = db.parts[st.part - 1];
    a.in = in;
    a.nrows = nrows;
    a.out = out;
    a.off = P.off;
    a.adj = P.adj;
    a.k = st.width_in;
    a.L = db.kernel_L();
    a.lab = st.label;
    a.src_col = st.src_col;
    a.bound_col = st.bound_col;
    a.bound_incl = st.bound_inclusive;
    a.n_eq = st.n_eq;
    for (uint32_t i = 0; i < st.n_eq; ++i) a.eq_cols[i] = st.eq_cols[i];
}

void fill_red(RedArgs& a, const DevDB& db, const Step& st, const uint32_t* in, uint64_t nrows, uint32_t* out) {
    memset(&a, 0, sizeof a);
    const DevPart& P = db.parts[st.part - 1];
    a.in = in;
    a.nrows = nrows;
    a.out = out;
    a.off = P.off;
    a.adj = P.adj;
    a.k = st.width_in;
    a.L = db.kernel_L();
    a.n_pairs = st.n_pairs;
    for (uint32_t i = 0; i < st.n_pairs; ++i) {
        a.rs[i] = st.rs_col[i];
        a.re[i] = st.re_col[i];
        a.rl[i] = st.re_label[i];
    }
}

// Ordinals of one CTA of an extension's write (block_key): about 24 CTAs per
// SM, at least a block's worth and at most 32,768.  On a graph without long
// lists the blocks' outputs are alike and a CTA takes its block without a
// search (chunk 0; 6.0 against 8.6 us for 1,144 blocks).
uint64_t chunk_of(const DevDB& db, uint64_t total, uint64_t nb) {
    const uint64_t all = total + nb * kBlockWork;
    const uint64_t ctas = (uint64_t)db.sms * 24;
    return std::min<uint64_t>(std::max<uint64_t>((all + ctas - 1) / ctas, kBlockWork + 256), 32768);
}
uint64_t num_chunks(const DevDB& db, uint64_t total, uint64_t nb) {
    const uint64_t c = chunk_of(db, total, nb);
    return (total + nb * kBlockWork + c - 1) / c;
}

// Verdict bytes of one CTA of ext_red_kernel: one per eight candidates, and
// per row of the blocks that a chunk meets a started one and its matched
// vertices' (n_eq candidates more than output rows).
uint32_t mask_cap(uint64_t chunk, uint32_t n_eq) {
    return (uint32_t)(chunk / kTestRun + (kRowsPerBlock + kRowsPerBlock / kTestRun * n_eq) * (chunk / kBlockWork + 2));
}

// Exclusive scan of n block sums in place, their total in sums[n].
void launch_scan(uint64_t* sums, uint64_t n, cudaStream_t s) {
    if (n <= 4096)
        scan_block_sums_kernel<<<1, kScanThreads, 0, s>>>(sums, n);
    else
        scan_cluster_kernel<<<kScanCtas, kScanThreads, 0, s>>>(sums, n);
}

// Whether reduction `r` only checks edges of the vertex that extension `e`
// adds, so that ext_red_kernel can run both.
bool can_fuse(const DevDB& db, const Step& e, const Step& r) {
    if (db.max_degree <= kEvenDegree) return false;  // frontiers are small: the two steps are as fast
    if (e.kind != STEP_EXT || r.kind != STEP_REDUCE || e.always_empty || r.always_empty) return false;
    if (r.n_pairs == 0 || r.n_pairs > (uint32_t)kMaxChecks || r.width_in != e.width_in + 1) return false;
    for (const Step* st : {&e, &r})
        if (st->part == 0 || st->part > db.parts.size() || !db.parts[st->part - 1].off) return false;
    for (uint32_t i = 0; i < r.n_pairs; ++i)
        if ((r.rs_col[i] == e.width_in) == (r.re_col[i] == e.width_in)) return false;
    return true;
}

// count + scan; leaves exclusive block offsets in sums[0..nb) and the total in sums[nb]
int launch_count(const DevDB& db, const Step& st, const uint32_t* in, uint64_t nrows, uint64_t* sums,
                 cudaStream_t s, Profiler* prof) {
    const uint64_t nb = (nrows + kRowsPerBlock - 1) / kRowsPerBlock;
    if (nb > 0x7fffffffull) return fail(GVA_ERR_UNSUPPORTED, "frontier too large for one launch");
    const double k = st.width_in;
    cudaEvent_t ev = nullptr;
    if (st.kind == STEP_EXT) {
        ExtArgs a;
        fill_ext(a, db, st, in, nrows, nullptr);
        const double bytes = (4.0 * k + 8.0) * (double)nrows;
        if (prof) prof->begin(K_EXT_COUNT, bytes, s, ev);
        ext_count_kernel<<<(unsigned)nb, kThreads, 0, s>>>(a, sums);
        if (prof) prof->end(ev, K_EXT_COUNT, bytes, s, (double)nrows);
    } else {
        RedArgs a;
        fill_red(a, db, st, in, nrows, nullptr);
        const double bytes = (4.0 * k + 8.0 * st.n_pairs) * (double)nrows;
        if (prof) prof->begin(K_RED_COUNT, bytes, s, ev);
        red_count_kernel<<<(unsigned)nb, kThreads, 0, s>>>(a, sums);
        if (prof) prof->end(ev, K_RED_COUNT, bytes, s, (double)nrows);
    }
    GVA_CUDA(cudaGetLastError());
    const double sbytes = 16.0 * (double)nb;
    if (prof) prof->begin(K_SCAN, sbytes, s, ev);
    launch_scan(sums, nb, s);
    if (prof) prof->end(ev, K_SCAN, sbytes, s, (double)nb);
    GVA_CUDA(cudaGetLastError());
    g_launches += 2;
    return GVA_OK;
}

int launch_write(const DevDB& db, const Step& st, const uint32_t* in, uint64_t nrows, uint32_t* out,
                 const uint64_t* sums, uint64_t nout, cudaStream_t s, Profiler* prof) {
    const uint64_t nb = (nrows + kRowsPerBlock - 1) / kRowsPerBlock;
    int rc = set_smem_limits();
    if (rc) return rc;
    const double k = st.width_in;
    cudaEvent_t ev = nullptr;
    if (st.kind == STEP_EXT) {
        ExtArgs a;
        fill_ext(a, db, st, in, nrows, out);
        const double bytes = (4.0 * k + 8.0) * (double)nrows + (4.0 + 4.0 * (k + 1)) * (double)nout;
        if (prof) prof->begin(K_EXT_WRITE, bytes, s, ev);
        const bool even = db.max_degree <= kEvenDegree;
        const uint64_t nch = even ? nb : num_chunks(db, nout, nb);
        if (nch > 0x7fffffffull) return fail(GVA_ERR_UNSUPPORTED, "frontier too large for one launch");
        ext_write_kernel<<<(unsigned)nch, kThreads, ext_smem_bytes(a.k, a.n_eq), s>>>(a, sums, nb,
                                                                                      even ? 0 : chunk_of(db, nout, nb));
        if (prof) prof->end(ev, K_EXT_WRITE, bytes, s, (double)nrows);
    } else {
        RedArgs a;
        fill_red(a, db, st, in, nrows, out);
        const double bytes = (4.0 * k + 8.0 * st.n_pairs) * (double)nrows + 4.0 * k * (double)nout;
        if (prof) prof->begin(K_RED_WRITE, bytes, s, ev);
        red_write_kernel<<<(unsigned)nb, kThreads, red_smem_bytes(a.k), s>>>(a, sums);
        if (prof) prof->end(ev, K_RED_WRITE, bytes, s, (double)nrows);
    }
    GVA_CUDA(cudaGetLastError());
    g_launches += 1;
    return GVA_OK;
}

// The counted rows of extension `st` (offsets in sums, `total` rows) that pass
// reduction `rd`: counted per CTA into csums and scanned (out null), or
// written to out at the scanned offsets.
int launch_ext_red(const DevDB& db, const Step& st, const Step& rd, const uint32_t* in, uint64_t nrows, uint64_t total,
                   const uint64_t* sums, uint64_t* csums, uint8_t* masks, uint32_t* out, uint64_t kept, cudaStream_t s,
                   Profiler* prof) {
    int rc = set_smem_limits();
    if (rc) return rc;
    const uint64_t nb = (nrows + kRowsPerBlock - 1) / kRowsPerBlock, nch = num_chunks(db, total, nb);
    if (nch > 0x7fffffffull) return fail(GVA_ERR_UNSUPPORTED, "frontier too large for one launch");
    ExtArgs a;
    fill_ext(a, db, st, in, nrows, out);
    const DevPart& P = db.parts[rd.part - 1];
    a.n_chk = rd.n_pairs;
    for (uint32_t i = 0; i < rd.n_pairs; ++i) {
        // the new vertex on the right: it must lie in the partner's segment;
        // on the left: the partner in the new vertex's
        a.chk_dir[i] = rd.rs_col[i] == st.width_in ? 1 : 0;
        a.chk_col[i] = a.chk_dir[i] ? rd.re_col[i] : rd.rs_col[i];
        a.chk_lab[i] = rd.re_label[i];
        a.chk_off[i] = P.off;
        a.chk_adj[i] = P.adj;
    }
    const double k = st.width_in;
    cudaEvent_t ev = nullptr;
    const size_t smem = ext_red_smem_bytes(a.k, a.n_eq);
    if (!out) {
        const double bytes = (4.0 * k + 8.0) * (double)nrows + (4.0 + 8.0 * rd.n_pairs) * (double)total;
        if (prof) prof->begin(K_RED_COUNT, bytes, s, ev);
        ext_red_kernel<false><<<(unsigned)nch, kThreads, smem, s>>>(a, sums, nb, chunk_of(db, total, nb), csums, masks,
                                                                        mask_cap(chunk_of(db, total, nb), a.n_eq));
        if (prof) prof->end(ev, K_RED_COUNT, bytes, s, (double)total);
        GVA_CUDA(cudaGetLastError());
        if (prof) prof->begin(K_SCAN, 16.0 * (double)nch, s, ev);
        launch_scan(csums, nch, s);
        if (prof) prof->end(ev, K_SCAN, 16.0 * (double)nch, s, (double)nch);
        g_launches += 2;
    } else {
        const double bytes = (4.0 * k + 8.0) * (double)nrows + (4.0 + 8.0 * rd.n_pairs) * (double)total +
                             4.0 * (k + 1) * (double)kept;
        if (prof) prof->begin(K_RED_WRITE, bytes, s, ev);
        ext_red_kernel<true><<<(unsigned)nch, kThreads, smem, s>>>(a, sums, nb, chunk_of(db, total, nb), csums, masks,
                                                                        mask_cap(chunk_of(db, total, nb), a.n_eq));
        if (prof) prof->end(ev, K_RED_WRITE, bytes, s, (double)total);
        g_launches += 1;
    }
    GVA_CUDA(cudaGetLastError());
    return GVA_OK;
}

// Per-thread, per-device host staging reused by every query: a pinned word
// for count read-backs and two timing events (creating these per call costs
// more than a small query's kernels).
struct HostStage {
    uint64_t* pinned = nullptr;
    cudaEvent_t ev0 = nullptr, ev1 = nullptr;
};

int host_stage(int device, HostStage*& out) {
    static thread_local HostStage stages[64];
    if (device < 0 || device >= 64) return fail(GVA_ERR_ARG, "device index out of range");
    HostStage& h = stages[device];
    if (!h.pinned) {
        GVA_CUDA(cudaMallocHost(&h.pinned, 1024));
        GVA_CUDA(cudaEventCreate(&h.ev0));
        GVA_CUDA(cudaEventCreate(&h.ev1));
    }
    out = &h;
    return GVA_OK;
}

// Rows of the first step's input up to which a query runs as a chain, and the
// room of its result (a larger one is written by a second launch of the last
// step).
constexpr uint64_t kChainRows = 1ull << 22;
constexpr size_t kChainResult = 256u << 10;
constexpr size_t kChainSteps = 64;

// What a query's step leads one to expect of its rows, of the steps before it:
// the degrees as the database has them, labels and edges as if independent.
// Column labels are kept in `lab`.
double expected_rows(const DevDB& db, const Step& st, size_t i, double rows, std::vector<uint32_t>& lab) {
    if (st.kind == STEP_REDUCE) return rows / 4;
    const double* ends = db.ends.data() + (size_t)(st.part - 1) * db.L;
    const uint32_t from = lab[st.src_col];
    const double of_label = db.seed_off[from + 1] - db.seed_off[from];
    double all = 0;
    for (uint32_t l = 0; l < db.L; ++l) all += ends[l];
    lab.push_back(st.label);
    if (all == 0 || of_label == 0) return 0;
    rows *= ends[from] / of_label * (ends[st.label] / all);
    if (i > 1) rows *= db.bias[st.part - 1];  // only the first step's sources are any vertices
    return st.bound_col >= 0 ? rows / 2 : rows;
}

// Runs every step of a query at once (Chain).  `done` is set when the query is
// finished: res and the totals are as run_match leaves them, `final` the last
// step's rows.  Not set: the query does not qualify, an output had no room or a
// wait ran out; nothing is kept.
int run_chain(DevDB& db, const std::vector<Step>& steps, cudaStream_t s, uint64_t budget, bool count_only,
              HostStage* hs, std::vector<uint64_t>& totals, uint32_t*& final, bool& done) {
    done = false;
    final = nullptr;
    const size_t n = steps.size();
    if (db.max_degree > kEvenDegree || n < 2 || n > kChainSteps || steps[0].kind != STEP_SEED) return GVA_OK;
    for (const Step& st : steps)
        if (st.always_empty) return GVA_OK;
    uint32_t wmax = 1;
    for (size_t i = 1; i < n; ++i) {
        const Step& st = steps[i];
        if (st.kind == STEP_SEED || st.part == 0 || st.part > db.parts.size() || !db.parts[st.part - 1].off) return GVA_OK;
        wmax = std::max(wmax, st.kind == STEP_EXT ? st.width_in + 1 : st.width_in);
    }
    const uint64_t rows0 = db.seed_off[steps[0].label + 1] - db.seed_off[steps[0].label];
    if (rows0 == 0 || rows0 > kChainRows) return GVA_OK;
    // room for four times the seeds in every step: the frontiers of labelled
    // queries on such graphs mostly shrink
    const uint64_t cap = 4 * rows0 + 65536;
    const size_t bytes = cap * wmax * 4;
    // With few labels frontiers grow instead: a query that has no room runs
    // twice, as a chain that fails and counted.  A path / a star of four
    // vertices / a triangle on one label over 20,000 graphs of 20 to 60 vertices
    // took 530 / 715 / 203 us after an attempt, 340 / 388 / 201 us counted alone.
    double rows = (double)rows0;
    std::vector<uint32_t> lab(1, steps[0].label);
    for (size_t i = 1; i < n; ++i) {
        rows = expected_rows(db, steps[i], i, rows, lab);
        if (rows > (double)cap && !(count_only && i + 1 == n)) return GVA_OK;
    }
    const uint64_t most_tiles = (cap + kRowsPerBlock - 1) / kRowsPerBlock;
    // control: failed | tile counters | totals | statuses (one step more, for
    // the last step's second launch)
    const size_t o_tiles = 8, o_tot = o_tiles + 8 * (n + 1), o_status = o_tot + 8 * (n + 1);
    std::vector<size_t> status_at(n + 1);
    size_t ctl = o_status;
    for (size_t i = 1; i <= n; ++i) {
        status_at[i] = ctl;
        ctl += 8 * (i == 1 ? (rows0 + kRowsPerBlock - 1) / kRowsPerBlock : most_tiles);
    }
    const bool keep_rows = !count_only;
    const uint32_t w_last = steps[n - 1].kind == STEP_EXT ? steps[n - 1].width_in + 1 : steps[n - 1].width_in;
    // a result that is surely larger than kChainResult is written to the chain's
    // own memory and copied, for which a small one pays (its four-vertex paths on
    // labelled graphs, 100 KB: 97 us without, 111 with the copy); a second launch
    // of the last step takes as long as its first
    const bool via_buf = keep_rows && rows * w_last * 4 > 2.0 * kChainResult;
    const uint64_t room = via_buf ? cap : kChainResult / 4 / w_last;
    const size_t o_buf = align256(ctl), o_buf2 = o_buf + align256(bytes), need = o_buf2 + align256(bytes);
    if (need + (keep_rows && !via_buf ? kChainResult : 0) > budget) return GVA_OK;
    const int rc = set_smem_limits();
    if (rc) return rc;
    char* mem = nullptr;
    uint32_t* fin = nullptr;
    if (cudaMallocAsync((void**)&mem, need, s) != cudaSuccess) {
        cudaGetLastError();
        return GVA_OK;
    }
    struct Free {
        char* mem;
        cudaStream_t s;
        ~Free() { cudaFreeAsync(mem, s); }
    } free_mem{mem, s};
    if (keep_rows && !via_buf && cudaMallocAsync((void**)&fin, kChainResult, s) != cudaSuccess) {
        cudaGetLastError();
        return GVA_OK;
    }
    auto drop = [&]() {
        if (fin) cudaFreeAsync(fin, s);
        fin = nullptr;
    };
    volatile uint64_t* h_tot = hs->pinned + 8;
    volatile uint32_t* h_failed = (volatile uint32_t*)(hs->pinned + 7);
    for (size_t i = 0; i < n; ++i) h_tot[i] = 0;
    *h_failed = 0;
    cudaError_t e = cudaSuccess;
    auto launch = [&](size_t i, size_t slot, uint32_t* out, uint64_t cap_out) {
        const Step& st = steps[i];
        Chain c{};
        c.n_in = i == 1 ? nullptr : (uint64_t*)(mem + o_tot) + (i - 1);
        c.cap_in = cap;
        c.cap_out = cap_out;
        c.tiles = (unsigned long long*)(mem + o_tiles) + slot;
        c.status = (unsigned long long*)(mem + status_at[slot]);
        c.n_out = (uint64_t*)(mem + o_tot) + slot;
        c.host_out = const_cast<uint64_t*>(h_tot) + (i == slot ? i : 0);
        c.failed = (uint32_t*)mem;
        c.host_failed = const_cast<uint32_t*>(h_failed);
        c.polls = db.chain_polls;
        const uint32_t* in = i == 1 ? db.seed_verts + db.seed_off[steps[0].label] : (uint32_t*)(mem + (i & 1 ? o_buf2 : o_buf));
        // a CTA per tile of the seeds while they fit the chip at once (a tile
        // waits for the ones before it); later steps mostly have fewer, and a
        // CTA that finds none costs a launch slot: 1,184 CTAs for 228 tiles
        // took 16 us, 444 take 11
        const uint64_t tiles = (rows0 + kRowsPerBlock - 1) / kRowsPerBlock;
        const unsigned grid = (unsigned)(i == 1 ? std::min<uint64_t>(tiles, db.sms * 8)
                                                : std::min<uint64_t>(std::max<uint64_t>(2 * tiles, 64), db.sms * 3));
        const bool counts = count_only && i + 1 == n;
        auto start = [&](auto kernel, size_t smem, auto args) {
            cudaLaunchConfig_t cfg{};
            cfg.gridDim = dim3(grid);
            cfg.blockDim = dim3(kThreads);
            cfg.dynamicSmemBytes = smem;
            cfg.stream = s;
            cudaLaunchAttribute at{};
            at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
            at.val.programmaticStreamSerializationAllowed = 1;
            cfg.attrs = &at;
            cfg.numAttrs = i > 1 && slot == i ? 1 : 0;
            const cudaError_t le = cudaLaunchKernelEx(&cfg, kernel, args, c);
            if (e == cudaSuccess) e = le;
        };
        if (st.kind == STEP_EXT) {
            ExtArgs a;
            fill_ext(a, db, st, in, rows0, out);
            if (counts)
                start(chain_count_kernel<ExtArgs>, 0, a);
            else
                start(chain_ext_kernel, ext_smem_bytes(a.k, a.n_eq), a);
        } else {
            RedArgs a;
            fill_red(a, db, st, in, rows0, out);
            if (counts)
                start(chain_count_kernel<RedArgs>, 0, a);
            else
                start(chain_red_kernel, red_smem_bytes(a.k), a);
        }
        g_launches += 1;
    };
    // from here on errors of the driver end the query
    e = cudaMemsetAsync(mem, 0, ctl, s);
    uint32_t* const last_buf = (uint32_t*)(mem + ((n - 1) & 1 ? o_buf : o_buf2));
    for (size_t i = 1; i < n; ++i) {
        const bool last = i + 1 == n;
        uint32_t* out = last ? (via_buf ? last_buf : fin) : (uint32_t*)(mem + (i & 1 ? o_buf : o_buf2));
        launch(i, i, out, last ? room : cap);
    }
    if (e == cudaSuccess) e = cudaGetLastError();
    if (e == cudaSuccess) e = cudaEventRecord(hs->ev1, s);
    if (e == cudaSuccess) e = cudaEventSynchronize(hs->ev1);
    if (e != cudaSuccess) {
        drop();
        return fail(GVA_ERR_CUDA, cudaGetErrorString(e));
    }
    totals.assign(n, 0);
    totals[0] = rows0;
    bool reached = true;  // the last step's total is known
    for (size_t i = 1; i < n; ++i) totals[i] = h_tot[i];
    for (size_t i = 1; i + 1 < n; ++i) reached = reached && totals[i] <= cap;
    const bool big = keep_rows && *h_failed == 1 && reached && totals[n - 1] > room;
    if (*h_failed && !big) {  // an output had no room (or a wait ran out): counted steps
        drop();
        return GVA_OK;
    }
    // as the counted steps check it: every frontier that is written
    for (size_t i = 1; i < n; ++i) {
        const uint32_t w = steps[i].kind == STEP_EXT ? steps[i].width_in + 1 : steps[i].width_in;
        if (i + 1 == n && count_only) break;
        if (totals[i] * w * 4ull > budget) {
            drop();
            return fail(GVA_ERR_NOMEM, "frontier of " + std::to_string(totals[i]) + " rows exceeds the memory budget");
        }
    }
    if (keep_rows && totals[n - 1] == 0) drop();
    if (big || (via_buf && totals[n - 1])) {
        drop();
        if (cudaMallocAsync((void**)&fin, totals[n - 1] * w_last * 4, s) != cudaSuccess) {
            fin = nullptr;
            return fail(GVA_ERR_NOMEM, "frontier allocation failed");
        }
        *h_failed = 0;
        if (big) {
            e = cudaMemsetAsync(mem, 0, 8, s);  // the failure mark
            launch(n - 1, n, fin, totals[n - 1]);
        } else {
            e = cudaMemcpyAsync(fin, last_buf, totals[n - 1] * w_last * 4, cudaMemcpyDeviceToDevice, s);
        }
        if (e == cudaSuccess) e = cudaGetLastError();
        if (e == cudaSuccess) e = cudaEventRecord(hs->ev1, s);
        if (e == cudaSuccess) e = cudaEventSynchronize(hs->ev1);
        if (e != cudaSuccess || *h_failed) {  // a wait ran out, this time: counted steps
            drop();
            return e != cudaSuccess ? fail(GVA_ERR_CUDA, cudaGetErrorString(e)) : GVA_OK;
        }
    }
    final = fin;
    done = true;
    return GVA_OK;
}

int ensure_pool(int device) {
    static std::atomic<bool> done[64];
    if (device < 64 && done[device].load(std::memory_order_acquire)) return GVA_OK;
    cudaMemPool_t pool;
    GVA_CUDA(cudaDeviceGetDefaultMemPool(&pool, device));
    uint64_t keep = UINT64_MAX;  // keep freed frontier memory cached for the next phase / query
    GVA_CUDA(cudaMemPoolSetAttribute(pool, cudaMemPoolAttrReleaseThreshold, &keep));
    if (device < 64) done[device].store(true, std::memory_order_release);
    return GVA_OK;
}

}  // namespace

const char* const kKernelNames[K_NUM] = {"ext_count", "ext_write", "red_count", "red_write", "scan_block_sums",
                                         "mni_search"};

uint64_t kernel_launches() { return g_launches.load() + batch_kernel_launches() + mni_kernel_launches(); }

void Profiler::begin(int kind, double bytes, cudaStream_t s, cudaEvent_t& a) {
    (void)kind;
    (void)bytes;
    cudaEventCreate(&a);
    cudaEventRecord(a, s);
}

void Profiler::end(cudaEvent_t a, int kind, double bytes, cudaStream_t s, double rows) {
    cudaEvent_t b;
    cudaEventCreate(&b);
    cudaEventRecord(b, s);
    pending.push_back({kind, a, b, bytes, rows});
}

void Profiler::resolve() {
    for (auto& p : pending) {
        float ms = 0.f;
        cudaEventSynchronize(p.b);
        cudaEventElapsedTime(&ms, p.a, p.b);
        stat[p.kind].launches += 1;
        stat[p.kind].ms += ms;
        stat[p.kind].bytes += p.bytes;
        stat[p.kind].rows += p.rows;
        cudaEventDestroy(p.a);
        cudaEventDestroy(p.b);
    }
    pending.clear();
}

// ------------------------------------------------------------- database ----
int upload_graph(HostGraph& g, int device, DevDB*& out) {
    out = nullptr;
    int ndev = 0;
    GVA_CUDA(cudaGetDeviceCount(&ndev));
    if (device < 0 || device >= ndev) return fail(GVA_ERR_ARG, "device index out of range");
    GVA_CUDA(cudaSetDevice(device));
    // every engine (per-query, batched, MNI) allocates frontiers and round
    // buffers from the stream-ordered pool: keep freed memory cached there
    // instead of returning it to the driver at each synchronisation
    int prc = ensure_pool(device);
    if (prc) return prc;
    const uint32_t L = g.num_labels();
    // vertices grouped by dense label: the seed frontiers of init phases; the
    // same groups by total degree for rooted existence searches, which try
    // the vertices most likely to succeed first
    std::vector<uint32_t> seed_off, seed_verts, seed_deg;
    seed_groups(g, seed_off, seed_verts, seed_deg);
    // segment index per partition: packed 32-byte vertex records when the
    // label count allows (seg_of), else the dense (vertex, label) table
    bool packed = L >= 1 && L <= 28;
    for (auto& p : g.parts)
        if (!p.off.empty() && p.adj.size() >= 0x80000000ull) packed = false;
    std::vector<std::vector<uint32_t>> pidx(g.parts.size());
    if (packed) {
        const uint64_t nv = (uint64_t)g.max_id + 1;
        for (size_t i = 0; i < g.parts.size(); ++i) {
            const HostPartition& hp = g.parts[i];
            if (hp.off.empty()) continue;
            std::vector<uint32_t>& rec = pidx[i];
            rec.assign(nv * 8, 0);
            std::vector<uint32_t> wide;
            for (uint64_t v = 0; v < nv; ++v) {
                const uint32_t* o = hp.off.data() + v * L;
                const uint32_t base = o[0];
                uint32_t* r = rec.data() + v * 8;
                if (o[L] - base > 255) {
                    r[0] = base | 0x80000000u;
                    r[1] = (uint32_t)(nv * 8 + wide.size());
                    for (uint32_t j = 0; j <= L; ++j) wide.push_back(o[j] - base);
                } else {
                    r[0] = base;
                    unsigned char* b = reinterpret_cast<unsigned char*>(r);
                    for (uint32_t j = 1; j <= L; ++j) b[3 + j] = (unsigned char)(o[j] - base);
                }
            }
            if (nv * 8 + wide.size() >= 0x80000000ull) {
                packed = false;
                break;
            }
            rec.insert(rec.end(), wide.begin(), wide.end());
        }
        if (!packed) pidx.assign(g.parts.size(), {});
    }
    size_t bytes = 2 * align256(seed_verts.size() * 4 + 16);
    for (size_t i = 0; i < g.parts.size(); ++i)
        bytes += align256((packed ? pidx[i].size() : g.parts[i].off.size()) * 4) + align256(g.parts[i].adj.size() * 4 + 16);
    void* arena = nullptr;
    cudaError_t e = cudaMalloc(&arena, bytes);
    if (e != cudaSuccess) return fail(GVA_ERR_NOMEM, std::string("database allocation failed: ") + cudaGetErrorString(e));
    DevDB* db = new DevDB();
    db->device = device;
    cudaDeviceGetAttribute(&db->sms, cudaDevAttrMultiProcessorCount, device);
    db->max_id = g.max_id;
    db->L = L;
    db->packed = packed;
    db->labels = g.labels;
    db->seed_off = seed_off;
    for (uint32_t l = 0; l < L; ++l) {  // the first of each label's group by degree
        if (seed_off[l] == seed_off[l + 1]) continue;
        const uint64_t v = seed_deg[seed_off[l]];
        uint64_t deg = 0;
        for (const HostPartition& p : g.parts)
            if (!p.off.empty()) deg += p.off[v * L + L] - p.off[v * L];
        db->max_degree = std::max(db->max_degree, deg);
    }
    if (db->max_degree <= kEvenDegree) {  // for expected_rows: some of each label's vertices
        const size_t P = g.parts.size(), most = std::max<size_t>(16, 16384 / std::max<uint32_t>(L, 1));
        db->ends.assign(P * L, 0.0);
        db->bias.assign(P, 1.0);
        for (size_t p = 0; p < P; ++p) {
            const HostPartition& hp = g.parts[p];
            if (hp.off.empty()) continue;
            double all = 0, squares = 0;
            for (uint32_t l = 0; l < L; ++l) {
                const size_t n = seed_off[l + 1] - seed_off[l], m = std::min(n, most);
                uint64_t sum = 0, sq = 0;
                for (size_t i = 0; i < m; ++i) {
                    const uint32_t* o = hp.off.data() + (uint64_t)seed_verts[seed_off[l] + n * i / m] * L;
                    const uint64_t d = o[L] - o[0];
                    sum += d;
                    sq += d * d;
                }
                if (m == 0) continue;
                db->ends[p * L + l] = (double)sum * (double)n / (double)m;
                squares += (double)sq * (double)n / (double)m;
                all += db->ends[p * L + l];
            }
            if (all > 0) db->bias[p] = std::max(1.0, squares * (double)seed_verts.size() / (all * all));
        }
    }
    db->arena = arena;
    db->arena_bytes = bytes;
    char* cur = (char*)arena;
    auto put = [&](const std::vector<uint32_t>& v) -> const uint32_t* {
        const uint32_t* at = (const uint32_t*)cur;
        if (!v.empty()) cudaMemcpy(cur, v.data(), v.size() * 4, cudaMemcpyHostToDevice);
        cur += align256(v.size() * 4 + 16);
        return at;
    };
    db->seed_verts = put(seed_verts);
    db->seed_by_degree = put(seed_deg);
    db->parts.resize(g.parts.size());
    for (size_t i = 0; i < g.parts.size(); ++i) {
        HostPartition& hp = g.parts[i];
        if (hp.off.empty()) continue;
        const uint32_t* off = (const uint32_t*)cur;
        if (packed) {
            cudaMemcpy(cur, pidx[i].data(), pidx[i].size() * 4, cudaMemcpyHostToDevice);
            cur += align256(pidx[i].size() * 4);
        } else {
            cudaMemcpy(cur, hp.off.data(), hp.off.size() * 4, cudaMemcpyHostToDevice);
            cur += align256(hp.off.size() * 4);
        }
        db->parts[i].off = off;
        db->parts[i].adj = put(hp.adj);
        db->parts[i].n_adj = hp.adj.size();
        db->n_adj += hp.adj.size();
    }
    e = cudaDeviceSynchronize();
    if (e != cudaSuccess) {
        cudaFree(arena);
        delete db;
        return fail(GVA_ERR_CUDA, std::string("database upload failed: ") + cudaGetErrorString(e));
    }
    // keep label tables and partition presence for planning; drop host adjacency
    db->meta.max_id = g.max_id;
    db->meta.labels = g.labels;
    db->meta.parts.resize(g.parts.size());
    for (size_t i = 0; i < g.parts.size(); ++i)
        if (!g.parts[i].off.empty()) db->meta.parts[i].off.assign(1, 0);
    out = db;
    return GVA_OK;
}

void free_devdb(DevDB* db) {
    if (!db) return;
    if (db->arena || db->vgraph) cudaSetDevice(db->device);
    if (db->arena) {
        cudaFree(db->arena);
        trim_round_pool(db->device);
    }
    if (db->vgraph) cudaFree(db->vgraph);
    delete db;
}

size_t step_scratch_bytes(uint64_t in_rows) {
    const uint64_t nb = (in_rows + kRowsPerBlock - 1) / kRowsPerBlock;
    return align256((nb + 1) * sizeof(uint64_t));
}

// ---------------------------------------------------------- one step (L4) --
int run_step(DevDB& db, const Step& st, const uint32_t* in, uint64_t in_rows, uint32_t* out, uint64_t out_cap,
             uint64_t* out_rows, void* scratch, size_t scratch_bytes, cudaStream_t s) {
    if (!out_rows) return fail(GVA_ERR_ARG, "out_rows is null");
    *out_rows = 0;
    GVA_CUDA(cudaSetDevice(db.device));
    if (st.always_empty) return GVA_OK;
    if (st.kind == STEP_SEED) {
        const uint64_t n = db.seed_off[st.label + 1] - db.seed_off[st.label];
        *out_rows = n;
        if (n > out_cap) return fail(GVA_ERR_NOMEM, "output capacity too small");
        if (n) GVA_CUDA(cudaMemcpyAsync(out, db.seed_verts + db.seed_off[st.label], n * 4, cudaMemcpyDeviceToDevice, s));
        return GVA_OK;
    }
    if (in_rows == 0) return GVA_OK;
    if (!in || !scratch) return fail(GVA_ERR_ARG, "null device buffer");
    if (scratch_bytes < step_scratch_bytes(in_rows)) return fail(GVA_ERR_ARG, "scratch too small");
    uint64_t* sums = (uint64_t*)scratch;
    int rc = launch_count(db, st, in, in_rows, sums, s, nullptr);
    if (rc) return rc;
    const uint64_t nb = (in_rows + kRowsPerBlock - 1) / kRowsPerBlock;
    uint64_t total = 0;
    GVA_CUDA(cudaMemcpyAsync(&total, sums + nb, 8, cudaMemcpyDeviceToHost, s));
    GVA_CUDA(cudaStreamSynchronize(s));
    *out_rows = total;
    if (total > out_cap) return fail(GVA_ERR_NOMEM, "output capacity too small");
    if (total == 0) return GVA_OK;
    if (!out) return fail(GVA_ERR_ARG, "null output buffer");
    return launch_write(db, st, in, in_rows, out, sums, total, s, nullptr);
}

// ------------------------------------------------------- whole query (L3) --
int run_match(DevDB& db, const Plan& plan, const std::vector<Step>& steps, cudaStream_t s, uint64_t budget,
              bool count_only, bool profile, MatchResult& res) {
    Profiler profiler;
    Profiler* prof = profile ? &profiler : nullptr;
    GVA_CUDA(cudaSetDevice(db.device));
    int rc = ensure_pool(db.device);
    if (rc) return rc;
    res = MatchResult();
    res.device = db.device;
    res.stream = s;
    res.columns = plan.columns;
    res.phase_rows.assign(plan.phases.size(), 0);
    if (budget == 0) {  // 3/4 of the memory free at the database's first run (a driver query per call is costly)
        if (db.default_budget == 0) {
            size_t fr = 0, tot = 0;
            GVA_CUDA(cudaMemGetInfo(&fr, &tot));
            db.default_budget = (uint64_t)fr / 4 * 3;
        }
        budget = db.default_budget;
    }
    HostStage* hs = nullptr;
    rc = host_stage(db.device, hs);
    if (rc) return rc;
    cudaEvent_t ev0 = hs->ev0, ev1 = hs->ev1;
    GVA_CUDA(cudaEventRecord(ev0, s));

    if (!profile) {
        std::vector<uint64_t> totals;
        uint32_t* final = nullptr;
        bool done = false;
        rc = run_chain(db, steps, s, budget, count_only, hs, totals, final, done);
        if (rc) return rc;
        if (done) {
            float ms = 0.f;
            cudaEventElapsedTime(&ms, ev0, ev1);
            res.gpu_ms = ms;
            res.rows = totals.back();
            for (size_t i = 0; i < steps.size(); ++i) {
                if (steps[i].phase_end >= 0) res.phase_rows[steps[i].phase_end] = totals[i];
                if (totals[i] == 0) {
                    res.rows = 0;
                    break;
                }
            }
            res.width = (uint32_t)plan.columns.size();
            res.rows_dev = final;
            return GVA_OK;
        }
    }
    const uint32_t* cur = nullptr;
    uint32_t* owned = nullptr;  // frontier we must free
    uint64_t rows = 0;
    uint32_t width = 0;
    uint64_t* sums = nullptr;
    size_t sums_bytes = 0;
    uint64_t* total_h = hs->pinned;
    cudaError_t ce = cudaSuccess;
    int status = GVA_OK;
    bool counted_only = false;

    for (size_t i = 0; i < steps.size(); ++i) {
        const Step& st = steps[i];
        const bool last = (i + 1 == steps.size());
        const uint32_t out_w = st.kind == STEP_SEED ? 1 : (st.kind == STEP_EXT ? width + 1 : width);
        if (st.always_empty) {
            rows = 0;
        } else if (st.kind == STEP_SEED) {
            cur = db.seed_verts + db.seed_off[st.label];
            rows = db.seed_off[st.label + 1] - db.seed_off[st.label];
        } else if (rows > 0) {
            const size_t need = step_scratch_bytes(rows);
            if (need > sums_bytes) {
                if (sums) cudaFreeAsync(sums, s);
                ce = cudaMallocAsync((void**)&sums, need, s);
                if (ce != cudaSuccess) { status = fail(GVA_ERR_NOMEM, "scratch allocation failed"); sums = nullptr; break; }
                sums_bytes = need;
            }
            status = launch_count(db, st, cur, rows, sums, s, prof);
            if (status) break;
            const uint64_t nb = (rows + kRowsPerBlock - 1) / kRowsPerBlock;
            ce = cudaMemcpyAsync(total_h, sums + nb, 8, cudaMemcpyDeviceToHost, s);
            if (ce == cudaSuccess) ce = cudaStreamSynchronize(s);
            if (ce != cudaSuccess) { status = fail(GVA_ERR_CUDA, cudaGetErrorString(ce)); break; }
            uint64_t total = *total_h;
            if (total > 0 && !last && can_fuse(db, st, steps[i + 1])) {
                // this extension's rows are only needed by the reduction
                // after it: tested as they are generated, never written
                if (total * out_w * 4ull > budget) {
                    status = fail(GVA_ERR_NOMEM, "frontier of " + std::to_string(total) + " rows exceeds the memory budget");
                    break;
                }
                if (st.phase_end >= 0) res.phase_rows[st.phase_end] = total;
                const Step& rd = steps[i + 1];
                const uint64_t nch = num_chunks(db, total, nb);
                uint64_t* csums = nullptr;
                ce = cudaMallocAsync((void**)&csums, (nch + 1) * 8 + nch * mask_cap(chunk_of(db, total, nb), st.n_eq), s);
                if (ce != cudaSuccess) { status = fail(GVA_ERR_NOMEM, "scratch allocation failed"); break; }
                uint8_t* masks = (uint8_t*)(csums + nch + 1);
                status = launch_ext_red(db, st, rd, cur, rows, total, sums, csums, masks, nullptr, 0, s, prof);
                uint64_t kept = 0;
                if (!status) {
                    ce = cudaMemcpyAsync(total_h, csums + nch, 8, cudaMemcpyDeviceToHost, s);
                    if (ce == cudaSuccess) ce = cudaStreamSynchronize(s);
                    if (ce != cudaSuccess) status = fail(GVA_ERR_CUDA, cudaGetErrorString(ce));
                    kept = *total_h;
                }
                uint32_t* out = nullptr;
                const bool only_count = i + 2 == steps.size() && count_only;
                if (!status && kept && !only_count) {
                    if (kept * out_w * 4ull > budget) {
                        status = fail(GVA_ERR_NOMEM, "frontier of " + std::to_string(kept) + " rows exceeds the memory budget");
                    } else if (cudaMallocAsync((void**)&out, kept * out_w * 4ull, s) != cudaSuccess) {
                        out = nullptr;
                        status = fail(GVA_ERR_NOMEM, "frontier allocation failed");
                    } else {
                        status = launch_ext_red(db, st, rd, cur, rows, total, sums, csums, masks, out, kept, s, prof);
                        if (status) cudaFreeAsync(out, s);
                    }
                }
                cudaFreeAsync(csums, s);
                if (status) break;
                if (out) {
                    if (owned) cudaFreeAsync(owned, s);
                    owned = out;
                    cur = out;
                }
                rows = kept;
                counted_only = only_count;
                width = out_w;
                if (rd.phase_end >= 0) res.phase_rows[rd.phase_end] = rows;
                ++i;
                if (rows == 0) break;
                continue;
            }
            if (last && count_only) {
                rows = total;
                counted_only = true;
            } else if (total == 0) {
                rows = 0;
            } else {
                const uint64_t bytes = total * out_w * 4ull;
                if (bytes > budget) {
                    status = fail(GVA_ERR_NOMEM, "frontier of " + std::to_string(total) + " rows exceeds the memory budget");
                    break;
                }
                uint32_t* out = nullptr;
                ce = cudaMallocAsync((void**)&out, bytes, s);
                if (ce != cudaSuccess) { status = fail(GVA_ERR_NOMEM, "frontier allocation failed"); break; }
                status = launch_write(db, st, cur, rows, out, sums, total, s, prof);
                if (status) { cudaFreeAsync(out, s); break; }
                if (owned) cudaFreeAsync(owned, s);
                owned = out;
                cur = out;
                rows = total;
            }
        }
        width = out_w;
        if (st.phase_end >= 0) res.phase_rows[st.phase_end] = rows;
        if (rows == 0) break;
    }
    if (sums) cudaFreeAsync(sums, s);
    if (status) {
        if (owned) cudaFreeAsync(owned, s);
        if (prof) prof->resolve();
        return status;
    }
    GVA_CUDA(cudaEventRecord(ev1, s));
    GVA_CUDA(cudaEventSynchronize(ev1));
    float ms = 0.f;
    cudaEventElapsedTime(&ms, ev0, ev1);
    res.gpu_ms = ms;
    if (prof) {
        prof->resolve();
        for (int i = 0; i < K_NUM; ++i) res.kstat[i] = prof->stat[i];
    }
    // the final width is the number of columns of the plan
    res.width = (uint32_t)plan.columns.size();
    res.rows = rows;
    if (rows == 0 || counted_only) {
        if (owned) cudaFreeAsync(owned, s);
        res.rows_dev = nullptr;
    } else if (owned) {
        res.rows_dev = owned;
    } else {
        // the final frontier is still the seed list (cannot happen: a plan ends with an extension or reduction)
        res.rows_dev = nullptr;
    }
    GVA_CUDA(cudaStreamSynchronize(s));
    return GVA_OK;
}

void free_result(MatchResult* r) {
    if (!r) return;
    if (r->rows_dev) {
        cudaSetDevice(r->device);
        cudaFreeAsync(r->rows_dev, r->stream);
        cudaStreamSynchronize(r->stream);
    }
    delete r;
}

}  // namespace gva
