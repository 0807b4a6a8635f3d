// Segment-linking kernels for sm_103a.
//
// Every stage follows the same pattern, batched over all events:
//   count  - per inner object, the number of candidate pairs the reference's
//            loop would test (Event.cc:257-301, 472-521, 635-691, ...);
//   scan   - exclusive prefix sum -> a flat candidate space [0, total);
//   enum   - a persistent, work-stealing grid: each warp takes 256
//            consecutive candidates, maps them back to (inner, outer) objects,
//            applies the reference's cuts and appends the survivors with a
//            warp-aggregated atomic, ranking each survivor inside its inner
//            module;
//   group  - per-module counts are scanned and the survivors scattered into
//            dense arrays grouped by inner module (objects of one event stay
//            contiguous).
// Triplets and track candidates are exact equi-joins on the shared
// mini-doublet / segment instead of the reference's all-pairs loops.
#include <cstdio>

#include "sdl_kernels.h"

namespace sdlg {

namespace {

// Bounds checks of every global-memory index (debug builds with
// -DSDL_DEVICE_CHECKS): a bad index is recorded in b.dbg (count, source line,
// index, limit) and the access is redirected to element 0 instead of faulting.
#ifdef SDL_DEVICE_CHECKS
__device__ __forceinline__ int64_t checked_idx(int64_t i, int64_t lim, int line, unsigned long long* dbg) {
    if (i >= 0 && i < lim) return i;
    if (atomicAdd(dbg, 1ull) == 0ull) {
        dbg[1] = (unsigned long long)line;
        dbg[2] = (unsigned long long)i;
        dbg[3] = (unsigned long long)lim;
    }
    return 0;
}
#define IX(i, lim) checked_idx((int64_t)(i), (int64_t)(lim), __LINE__, b.dbg)
#else
#define IX(i, lim) (i)
#endif
#define AT(arr, i, lim) (arr)[IX(i, lim)]

constexpr int kWarp = 32;
constexpr int kEnumThreads = 256;

// the launch's device time stamps (none for most launches)
__device__ __forceinline__ void stamp(const BatchDev& b) {
    if (b.ts == 0u || (blockIdx.x | blockIdx.y | threadIdx.x) != 0u) return;
    unsigned long long t;
    asm volatile("mov.u64 %0, %globaltimer;" : "=l"(t));
    for (uint32_t m = b.ts; m; m &= m - 1u) b.stamps[__ffs(m) - 1] = t;
}

// the start of every kernel behind a stage that can overflow: true when the
// run stops there
__device__ __forceinline__ bool halted(const BatchDev& b) {
    stamp(b);
    return (*b.status & kStatusHalt) != 0;
}

// add v to *addr with one atomic per group of lanes sharing the address;
// every lane of the warp must call it
__device__ __forceinline__ void warp_add(uint32_t* addr, uint32_t v, bool active) {
    const unsigned act = __ballot_sync(0xffffffffu, active);
    if (!active) return;
    const unsigned peers = __match_any_sync(act, (unsigned long long)(uintptr_t)addr);
    const uint32_t sum = __reduce_add_sync(peers, v);
    if ((int)(threadIdx.x & 31) == __ffs(peers) - 1) atomicAdd(addr, sum);
}

// largest i in [lo, hi] with off[i] <= c (off has `lim` entries)
__device__ __forceinline__ int find_obj(const BatchDev& b, const int64_t* off, int64_t lim, int lo, int hi, int64_t c) {
    while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (AT(off, mid, lim) <= c) lo = mid;
        else hi = mid - 1;
    }
    return lo;
}

// Bucket table of a stage's flat candidate space: bucket[k] is the inner
// object that holds candidate k * 2^kBucketShift, plus a last entry nobj - 1.
// A candidate c then lies in an inner object between bucket[c >> shift] and
// bucket[(c >> shift) + 1], so the enumerators search a few objects instead
// of all of them.  A table too small for the candidate space is not built
// and the search covers the whole range.
constexpr int kBucketShift = 8;

__device__ __forceinline__ bool buckets_ok(const BatchDev& b, int64_t total) {
    return ((total + (1ll << kBucketShift) - 1) >> kBucketShift) + 1 <= b.bucket_cap;
}

// search bounds of the inner objects of candidates c0 <= c1
__device__ __forceinline__ void obj_bounds(const BatchDev& b, int64_t nobj, int64_t total, int64_t c0, int64_t c1, int& lo,
                                           int& hi) {
    if (buckets_ok(b, total)) {
        lo = AT(b.bucket, c0 >> kBucketShift, b.bucket_cap);
        hi = AT(b.bucket, (c1 >> kBucketShift) + 1, b.bucket_cap);
    } else {
        lo = 0;
        hi = (int)nobj - 1;
    }
}

// array sizes
__device__ __forceinline__ int64_t H(const BatchDev& b) { return b.n_hit_cap; }
__device__ __forceinline__ int64_t NG1(const BatchDev& b) { return (int64_t)b.n_gm + 1; }
// event and module of a global module index g = event * n_mod + module
// (0 <= g < 2^31): floor(g * ceil(2^64 / n) / 2^64) is floor(g / n) exactly
// for g and n = n_mod below 2^32 (the rounding-up error is below 2^-32 < 1 / n)
__device__ __forceinline__ int ev_of(const BatchDev& b, int64_t g) {
    return b.geo.n_mod == 1 ? (int)g : (int)__umul64hi((unsigned long long)g, b.geo.n_mod_inv);
}
__device__ __forceinline__ int mod_of(const BatchDev& b, int64_t g) {
    return (int)(g - (int64_t)ev_of(b, g) * b.geo.n_mod);
}
__device__ __forceinline__ int64_t NM(const BatchDev& b) { return b.geo.n_mod; }
__device__ __forceinline__ int64_t NC(const BatchDev& b) { return b.geo.n_conn > 0 ? b.geo.n_conn : 1; }
__device__ __forceinline__ int64_t NCP(const BatchDev& b) {
    const int64_t v = (int64_t)b.n_ev * b.geo.n_conn;
    return v > 0 ? v : 1;
}
__device__ __forceinline__ const ModDev& MOD(const BatchDev& b, int64_t m) { return AT(b.geo.mod, m, NM(b)); }

// ------------------------------------------------------------------ scan
// Exclusive prefix sums in one pass (decoupled look-back, after Merrill and
// Garland 2016): each CTA takes the next tile from a counter, so that every
// tile before its own has been started, publishes the tile's sum, adds up
// its predecessors' words (a sum, or already a whole prefix), one per thread,
// and publishes its prefix.  The whole CTA looks back because the tiles in
// flight publish their sums at about the same time, so that a tile has
// hundreds of sums to add before it meets a prefix.  What is summed is computed where it is loaded (the
// candidate counts with their layer counters) and what is derived from the
// prefix is written where it is stored (offsets, bucket and tile tables), so
// one launch does what took a count kernel, three scan kernels and a table
// kernel: 17 of a run's launches instead of 85, and of a 2.3k-hit event's
// 646 us in kernels those took 290.
//
// A word holds its kind in the top two bits (0: not there yet, 1: the tile's
// sum, 2: the prefix through the tile).  The words are cleared with the run's
// other counts, one slot per scan of a run.  A wait for a predecessor is
// bounded: past kScanPolls the CTA sets kStatusScan, which halts the run.
constexpr int kScanThreads = 512;
constexpr int kScanPolls = 1 << 20;
constexpr unsigned long long kScanSum = 1ull << 62, kScanPrefix = 2ull << 62, kScanValue = (1ull << 62) - 1;

__device__ __forceinline__ unsigned long long scan_peek(const unsigned long long* p) {
    unsigned long long v;
    asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ void scan_post(unsigned long long* p, unsigned long long v) {
    asm volatile("st.relaxed.gpu.global.u64 [%0], %1;" ::"l"(p), "l"(v) : "memory");
}

// the sums of the tiles before `tile` (kK values per tile); the whole CTA
// calls it, and every thread gets them
template <int kK>
struct ScanBack {
    int64_t sum[kK][kScanThreads / kWarp];
    bool done[kK][kScanThreads / kWarp];  // a prefix is among the warp's words
    int ok;
};
template <int kK>
__device__ __forceinline__ bool scan_lookback(const unsigned long long* words, int64_t tile, ScanBack<kK>& sb, int64_t* pre) {
    constexpr int kWarps = kScanThreads / kWarp;
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    bool open[kK];
#pragma unroll
    for (int q = 0; q < kK; ++q) {
        pre[q] = 0;
        open[q] = true;
    }
    for (int64_t t = tile - 1;; t -= kScanThreads) {
        const int64_t k = t - threadIdx.x;
#pragma unroll
        for (int q = 0; q < kK; ++q) {
            unsigned long long x = kScanPrefix;  // before the first tile: a prefix of 0
            if (k >= 0) {
                for (int polls = 0; ((x = scan_peek(words + k * kK + q)) >> 62) == 0ull; ++polls)
                    if (polls == kScanPolls) {
                        sb.ok = 0;
                        break;
                    }
            }
            const unsigned m = __ballot_sync(0xffffffffu, (x >> 62) == 2ull);
            const int last = m ? __ffs(m) - 1 : kWarp;  // the nearest prefix
            int64_t v = lane <= last ? (int64_t)(x & kScanValue) : 0;
            for (int o = 16; o; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
            if (lane == 0) {
                sb.sum[q][w] = v;
                sb.done[q][w] = m != 0u;
            }
        }
        __syncthreads();
        if (!sb.ok) return false;
        bool all = true;
#pragma unroll
        for (int q = 0; q < kK; ++q) {
            for (int j = 0; j < kWarps && open[q]; ++j) {
                pre[q] += sb.sum[q][j];
                open[q] = !sb.done[q][j];
            }
            all = all && !open[q];
        }
        if (all) return true;
        __syncthreads();  // the words' sums have been read
    }
}

template <class Op, int kI>
__global__ void __launch_bounds__(kScanThreads) k_scan(BatchDev b, int slot) {
    constexpr int kK = Op::kVals, kWarps = kScanThreads / kWarp;
    constexpr int kTile = kScanThreads * kI;
    // (a scan can halt the run itself while its last CTAs start, so the CTA
    // decides as one)
    if (__syncthreads_or(halted(b))) return;
    Op::begin(b);
    const int64_t n = Op::size(b);
    const int64_t ntile = n > 0 ? (n + kTile - 1) / kTile : 1;
    unsigned long long* ticket = b.scan_state + (int64_t)slot * b.scan_cap;
    unsigned long long* words = ticket + 1;
    __shared__ int64_t s_tile, s_sum[kK][kWarps];
    __shared__ ScanBack<kK> s_back;
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    for (;;) {
        if (threadIdx.x == 0) {
            s_tile = (int64_t)atomicAdd(ticket, 1ull);
            s_back.ok = 1;
        }
        __syncthreads();
        const int64_t tile = s_tile;
        if (tile >= ntile) return;
        const int64_t base = tile * kTile + w * (kWarp * kI) + lane;
        int64_t v[kI][kK], e[kI][kK], carry[kK];
#pragma unroll
        for (int k = 0; k < kI; ++k) Op::load(b, base + k * kWarp, base + k * kWarp < n, v[k]);
#pragma unroll
        for (int q = 0; q < kK; ++q) {
            carry[q] = 0;
#pragma unroll
            for (int k = 0; k < kI; ++k) {
                int64_t x = v[k][q];
#pragma unroll
                for (int o = 1; o < kWarp; o <<= 1) {
                    const int64_t y = __shfl_up_sync(0xffffffffu, x, o);
                    if (lane >= o) x += y;
                }
                e[k][q] = carry[q] + x - v[k][q];
                carry[q] += __shfl_sync(0xffffffffu, x, kWarp - 1);
            }
            if (lane == 0) s_sum[q][w] = carry[q];
        }
        __syncthreads();
        int64_t total[kK], before[kK];
#pragma unroll
        for (int q = 0; q < kK; ++q) {
            total[q] = before[q] = 0;
#pragma unroll
            for (int j = 0; j < kWarps; ++j) {
                if (j < w) before[q] += s_sum[q][j];
                total[q] += s_sum[q][j];
            }
        }
        int64_t pre[kK];
#pragma unroll
        for (int q = 0; q < kK; ++q) {
            pre[q] = 0;
            if (threadIdx.x == 0 && tile > 0) scan_post(words + tile * kK + q, kScanSum | (unsigned long long)total[q]);
        }
        if (tile > 0 && !scan_lookback<kK>(words, tile, s_back, pre)) {
            if (threadIdx.x == 0) atomicOr(b.status, kStatusScan);
            return;
        }
        if (threadIdx.x == 0) {
#pragma unroll
            for (int q = 0; q < kK; ++q) scan_post(words + tile * kK + q, kScanPrefix | (unsigned long long)(pre[q] + total[q]));
        }
#pragma unroll
        for (int k = 0; k < kI; ++k) {
            const int64_t i = base + k * kWarp;
#pragma unroll
            for (int q = 0; q < kK; ++q) e[k][q] += pre[q] + before[q];
            if (i < n) Op::store(b, i, e[k], v[k]);
        }
        if (tile == ntile - 1 && threadIdx.x == 0) {
#pragma unroll
            for (int q = 0; q < kK; ++q) total[q] += pre[q];
            Op::total(b, n, total);
        }
    }
}
struct ScanOp {
    __device__ static void begin(const BatchDev&) {}
};

// ------------------------------------------------------------------ ingest
__global__ void k_hit_map(BatchDev b) {
    const int64_t n = *b.n_hit;
    for (int64_t h = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; h < n; h += (int64_t)gridDim.x * blockDim.x) {
        int lo = 0, hi = b.n_ev;  // event: largest e with ev_off[e] <= h
        while (hi - lo > 1) {
            const int mid = (lo + hi) >> 1;
            if (AT(b.ev_off, mid, b.n_ev + 1) <= h) lo = mid;
            else hi = mid;
        }
        const int ev = lo;
        const uint32_t d = AT(b.in_det, h, H(b));
        int a = 0, c = b.geo.n_mod;  // first module with detid >= d
        while (a < c) {
            const int mid = (a + c) >> 1;
            if (AT(b.geo.detid, mid, NM(b)) < d) a = mid + 1;
            else c = mid;
        }
        int gm = -1, rank = 0;
        if (a < b.geo.n_mod && AT(b.geo.detid, a, NM(b)) == d) {
            gm = ev * b.geo.n_mod + a;
            rank = (int)atomicAdd((unsigned long long*)&AT(b.mod_hit, gm, NG1(b)), 1ull);
        } else {
            atomicOr(b.status, kStatusUnknownModule);
        }
        AT(b.hit_gm, h, H(b)) = gm;
        AT(b.hit_rank, h, H(b)) = rank;
    }
}

// hits per global module -> offsets
struct ScanHits : ScanOp {
    static constexpr int kVals = 1, kSmall = 2, kBig = 8;
    __device__ static int64_t size(const BatchDev& b) { return b.n_gm; }
    __device__ static void load(const BatchDev& b, int64_t i, bool in, int64_t* v) { v[0] = in ? AT(b.mod_hit, i, NG1(b)) : 0; }
    __device__ static void store(const BatchDev& b, int64_t i, const int64_t* e, const int64_t*) { AT(b.mod_hit, i, NG1(b)) = e[0]; }
    __device__ static void total(const BatchDev& b, int64_t n, const int64_t* t) { AT(b.mod_hit, n, NG1(b)) = t[0]; }
};

// sorted position of every input hit in a known module -> hit_perm
__global__ void k_hit_perm(BatchDev b) {
    if (halted(b)) return;
    const int64_t n = *b.n_hit;
    for (int64_t h = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; h < n; h += (int64_t)gridDim.x * blockDim.x) {
        const int gm = AT(b.hit_gm, h, H(b));
        if (gm < 0) continue;
        AT(b.hit_perm, AT(b.mod_hit, gm, NG1(b)) + AT(b.hit_rank, h, H(b)), H(b)) = (int)h;
    }
}

// asin(min(rt * k, .95)) of a hit
__device__ __forceinline__ float rt_asin(float rt) { return g_asin(fmin_ref(rt * k2Rinv1GeVf / kPtCut, kSinAlphaMax)); }

// The sorted hit arrays, one thread per sorted position (coalesced writes;
// the input hit is gathered through hit_perm) and part (blockIdx.y): the hit,
// its direction and, where its pair's dPhiThreshold reads it, its asin term;
// and the strip shift of the hits that anchor their pair.  Bound by the
// instructions of the float-float functions (64 events: 588 us with every
// function for every hit in one thread, a third of it stalled on instruction
// fetches; 339 in two parts, with the segments' terms left to k_md_pack;
// 391 with the asin in a part of its own, which gathers each hit once more).
__global__ void k_hit_scatter(BatchDev b) {
    if (halted(b)) return;
    const int64_t n = min(AT(b.mod_hit, b.n_gm, NG1(b)), *b.n_hit);  // hits in known modules
    for (int64_t pos = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; pos < n; pos += (int64_t)gridDim.x * blockDim.x) {
        const int64_t h = AT(b.hit_perm, pos, H(b));
        const int gm = AT(b.hit_gm, h, H(b));
        const float x = AT(b.in_x, h, H(b)), y = AT(b.in_y, h, H(b)), z = AT(b.in_z, h, H(b));
        const int m = mod_of(b, gm);
        const ModDev& M = MOD(b, m);
        const int lmi = M.lower ? m : M.partner;
        const bool pair = lmi >= 0;
        const ModDev& lm = MOD(b, pair ? lmi : m);
        const bool lower = (bool)M.lower;
        if (blockIdx.y == 0) {
            const P3 p = mk(x, y, z);
            AT(b.hx, pos, H(b)) = x; AT(b.hy, pos, H(b)) = y; AT(b.hz, pos, H(b)) = z;
            AT(b.hrt, pos, H(b)) = p.rt; AT(b.hphi, pos, H(b)) = p.phi; AT(b.hr3, pos, H(b)) = p.r3;
            AT(b.hidx, pos, H(b)) = AT(b.in_idx, h, H(b));
            AT(b.hgm, pos, H(b)) = gm;
            AT(b.ha1, pos, H(b)) = pair && (lm.ltype == kPixel) == lower ? rt_asin(p.rt) : 0.f;
        } else {
            P3 p;
            p.x = x; p.y = y; p.z = z;
            p.rt = __fsqrt_rn(__fadd_rn(__fmul_rn(x, x), __fmul_rn(y, y)));
            float xa = 0.f, ya = 0.f, zn = 0.f;
            if (pair && md_shifts(lm) && md_upper_anchors(lm) != lower) shift_anchor(p, lm, xa, ya, zn);
            AT(b.hsx, pos, H(b)) = xa; AT(b.hsy, pos, H(b)) = ya; AT(b.hsz, pos, H(b)) = zn;
        }
    }
}

// ------------------------------------------------------------------ helpers
__device__ __forceinline__ uint32_t* counter_at(const BatchDev& b, int ev, int st, int kind, int slot) {
    return &AT(b.counters, (int64_t)ev * 110 + st * 22 + kind * 11 + slot, (int64_t)b.n_ev * 110);
}

__device__ __forceinline__ P3 hit(const BatchDev& b, int64_t k) {
    P3 p;
    p.x = AT(b.hx, k, H(b)); p.y = AT(b.hy, k, H(b)); p.z = AT(b.hz, k, H(b));
    p.rt = AT(b.hrt, k, H(b)); p.phi = AT(b.hphi, k, H(b)); p.r3 = AT(b.hr3, k, H(b));
    return p;
}

__device__ __forceinline__ int md_anchor(const ModDev& lm, int lo, int up) {
    return (lm.type == kPS && lm.ltype != kPixel) ? up : lo;  // MiniDoublet.cc:60-81
}

// object arrays of stage st
__device__ __forceinline__ int OI(const BatchDev& b, int st, int64_t k) { return AT(b.obj[st].i, k, b.obj[st].cap); }
__device__ __forceinline__ int OJ(const BatchDev& b, int st, int64_t k) { return AT(b.obj[st].j, k, b.obj[st].cap); }
__device__ __forceinline__ int OG(const BatchDev& b, int st, int64_t k) { return AT(b.obj[st].g, k, b.obj[st].cap); }
__device__ __forceinline__ float OF(const BatchDev& b, int st, int f, int64_t k) {
    const Objs& O = b.obj[st];
    return AT(O.f, (int64_t)f * O.cap + k, O.cap * (O.nf > 0 ? O.nf : 1));
}
__device__ __forceinline__ int64_t OFF(const BatchDev& b, int st, int64_t g) { return AT(b.obj[st].mod_cnt, g, NG1(b)); }
__device__ __forceinline__ int64_t n_objects(const BatchDev& b, int st) { return min(OFF(b, st, b.n_gm), b.obj[st].cap); }


// ------------------------------------------------------------------ stage functors
// mini-doublet candidate q of lower module gm: its two hits' sorted positions
__device__ __forceinline__ bool md_candidate(const BatchDev& b, int gm, int64_t q, int2& e) {
    const int ev = ev_of(b, gm);
    const int pg = ev * b.geo.n_mod + MOD(b, gm - ev * b.geo.n_mod).partner;
    const int64_t u0 = AT(b.mod_hit, pg, NG1(b)), nu = AT(b.mod_hit, pg + 1, NG1(b)) - u0;
    if (nu <= 0) {
#ifdef SDL_DEVICE_CHECKS
        IX(-1, 0);
#endif
        return false;
    }
    const int64_t i = (q | nu) >> 32 ? q / nu : (int64_t)((uint32_t)q / (uint32_t)nu);
    e = make_int2((int)(AT(b.mod_hit, gm, NG1(b)) + i), (int)(u0 + (q - i * nu)));
    return true;
}
// what the mini-doublet cuts read of a candidate
struct MDCand {
    P3 L, U;
    float pixAsin, sh[3];
};
__device__ __forceinline__ MDCand md_cand(const BatchDev& b, const ModDev& lm, int2 e) {
    const int lo = e.x, up = e.y;
    MDCand c;
    c.L = hit(b, lo);
    c.U = hit(b, up);
    c.pixAsin = lm.ltype == kPixel ? AT(b.ha1, lo, H(b)) : AT(b.ha1, up, H(b));
    const int anc = md_upper_anchors(lm) ? up : lo;
    c.sh[0] = AT(b.hsx, anc, H(b)); c.sh[1] = AT(b.hsy, anc, H(b)); c.sh[2] = AT(b.hsz, anc, H(b));
    return c;
}

// conn entry k of module m for the flat index q, given per-entry exclusive prefixes
__device__ __forceinline__ int conn_entry(const BatchDev& b, int ev, int m, int64_t q, int& pref) {
    const int k0 = AT(b.geo.conn_off, m, NM(b) + 1), k1 = AT(b.geo.conn_off, m + 1, NM(b) + 1);
    const int64_t base = (int64_t)ev * b.geo.n_conn;
    int lo = k0, hi = k1 - 1;
    while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (AT(b.conn_pref, base + mid, NCP(b)) <= q) lo = mid;
        else hi = mid - 1;
    }
    pref = AT(b.conn_pref, base + lo, NCP(b));
    return lo;
}

// One 64-byte record per mini-doublet for the segment stage (k_md_pack):
// the anchor hit with its derived quantities and asin / tan terms, the
// mini-doublet's four floats, the lower module and the anchor's module.
struct MDRec {
    MDView v;
    float a1, tf;  // asin(min(rt*k,.95)) and its float tan, of the anchor hit
    int anc_mod;   // module of the anchor hit
    float c0, c1;  // barrel: sdCut for the layer below (c0); endcap: strip-edge phis (hi, lo)
};
__device__ __forceinline__ MDRec md_rec(const BatchDev& b, int64_t a) {
    const float4* q = reinterpret_cast<const float4*>(&AT(b.mdpack, a * kMdPack, b.obj[kMD].cap * kMdPack));
    const float4 r0 = __ldg(q), r1 = __ldg(q + 1), r2 = __ldg(q + 2), r3 = __ldg(q + 3);
    MDRec r;
    r.v.a.x = r0.x; r.v.a.y = r0.y; r.v.a.z = r0.z; r.v.a.rt = r0.w;
    r.v.a.phi = r1.x; r.v.a.r3 = r1.y; r.a1 = r1.z; r.tf = r1.w;
    r.v.dz = r2.x; r.v.shiftedDz = r2.y; r.v.dphi = r2.z; r.v.dphichange = r2.w;
    r.v.m = &MOD(b, __float_as_int(r3.x));
    r.anc_mod = __float_as_int(r3.y);
    r.c0 = r3.z;
    r.c1 = r3.w;
    return r;
}

__device__ __forceinline__ MDLite md_lite(const BatchDev& b, int64_t a) {
    const float4* q = reinterpret_cast<const float4*>(&AT(b.mdlite, a * kMdLite, b.obj[kMD].cap * kMdLite));
    const float4 r0 = __ldg(q), r1 = __ldg(q + 1);
    return MDLite{r0.x, r0.y, r0.z, r0.w, r1.x, r1.y, r1.z, r1.w, __float_as_uint(r1.w) & kMdFlags};
}
// One thread per mini-doublet and part (blockIdx.y): the records with the
// anchor's bend terms; the endcap strip edges' phi and the third-layer asin.
__global__ void __launch_bounds__(256, 4) k_md_pack(BatchDev b) {
    if (halted(b)) return;
    const int64_t n = n_objects(b, kMD);
    const int part = blockIdx.y;
    for (int64_t a = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; a < n; a += (int64_t)gridDim.x * blockDim.x) {
        const int lm = mod_of(b, OG(b, kMD, a));
        const ModDev& M = MOD(b, lm);
        const int anc = md_anchor(M, OI(b, kMD, a), OJ(b, kMD, a));
        const bool barrel = M.subdet == kBarrel;
        float4* q = reinterpret_cast<float4*>(&AT(b.mdpack, a * kMdPack, b.obj[kMD].cap * kMdPack));
        float* bend = &AT(b.mdbend, 2 * a, 2 * b.obj[kMD].cap);
        const P3 p = hit(b, anc);
        if (part == 1) {
            bend[1] = g_asin(fmin_ref(p.rt * k2Rinv1GeVf / 3.0f, kSinAlphaMax));
            // what the segment algorithms compute from this mini-doublet alone
            // as the outer one: the endcap strip edges' phi
            if (barrel) continue;
            float c0 = p.phi, c1 = p.phi;
            if (M.type == kTwoS) {
                const ModDev& A = MOD(b, mod_of(b, AT(b.hgm, anc, H(b))));
                c0 = strip_edge(p, A, true).phi;
                c1 = strip_edge(p, A, false).phi;
            }
            reinterpret_cast<float2*>(q + 3)[1] = make_float2(c0, c1);
            continue;
        }
        // (the anchor that is not the pair's pixel side has no asin term yet)
        const float a1 = md_upper_anchors(M) || M.ltype == kPixel ? AT(b.ha1, anc, H(b)) : rt_asin(p.rt);
        float tf;
        g_tan_both(a1, tf, bend[0]);
        q[0] = make_float4(p.x, p.y, p.z, p.rt);
        q[1] = make_float4(p.phi, p.r3, a1, tf);
        q[2] = make_float4(OF(b, kMD, 0, a), OF(b, kMD, 1, a), OF(b, kMD, 2, a), OF(b, kMD, 3, a));
        reinterpret_cast<float2*>(q + 3)[0] = make_float2(__int_as_float(lm), __int_as_float(mod_of(b, AT(b.hgm, anc, H(b)))));
        // and the barrel cut for the layer below
        float c0 = 0.f;
        if (barrel) {
            if (M.layer >= 2) c0 = sg_barrel_cut(M.layer - 1, p.rt, a1);
            reinterpret_cast<float2*>(q + 3)[1] = make_float2(c0, 0.f);
        }
        // the first pass's record (sg_first_cuts, sg_later_cuts)
        float4* l = reinterpret_cast<float4*>(&AT(b.mdlite, a * kMdLite, b.obj[kMD].cap * kMdLite));
        l[0] = make_float4(p.rt, p.z, p.phi, barrel ? c0 : a1);
        const float lum = barrel ? (M.side != kCenter ? M.tilt : 0.f)
                                 : 15.f * OF(b, kMD, 2, a) / OF(b, kMD, M.type == kPS ? 1 : 0, a);
        const uint32_t fl = (uint32_t)(M.layer & 15) | (barrel ? kMdBarrel : kMdEndcap);
        l[1] = make_float4(barrel ? tf / a1 : a1 / tf, lum, OF(b, kMD, 3, a),
                           __uint_as_float((__float_as_uint(0.02f / M.gap) & ~kMdFlags) | fl));
    }
}

// segment algorithm on inner MD a and outer MD bmd (Segment.cc:337-859);
// `connected`: the outer MD's module is in the inner module's connection list
// (the endcap algorithm's first requirement, Segment.cc:613-633)
// kOuter: 0 either algorithm, 1 only the barrel one (outer MD in the barrel),
// 2 only the endcap one (a kernel compiled for one keeps the other's code out
// of its instruction caches); a candidate of the other kind fails
template <int kOuter = 0>
__device__ __forceinline__ bool sg_pair_rec(const MDView& im, const MDRec& orec, bool connected, float* fv) {
    const MDView& om = orec.v;
    SGVals v;
    v.dphi = v.dphimin = v.dphimax = v.dphichange = v.dphiminchange = v.dphimaxchange = 0.f;
    bool pass = false;
    const bool ob = om.m->subdet == kBarrel;
    if (kOuter != 2 && ob) pass = sg_barrel(im, om, orec.a1, orec.tf, orec.c0, v);
    else if (kOuter != 1 && !ob) pass = sg_endcap(im, om, orec.a1, orec.tf, connected, orec.c0, orec.c1, v);
    fv[0] = v.dphi; fv[1] = v.dphimin; fv[2] = v.dphimax;
    fv[3] = v.dphichange; fv[4] = v.dphiminchange; fv[5] = v.dphimaxchange;
    return pass;
}
__device__ __forceinline__ bool sg_pair(const BatchDev& b, int a, int bmd, bool connected, float* fv) {
    return sg_pair_rec(md_rec(b, a).v, md_rec(b, bmd), connected, fv);
}

// segment candidates along the module map (Event.cc:445-522): candidate q of
// inner MD a is an MD of a connected module, in connection-list order
__device__ __forceinline__ int sg_outer_conn(const BatchDev& b, int a, int64_t q) {
    const int n_mod = b.geo.n_mod;
    const int g1 = OG(b, kMD, a);
    const int ev = ev_of(b, g1), m1 = g1 - ev * n_mod;
    int pref;
    const int k = conn_entry(b, ev, m1, q, pref);
    const int g2 = ev * n_mod + AT(b.geo.conn_idx, k, NC(b));
    return (int)(OFF(b, kMD, g2) + (q - pref));
}
__device__ __forceinline__ int sg_outer_md(const BatchDev& b, int a, int64_t q) {
    const int g1 = OG(b, kMD, a);
    if (AT(b.toff, b.n_gm, NG1(b)) <= b.olist_cap) return AT(b.olist, AT(b.toff, g1, NG1(b)) + q, b.olist_cap);  // k_sg_lists
    return sg_outer_conn(b, a, q);
}

// ------------------------------------------------------------------ layer pairs
// Layer.cc:19-24: tracklet layer pairs are barrel (1,3), (2,4), (3,5)
__device__ __forceinline__ int tl_layer_outer(int si) { return si <= 2 ? si + 2 : -1; }

__device__ __forceinline__ int SR(const BatchDev& b, int k) { return AT(b.geo.slot_run, k, b.geo.n_slot_run); }

// objects of stage st in layer slot sl of event ev
__device__ __forceinline__ int64_t layer_count(const BatchDev& b, int st, int ev, int sl) {
    const int64_t base = (int64_t)ev * b.geo.n_mod;
    int64_t n = 0;
    for (int r = SR(b, sl); r < SR(b, sl + 1); ++r)
        n += OFF(b, st, base + SR(b, kNumSlots + 2 + 2 * r)) - OFF(b, st, base + SR(b, kNumSlots + 1 + 2 * r));
    return n;
}

// the q-th object of stage st in layer slot sl of event ev (q < layer_count)
__device__ __forceinline__ int layer_object(const BatchDev& b, int st, int ev, int sl, int64_t q) {
    const int64_t base = (int64_t)ev * b.geo.n_mod;
    for (int r = SR(b, sl); r < SR(b, sl + 1); ++r) {
        const int64_t o0 = OFF(b, st, base + SR(b, kNumSlots + 1 + 2 * r));
        const int64_t n = OFF(b, st, base + SR(b, kNumSlots + 2 + 2 * r)) - o0;
        if (q < n) return (int)(o0 + q);
        q -= n;
    }
#ifdef SDL_DEVICE_CHECKS
    (void)IX(-3, 0);
#endif
    return 0;
}

// Segment candidates by layer pairs (Event.cc:432-443, 793-821): candidate q
// of an inner MD runs over the MDs of the paired outer layers, in table order.
// Those are runs of consecutive MDs, the same for all MDs of an event's layer
// slot: one table row per event and slot (k_layer_runs) holds the runs' first
// MDs, then their cumulative counts.  A row has room for b.layer_width runs,
// kLayerRuns where those are enough (three endcap layers of four sides, the
// detId's two bits), else as many as the module table makes (detIds that
// differ in bits the decoding ignores).  kWide: rows of any width; the usual
// one is a constant of the kernel (48 registers and 111 to 120 us for the
// segment stage's candidates of 5 events with a variable width, 40 and 103 with
// the constant).
template <bool kWide>
__device__ __forceinline__ int layer_width(const BatchDev& b) { return kWide ? b.layer_width : kLayerRuns; }
template <bool kWide>
__device__ __forceinline__ const int* layer_row(const BatchDev& b, int a) {
    const int g1 = OG(b, kMD, a);
    const int ev = ev_of(b, g1);
    const int slot = MOD(b, g1 - ev * b.geo.n_mod).layer_slot;
    const int w = 2 * layer_width<kWide>(b);
    if (kWide) return &AT(b.layer_runs, (int64_t)(ev * kNumSlots + slot) * w, (int64_t)b.n_ev * kNumSlots * w);
    return &AT(b.layer_runs, (ev * kNumSlots + slot) * w, (int64_t)b.n_ev * kNumSlots * w);
}
__global__ void k_layer_runs(BatchDev b) {
    if (halted(b)) return;
    const int w = b.layer_width;
    for (int t = blockIdx.x * blockDim.x + threadIdx.x; t < b.n_ev * kNumSlots; t += gridDim.x * blockDim.x) {
        const int64_t base = (int64_t)(t / kNumSlots) * b.geo.n_mod;
        int* row = b.layer_runs + (int64_t)t * 2 * w;
        int n = 0, sum = 0;
        for (int k = 0; k < 3; ++k) {
            const int so = sg_layer_outer(t % kNumSlots, k);
            if (so < 0) break;
            for (int r = SR(b, so); r < SR(b, so + 1); ++r, ++n) {
                const int o0 = (int)OFF(b, kMD, base + SR(b, kNumSlots + 1 + 2 * r));
                row[n] = o0;
                sum += (int)OFF(b, kMD, base + SR(b, kNumSlots + 2 + 2 * r)) - o0;
                row[w + n] = sum;
            }
        }
        for (; n < w; ++n) {
            row[n] = 0;
            row[w + n] = sum;
        }
    }
}
template <bool kWide>
__device__ __forceinline__ int layer_md(const BatchDev& b, const int* row, int q) {
    const int w = layer_width<kWide>(b);
    int r = 0, before = 0;
    for (; r < w - 1; ++r) {
        const int end = row[w + r];
        if (q < end) break;
        before = end;
    }
    return row[r] + q - before;
}
// the endcap algorithm's first requirement for a layer pair: the outer MD's
// module is in the inner one's connection list (Segment.cc:613-633)
__device__ __forceinline__ bool sg_connected(const BatchDev& b, int a, int bmd) {
    const int g1 = OG(b, kMD, a);
    const int ev = ev_of(b, g1), m1 = g1 - ev * b.geo.n_mod, m2 = OG(b, kMD, bmd) - ev * b.geo.n_mod;
    for (int k = AT(b.geo.conn_off, m1, NM(b) + 1); k < AT(b.geo.conn_off, m1 + 1, NM(b) + 1); ++k)
        if (AT(b.geo.conn_idx, k, NC(b)) == m2) return true;
    return false;
}

// tracklet candidate q of inner segment s -> outer segment (Event.cc:635-663)
__device__ __forceinline__ int tl_outer(const BatchDev& b, int s, int64_t q) {
    const int n_mod = b.geo.n_mod;
    // module of the outer mini-doublet, from the packed segment record
    const int g2 = __float_as_int(AT(b.sgpack, (int64_t)s * PK_N + PK_G2, b.obj[kSG].cap * PK_N));
    const int ev = ev_of(b, g2), m2 = g2 - ev * n_mod;
    int pref;
    const int k = conn_entry(b, ev, m2, q, pref);
    const int g3 = ev * n_mod + AT(b.geo.conn_idx, k, NC(b));
    return (int)(OFF(b, kSG, g3) + (q - pref));
}

// tracklet candidate q of inner segment s by layer pairs (Event.cc:755-790):
// the q-th segment of the paired outer barrel layer
__device__ __forceinline__ int tl_outer_layer(const BatchDev& b, int s, int64_t q) {
    const int n_mod = b.geo.n_mod;
    const int g1 = OG(b, kSG, s);
    const int ev = ev_of(b, g1);
    return layer_object(b, kSG, ev, tl_layer_outer(MOD(b, g1 - ev * n_mod).layer_slot), q);
}

// The triplets and track candidates are equi-joins.  A triplet's segments
// share a mini-doublet: the join index lists the segments by their inner one
// (joff: offsets per mini-doublet, jidx: the segments), so that each join
// visits only matching objects.  A track candidate's tracklets share a segment
// (the same two mini-doublets): the tracklets by their inner segment (joft,
// jidt).  A connection list that repeats a module makes its segments several
// times; all of them go by the first of the same mini-doublets (sgkey).
__device__ __forceinline__ int join_key(const BatchDev& b, int st, int64_t o) {
    return st == kSG ? OI(b, kSG, o) : OI(b, kSG, OI(b, st, o));  // triplets: inner segment's inner MD
}
__device__ __forceinline__ int sg_key(const BatchDev& b, int s) {
    return b.geo.conn_dup ? AT(b.sgkey, s, b.obj[kSG].cap) : s;
}
// the second index (the triplets by their innermost MD)
__device__ __forceinline__ int64_t join2_n(const BatchDev& b, int md) {
    return AT(b.joff2, md + 1, b.obj[kMD].cap + 1) - AT(b.joff2, md, b.obj[kMD].cap + 1);
}
__device__ __forceinline__ int join2_obj(const BatchDev& b, int md, int64_t k) {
    return AT(b.jidx2, AT(b.joff2, md, b.obj[kMD].cap + 1) + k, b.obj[kTP].cap);
}
__device__ __forceinline__ int64_t join_n(const BatchDev& b, int md) {
    return AT(b.joff, md + 1, b.obj[kMD].cap + 1) - AT(b.joff, md, b.obj[kMD].cap + 1);
}
__device__ __forceinline__ int join_obj(const BatchDev& b, int md, int64_t k) {
    return AT(b.jidx, AT(b.joff, md, b.obj[kMD].cap + 1) + k, b.obj[kSG].cap);
}

// inner-object count of a stage (device), clamped to the inner capacity
__device__ __forceinline__ int64_t n_inner(const BatchDev& b, int st) {
    switch (st) {
        case kMD: return b.n_gm;
        case kSG: return n_objects(b, kMD);
        case kTL:
        case kTP: return n_objects(b, kSG);
        default:  // track candidates: tracklets, or triplets (createTrackCandidatesFromTriplets)
            return n_objects(b, (b.flags & kFlagTCFromTP) ? kTP : kTL);
    }
}

// the scan of stage st's candidate counts: offsets per inner object, and the
// bucket table (an inner object names the buckets that start in it)
template <int st>
struct ScanCand : ScanOp {
    static constexpr int kVals = 1, kSmall = 1, kBig = 4;
    __device__ static int64_t size(const BatchDev& b) { return n_inner(b, st); }
    __device__ static void put(const BatchDev& b, int64_t i, int64_t e, int64_t v) {
        AT(b.cand[st], i, b.cand_cap[st] + 1) = e;
        for (int64_t k = (e + (1ll << kBucketShift) - 1) >> kBucketShift; (k << kBucketShift) < e + v; ++k)
            if (k < b.bucket_cap) AT(b.bucket, k, b.bucket_cap) = (int)i;
    }
    // and the candidates per warp task of the enumeration: the stage's size
    // where there are enough candidates, less where that would leave warps
    // without a task (a 2.3k-hit event's 2,000 mini-doublet candidates were
    // nine tasks of 256, eight dependent rounds each: 67 us for the stage
    // against 31 us)
    __device__ static void put_total(const BatchDev& b, int64_t n, int64_t t) {
        AT(b.cand[st], n, b.cand_cap[st] + 1) = t;
        const int64_t warps = (int64_t)b.n_sm * (b.enum_grid[st] > 0 ? b.enum_grid[st] : kGridDefault) * (kEnumThreads / kWarp);
        int task = b.enum_task[st] > 0 ? b.enum_task[st] : kTaskDefault;
        while (task > kWarp && t < warps * task) task = max(kWarp, (task >> 1) / kWarp * kWarp);
        b.task_size[st] = task;
        const int64_t nb = (t + (1ll << kBucketShift) - 1) >> kBucketShift;
        if (n > 0 && nb < b.bucket_cap) AT(b.bucket, nb, b.bucket_cap) = (int)(n - 1);
    }
    __device__ static void store(const BatchDev& b, int64_t i, const int64_t* e, const int64_t* v) { put(b, i, e[0], v[0]); }
    __device__ static void total(const BatchDev& b, int64_t n, const int64_t* t) { put_total(b, n, t[0]); }
};

// A warp's accepted objects, collected in shared memory and appended to the
// stage's record list in batches of up to kRecBuf: one atomic on the list's
// count per batch instead of one per 32 candidates (atomics on one address
// serialise at its L2 slice), and coalesced record writes.  The ranks within
// the objects' modules are taken at the flush (atomics on distinct module
// counters, issued together).  Every lane of the warp calls rec_flush.
constexpr int kRecBuf = 64;
template <int kNF>
struct RecBuf {
    int (*e)[kRecBuf];  // this warp's [3 + kNF][kRecBuf] words: inner, outer, module, float values
    int n = 0;          // records held (warp-uniform)
};
template <int kNF>
__device__ __forceinline__ void rec_flush(const BatchDev& b, int st, RecBuf<kNF>& rb) {
    __syncwarp();
    const int lane = threadIdx.x & 31;
    const Recs& R = b.rec[st];
    const Objs& O = b.obj[st];
    unsigned long long p0 = 0;
    if (lane == 0 && rb.n) p0 = atomicAdd((unsigned long long*)(b.n_rec + st * kLine), (unsigned long long)rb.n);
    p0 = __shfl_sync(0xffffffffu, p0, 0);
    for (int k = lane; k < rb.n; k += kWarp) {
        const int64_t pos = (int64_t)p0 + k;
        if (pos < O.cap) {
            const int g = rb.e[2][k];
            AT(R.i, pos, O.cap) = rb.e[0][k];
            AT(R.j, pos, O.cap) = rb.e[1][k];
            AT(R.g, pos, O.cap) = g;
            AT(R.rank, pos, O.cap) = (int)atomicAdd((unsigned long long*)&AT(O.mod_cnt, g, NG1(b)), 1ull);
#pragma unroll
            for (int q = 0; q < kNF; ++q) AT(R.f, (int64_t)q * O.cap + pos, O.cap * kNF) = __int_as_float(rb.e[3 + q][k]);
        } else {
            atomicOr(b.status, 1u << st);
        }
    }
    __syncwarp();
    rb.n = 0;
}

// Mini-doublet candidates (the pairs of a module's lower and upper hits), in
// tasks of consecutive ones: those that the cuts do not certainly reject
// (md_first_cuts; 8 to 11 % of the candidates are mini-doublets) are gathered
// to full warps, which run the whole algorithm (float-float arctangents and
// square roots).  Bound by instruction issue: with the algorithm on every
// candidate in place, 13 of 32 lanes idle on average, it took 545 us for 64
// events, 382 now (128 dense events: the stage 2.08 -> 1.40 ms).  Where a
// task is a single round the candidates are judged in place: the gathering
// would only add its round (one 2.3k-hit event: 33.2 us for the stage with
// it, 31.2 without).
__global__ void __launch_bounds__(kEnumThreads) k_md_enum(BatchDev b) {
    __shared__ int rbuf[kEnumThreads / kWarp][3 + 4][kRecBuf];
    __shared__ int2 mbuf[kEnumThreads / kWarp][2 * kWarp];
    if (halted(b)) return;
    const int64_t* off = b.cand[kMD];
    const int64_t offlim = b.cand_cap[kMD] + 1;
    const int64_t nobj = b.n_gm;
    const int64_t total = AT(off, nobj, offlim);
    const int task = b.task_size[kMD];
    const int64_t ntask = (total + task - 1) / task;
    const int lane = threadIdx.x & 31;
    const unsigned lt = (1u << lane) - 1u;
    int2* mb = mbuf[threadIdx.x >> 5];
    int nm = 0;
    RecBuf<4> rb{rbuf[threadIdx.x >> 5]};
    const bool direct = task <= kWarp;
    bool open = true;  // candidates left
    int i0 = 0, i1 = 0;
    for (int64_t cb = 0, end = 0;;) {
        if (open && cb >= end) {
            unsigned long long t = 0;
            if (lane == 0) t = atomicAdd(b.task + kMD * kLine, 1ull);
            t = __shfl_sync(0xffffffffu, t, 0);
            open = (int64_t)t < ntask;
            if (open) {
                cb = (int64_t)t * task;
                end = min(cb + task, total);
                int ilo = 0;
                if (lane < 2) {
                    int lo, hi;
                    obj_bounds(b, nobj, total, cb, end - 1, lo, hi);
                    ilo = find_obj(b, off, offlim, lo, hi, lane == 0 ? cb : end - 1);
                }
                i0 = __shfl_sync(0xffffffffu, ilo, 0);
                i1 = __shfl_sync(0xffffffffu, ilo, 1);
            }
        }
        // the next 32 candidates: to the buffer, or kept for now
        int g = 0;
        int2 e = make_int2(0, 0);
        bool has = false;
        if (open) {
            const int64_t c = cb + lane;
            cb += kWarp;
            if (c < end) {
                g = (i0 == i1) ? i0 : find_obj(b, off, offlim, i0, i1, c);
                has = md_candidate(b, g, c - AT(off, g, offlim), e);
                if (has && !direct) {
                    const ModDev& lm = MOD(b, mod_of(b, g));
                    const MDCand d = md_cand(b, lm, e);
                    has = md_first_cuts(d.L, d.U, d.pixAsin, lm, d.sh);
                }
            }
        }
        if (!direct) {
            const unsigned m = __ballot_sync(0xffffffffu, has);
            if (has) mb[nm + __popc(m & lt)] = e;
            nm += __popc(m);
            __syncwarp();
            const int n = open && nm < kWarp ? 0 : min(nm, kWarp);
            has = lane < n;
            if (has) {
                e = mb[nm - n + lane];
                g = AT(b.hgm, e.x, H(b));
            }
            __syncwarp();
            nm -= n;
            if (open && n == 0) continue;
        }
        if (!__any_sync(0xffffffffu, has)) {
            if (open) continue;
            break;
        }
        // the whole algorithm
        MDVals v;
        v.dz = 0.f; v.shiftedDz = 0.f; v.dphi = 0.f; v.dphichange = 0.f;
        if (has) {
            const ModDev& lm = MOD(b, mod_of(b, g));
            const MDCand c = md_cand(b, lm, e);
            has = lm.subdet == kBarrel ? md_barrel(c.L, c.U, c.pixAsin, lm, c.sh, v) : md_endcap(c.L, c.U, c.pixAsin, lm, c.sh, v);
        }
        const unsigned m = __ballot_sync(0xffffffffu, has);
        if (rb.n + __popc(m) > kRecBuf) rec_flush<4>(b, kMD, rb);
        if (has) {
            const int k = rb.n + __popc(m & lt);
            rb.e[0][k] = e.x;
            rb.e[1][k] = e.y;
            rb.e[2][k] = g;
            rb.e[3][k] = __float_as_int(v.dz);
            rb.e[4][k] = __float_as_int(v.shiftedDz);
            rb.e[5][k] = __float_as_int(v.dphi);
            rb.e[6][k] = __float_as_int(v.dphichange);
        }
        rb.n += __popc(m);
    }
    rec_flush<4>(b, kMD, rb);
}

// One packed record per segment for the tracklet stage (the anchors of both
// mini-doublets, the segment's angles and the per-segment sub-expressions of
// Tracklet.cc that depend on one segment only).
// the packed record of the segment from mini-doublet im to mini-doublet om
// with the segment algorithm's six values f6 (dPhi, dPhiMin, dPhiMax,
// dPhiChange, dPhiMinChange, dPhiMaxChange)
__device__ __forceinline__ void sg_pack_record(const BatchDev& b, int im, int om, const float* f6, float* v) {
    const MDRec I = md_rec(b, im), O = md_rec(b, om);
    const float2 bend = __ldg(reinterpret_cast<const float2*>(&AT(b.mdbend, 2 * (int64_t)im, 2 * b.obj[kMD].cap)));
    const P3 lo = I.v.a, up = O.v.a;
    const ModDev& lam = MOD(b, I.anc_mod);
    const ModDev& uam = MOD(b, O.anc_mod);
    uint32_t fl = 0;
    fl |= lam.subdet == kBarrel ? F_LO_B : 0u;
    fl |= lam.subdet == kEndcap ? F_LO_E : 0u;
    fl |= lam.type == kPS ? F_LO_PS : 0u;
    fl |= uam.subdet == kBarrel ? F_UP_B : 0u;
    fl |= uam.subdet == kEndcap ? F_UP_E : 0u;
    fl |= uam.type == kPS ? F_UP_PS : 0u;
    fl |= uam.type == kTwoS ? F_UP_2S : 0u;
    v[PK_LX] = lo.x; v[PK_LY] = lo.y; v[PK_LZ] = lo.z; v[PK_LRT] = lo.rt;
    v[PK_LPHI] = lo.phi; v[PK_LR3] = lo.r3; v[PK_LA1] = I.a1; v[PK_LTD] = bend.x;
    v[PK_LA3] = bend.y;
    v[PK_LR3Z] = __fsqrt_rn(lo.z * lo.z + lo.rt * lo.rt);
    v[PK_UX] = up.x; v[PK_UY] = up.y; v[PK_UZ] = up.z; v[PK_URT] = up.rt; v[PK_UPHI] = up.phi; v[PK_UR3] = up.r3;
    v[PK_DPC] = f6[3]; v[PK_DPMIN] = f6[1]; v[PK_DPMAX] = f6[2];
    v[PK_DPMINC] = f6[4]; v[PK_DPMAXC] = f6[5];
    v[PK_RTSEG] = rt_of_diff(up, lo);
    v[PK_ALPHAUP] = dphi(up, sub(up, lo));
    v[PK_DPHILU] = dphi(lo, up);
    v[PK_EX] = uam.edge_x; v[PK_EY] = uam.edge_y;
    v[PK_FLAGS] = __uint_as_float(fl);
    v[PK_G2] = __int_as_float(OG(b, kMD, om));
    // the inner role's per-segment terms of phase A (the same float
    // operations as there)
    v[PK_S0] = (up.z - lo.z) / (up.rt - lo.rt);
    v[PK_S1] = (up.r3 - lo.r3) / (up.rt - lo.rt);
    const float q = v[PK_LR3Z] / lo.rt;
    if (q > 0x1p-60f && q < 0x1p60f) {
        const ffm::ff sq = ffm::sqrt_ff(ffm::ff{q, 0.f});
        v[PK_S2] = sq.hi;
        v[PK_S3] = sq.lo;
    } else {
        v[PK_S2] = v[PK_S3] = __int_as_float(0x7fc00000);  // NaN: muls takes its double path
    }
}

// what the tracklet and triplet stages read of segment s (mini-doublets im
// and om, f6 as kept): the packed record, the outer-role fields, the
// pre-filter's features; and its place among the segments that end in its
// outer module (eoff counts, erank) and that start at its inner mini-doublet
// (joff counts, jrank)
__device__ __forceinline__ void sg_pack_write(const BatchDev& b, int64_t s, int im, int om, const float* f6, float* v, float4* fd) {
    sg_pack_record(b, im, om, f6, v);
    const uint32_t fl = __float_as_uint(v[PK_FLAGS]);
    const int64_t C = b.obj[kSG].cap;
    AT(b.erank, s, C) = (int)atomicAdd((unsigned long long*)&AT(b.eoff, __float_as_int(v[PK_G2]), NG1(b)), 1ull);
    AT(b.jrank, s, C) = (int)atomicAdd((unsigned long long*)&AT(b.joff, im, b.obj[kMD].cap + 1), 1ull);
    const int fo[10] = {PK_LRT, PK_LZ, PK_LTD, PK_LA1, PK_UPHI, PK_FLAGS, -1, PK_LX, PK_LY, PK_UX};
#pragma unroll
    for (int k = 0; k < 10; ++k)
        if (k != 6) AT(b.sgouter, k * C + s, kSgOuter * C) = v[fo[k]];
    AT(b.sgouter, 6 * C + s, kSgOuter * C) = 0.1f / v[PK_LRT];  // the PV-offset term of an outer segment
    AT(b.sgouter, 10 * C + s, kSgOuter * C) = v[PK_UY];
    AT(b.sgouter, 11 * C + s, kSgOuter * C) = v[PK_ALPHAUP];
    AT(b.sgouter, 12 * C + s, kSgOuter * C) = v[PK_RTSEG];
    AT(b.sgouter, 13 * C + s, kSgOuter * C) = v[PK_URT] - v[PK_LRT];
    // the pre-filter's feature records (inner role, outer role)
    const float lz = v[PK_LZ], lrt = v[PK_LRT], uz = v[PK_UZ], urt = v[PK_URT];
    const float drIn = urt - lrt;
    const float slope = (uz - lz) / (fabsf(drIn) > 1e-3f ? drIn : copysignf(1e-3f, drIn));
    const float scode = ((fl & F_LO_E) ? 1.f : 0.f) + ((fl & F_LO_PS) ? 0.25f : 0.f);
    const float tcode = ((fl & F_UP_E) ? 0.5f : 0.f) + ((fl & F_UP_2S) ? 0.125f : 0.f);
    fd[0] = make_float4(v[PK_LX], v[PK_LY], lz, lrt);
    fd[1] = make_float4(v[PK_LPHI], v[PK_DPC], slope, scode);
    fd[2] = make_float4(v[PK_UX], v[PK_UY], uz, urt);
    fd[3] = make_float4(v[PK_UPHI], v[PK_ALPHAUP], tcode, 0.f);
}
// A warp's records of kQ 16-byte words, one a lane, written with neighbouring
// lanes on neighbouring words: through shared memory (32 * kQ words, the word
// of a record rotated by its lane so that neither side has bank conflicts).
// Every lane calls it; the first n lanes have a record.
template <int kQ>
__device__ __forceinline__ void store_records(float4* __restrict__ dst, float4* tmp, const float4* rec, int n) {
    const int lane = threadIdx.x & 31;
    __syncwarp();
#pragma unroll
    for (int k = 0; k < kQ; ++k) tmp[lane * kQ + (k ^ (lane & (kQ - 1)))] = rec[k];
    __syncwarp();
#pragma unroll
    for (int j = 0; j < kQ; ++j) {
        const int e = j * kWarp + lane, r = e / kQ;
        if (r < n) dst[e] = tmp[r * kQ + ((e & (kQ - 1)) ^ (r & (kQ - 1)))];
    }
}

// Bound by its stores' passes through L1: with each lane writing its own
// record it took 283 us for 64 events, 221 through shared memory.
__global__ void __launch_bounds__(256, 4) k_sg_pack(BatchDev b) {
    __shared__ float4 tmp[256 / kWarp][kWarp * (PK_N / 4)];
    if (halted(b)) return;
    const int64_t n = n_objects(b, kSG), C = b.obj[kSG].cap;
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int64_t stride = (int64_t)gridDim.x * blockDim.x;
    for (int64_t s0 = (int64_t)blockIdx.x * blockDim.x + w * kWarp; s0 < n; s0 += stride) {
        const int64_t s = s0 + lane;
        const int m = (int)min((int64_t)kWarp, n - s0);
        float v[PK_N];
        float4 fd[kFeatN / 4], rec[PK_N / 4];
        if (lane < m) {
            float f6[6];
#pragma unroll
            for (int k = 0; k < 6; ++k) f6[k] = OF(b, kSG, k, s);
            sg_pack_write(b, s, OI(b, kSG, s), OJ(b, kSG, s), f6, v, fd);
#pragma unroll
            for (int k = 0; k < PK_N / 4; ++k) rec[k] = make_float4(v[4 * k], v[4 * k + 1], v[4 * k + 2], v[4 * k + 3]);
        }
        store_records<PK_N / 4>(reinterpret_cast<float4*>(&AT(b.sgpack, s0 * PK_N, C * PK_N)), tmp[w], rec, m);
        if (lane < m) {
#pragma unroll
            for (int k = 0; k < kFeatN / 4; ++k) *reinterpret_cast<float4*>(&AT(b.sgfeat, 4 * (k * C + s), C * kFeatN)) = fd[k];
        }
    }
}

// createTrackCandidatesFromTriplets (Event.cc:874-982): candidate q of inner
// triplet p1 is a triplet p2 of a module connected to the module of p1's
// outermost MD (connection-list order, as the segment candidates); it passes
// when the trial segment from that MD to p2's innermost MD passes the segment
// algorithm and the tracklet (trial segment, p2's outer segment) passes the
// default tracklet algorithm.  The trial segment is not kept.
// (After layer-pair segments; after those of the module map see ScanTctp.)
__device__ __forceinline__ bool tctp_trial(const BatchDev& b, int p1, int64_t q, int& p2) {
    const int n_mod = b.geo.n_mod;
    const int mdA = OJ(b, kSG, OJ(b, kTP, p1));
    const int gA = OG(b, kMD, mdA);
    const int ev = ev_of(b, gA), mA = gA - ev * n_mod;
    int pref;
    const int k = conn_entry(b, ev, mA, q, pref);
    const int g3 = ev * n_mod + AT(b.geo.conn_idx, k, NC(b));
    p2 = (int)(OFF(b, kTP, g3) + (q - pref));
    const int mdB = OI(b, kSG, OI(b, kTP, p2));
    float f6[6];
    if (!sg_pair(b, mdA, mdB, true, f6)) return false;
    float v[PK_N];
    sg_pack_record(b, mdA, mdB, f6, v);
    const SGV S = sgv_from(v);
    const int so = OJ(b, kTP, p2);
    const SGV T = load_sgv(b.sgpack, so);
    float cut, muls;
    const int algo = tl_phaseA(S, T, cut, muls);
    if (algo == kAlgoNone || !tl_phaseB1_sgv(algo, S, T, cut)) return false;
    return tl_phaseB2_sgv<kB2All>(algo, S, T, muls, false);
}
__global__ void __launch_bounds__(kEnumThreads) k_tctp_trial(BatchDev b) {
    __shared__ int rbuf[kEnumThreads / kWarp][3][kRecBuf];
    if (halted(b)) return;
    const int64_t nobj = n_inner(b, kTC);
    if (nobj <= 0) return;
    const int64_t* off = b.cand[kTC];
    const int64_t offlim = b.cand_cap[kTC] + 1;
    const int64_t total = AT(off, nobj, offlim);
    const int task = b.task_size[kTC];
    const int64_t ntask = (total + task - 1) / task;
    const int lane = threadIdx.x & 31;
    RecBuf<0> rb{rbuf[threadIdx.x >> 5]};
    for (;;) {
        unsigned long long t = 0;
        if (lane == 0) t = atomicAdd(b.task + kTC * kLine, 1ull);
        t = __shfl_sync(0xffffffffu, t, 0);
        if ((int64_t)t >= ntask) break;
        const int64_t base = (int64_t)t * task;
        const int64_t end = min(base + task, total);
        int ilo = 0;
        if (lane < 2) {
            int lo, hi;
            obj_bounds(b, nobj, total, base, end - 1, lo, hi);
            ilo = find_obj(b, off, offlim, lo, hi, lane == 0 ? base : end - 1);
        }
        const int i0 = __shfl_sync(0xffffffffu, ilo, 0);
        const int i1 = __shfl_sync(0xffffffffu, ilo, 1);
        for (int64_t cb = base; cb < end; cb += kWarp) {
            const int64_t c = cb + lane;
            int p1 = 0, p2 = 0;
            bool pass = false;
            if (c < end) {
                p1 = (i0 == i1) ? i0 : find_obj(b, off, offlim, i0, i1, c);
                pass = tctp_trial(b, p1, c - AT(off, p1, offlim), p2);
            }
            const unsigned m = __ballot_sync(0xffffffffu, pass);
            if (!m) continue;
            if (rb.n + __popc(m) > kRecBuf) rec_flush<0>(b, kTC, rb);
            if (pass) {
                const int k = rb.n + __popc(m & ((1u << lane) - 1u));
                rb.e[0][k] = p1;
                rb.e[1][k] = p2;
                rb.e[2][k] = OG(b, kTP, p1);
            }
            rb.n += __popc(m);
        }
    }
    rec_flush<0>(b, kTC, rb);
}

// tracklet candidate q of inner segment s by navigation (Event.cc:694-751):
// over the segments leaving s's outer MD, the segments leaving their outer MD
// (both lists from the join index of segments by inner MD)
__device__ __forceinline__ int tl_outer_nav(const BatchDev& b, int s, int64_t q) {
    const int m = OJ(b, kSG, s);
    const int64_t nc = join_n(b, m);
    for (int64_t k = 0; k < nc; ++k) {
        const int mc = OJ(b, kSG, join_obj(b, m, k));
        const int64_t n = join_n(b, mc);
        if (q < n) return join_obj(b, mc, q);
        q -= n;
    }
#ifdef SDL_DEVICE_CHECKS
    IX(-3, 0);
#endif
    return 0;  // q is below the candidate count (ScanTlCand)
}

// the tracklet variant of a run: 0 module map, 1 layer pairs, 2 navigation
__device__ __forceinline__ int tl_variant(const BatchDev& b) {
    return (b.flags & kFlagTLLayers) ? 1 : ((b.flags & kFlagTLNav) ? 2 : 0);
}
__device__ __forceinline__ int tl_outer_of(const BatchDev& b, int var, int s, int64_t q) {
    return var == 1 ? tl_outer_layer(b, s, q) : (var == 2 ? tl_outer_nav(b, s, q) : tl_outer(b, s, q));
}

// Phases A and B1 of a candidate (inner segment s, outer segment t) from the
// single-precision decisions, with tl_phaseA where the first cannot decide:
// returns the algorithm (kAlgoNone: rejected by phase A or B1) and sets b1
// when phase B1 passed already (0: phase B1 is left to k_tl_b1); exact tells
// whether an exact evaluation was needed.  txy: the outer segment's anchors
// (load_sgo_xy).  The exact cut values are computed again in phase B1.
template <bool kEarly>
__device__ __forceinline__ int tl_ab1_decide(const TLRow& R, const TLOut& T, float4 txy, const float* __restrict__ pack, int s,
                                             int t, int& b1, bool& exact) {
    float cut;
    int algo = tl_phaseA_quick<kEarly>(R, T, cut);
    exact = algo == kAlgoUnsure;
    if (exact) algo = tl_phaseA_entry(pack, s, t, cut);
    b1 = 0;
    if (algo == kAlgoNone) return algo;
    const int q = tl_phaseB1_quick(algo, R, txy, cut);
    if (q == 0) return kAlgoNone;
    b1 = q > 0;
    exact = exact || q < 0;
    return algo;
}

// A warp's phase-A survivors, collected in shared memory and appended to
// the survivor list in batches of up to kPassBuf: one atomic on the list's
// count per batch instead of one per 32 candidates (atomics on one address
// serialise at its L2 slice, a few per nanosecond at most).  Positions past
// the list's capacity are not written and flag the overflow (the count keeps
// growing, so it holds the capacity needed).  Every lane of the warp calls
// passbuf_add and passbuf_flush.
constexpr int kPassBuf = 128;
constexpr int kPbBuf = 64;  // the phase-B2 (and segment first-pass) list's per-warp buffers
struct PassBuf {
    int4* e;    // this warp's kPassBuf entries in shared memory
    int n = 0;  // entries held (warp-uniform)
};
__device__ __forceinline__ void passbuf_flush(const BatchDev& b, PassBuf& pb) {
    __syncwarp();
    const int lane = threadIdx.x & 31;
    unsigned long long p0 = 0;
    if (lane == 0 && pb.n) p0 = atomicAdd(b.n_kept, (unsigned long long)pb.n);
    p0 = __shfl_sync(0xffffffffu, p0, 0);
    for (int i = lane; i < pb.n; i += kWarp) {
        const int64_t pos = (int64_t)p0 + i;
        if (pos < b.kept_cap) AT(b.passa, pos, b.kept_cap) = pb.e[i];
        else atomicOr(b.status, kStatusOverflowKept);
    }
    __syncwarp();
    pb.n = 0;
}
__device__ __forceinline__ void passbuf_put(const BatchDev& b, PassBuf& pb, bool pass, int4 e) {
    const int lane = threadIdx.x & 31;
    const unsigned m = __ballot_sync(0xffffffffu, pass);
    if (!m) return;
    const int c = __popc(m);
    if (pb.n + c > kPassBuf) passbuf_flush(b, pb);
    if (pass) pb.e[pb.n + __popc(m & ((1u << lane) - 1u))] = e;
    pb.n += c;
}
__device__ __forceinline__ void passbuf_add(const BatchDev& b, PassBuf& pb, int algo, int s, int tt, int b1) {
    passbuf_put(b, pb, algo != kAlgoNone, make_int4(s, tt, algo, b1));
}

// Tracklet candidates (Event.cc:611-693 with Tracklet.cc:144-2665) in three
// kernels: the enumeration (k_tl_enum_a here: tasks of consecutive
// candidates from a shared counter; k_tl_enum_tiles below for the module
// map) runs phase A (the float cuts) and, for its survivors, the
// single-precision decision of phase B1 on each candidate and lists the
// survivors, marking those through phase B1 already; k_tl_b1 and k_tl_b2 run
// the two parts of phase B on compacted lists and append the tracklets.  The
// survivor list shares the pre-filter's capacity and overflow handling (its
// count is n_kept).  A layer pair's candidates mostly fail the first window or
// the phi cut, so these are judged ahead of the row (tl_layer_out; one PU 200
// event, module-map segments: 3,425 us with the row of every candidate, 2,719
// so).
__global__ void __launch_bounds__(kEnumThreads) k_tl_enum_a(BatchDev b) {
    __shared__ int4 pbuf[kEnumThreads / kWarp][kPassBuf];
    if (halted(b)) return;
    const int64_t nobj = n_inner(b, kTL);
    if (nobj <= 0) return;
    const int64_t* off = b.cand[kTL];
    const int64_t offlim = b.cand_cap[kTL] + 1;
    const int64_t total = AT(off, nobj, offlim);
    const int task = b.task_size[kTL];
    const int64_t ntask = (total + task - 1) / task;
    const int lane = threadIdx.x & 31;
    const int lay = tl_variant(b);
    PassBuf pb{pbuf[threadIdx.x >> 5]};
    for (;;) {
        unsigned long long t = 0;
        if (lane == 0) t = atomicAdd(b.task + kTL * kLine, 1ull);
        t = __shfl_sync(0xffffffffu, t, 0);
        if ((int64_t)t >= ntask) break;
        const int64_t base = (int64_t)t * task;
        const int64_t end = min(base + task, total);
        int ilo = 0;
        if (lane < 2) {
            int lo, hi;
            obj_bounds(b, nobj, total, base, end - 1, lo, hi);
            ilo = find_obj(b, off, offlim, lo, hi, lane == 0 ? base : end - 1);
        }
        const int i0 = __shfl_sync(0xffffffffu, ilo, 0);
        const int i1 = __shfl_sync(0xffffffffu, ilo, 1);
        for (int64_t cb = base; cb < end; cb += kWarp) {
            const int64_t c = cb + lane;
            int algo = kAlgoNone, s = 0, tt = 0, b1 = 0;
            if (c < end) {
                s = (i0 == i1) ? i0 : find_obj(b, off, offlim, i0, i1, c);
                tt = tl_outer_of(b, lay, s, c - AT(off, s, offlim));
                (void)IX(s, b.obj[kSG].cap);
                (void)IX(tt, b.obj[kSG].cap);
                const int64_t C = b.obj[kSG].cap;
                const SGOuter T = load_sgo(b.sgouter, C, tt);
                bool exact;
                if (lay != 1 || !tl_layer_out(b.sgpack, s, T))
                    algo = tl_ab1_decide<true>(tl_row(load_sgv(b.sgpack, s)), tl_out(T), load_sgo_xy(b.sgouter, C, tt), b.sgpack, s, tt,
                                               b1, exact);
            }
            passbuf_add(b, pb, algo, s, tt, b1);
        }
    }
    passbuf_flush(b, pb);
}

// Module-map tracklet candidates in module-pair tiles.  The outer segments of
// an inner segment are those of the modules connected to the module of its
// outer mini-doublet (Event.cc:611-693), so all inner segments ending in one
// module g share one list of outer segments, and g's candidates are the
// product (segments ending in g) x (segments of g's connected modules, in
// connection-list order).  A warp task is a tile of that product: up to
// kTileA inner segments x 32 outer segments.  Each lane decodes and loads its
// outer segment once per tile, and the inner segments' records are
// warp-uniform loads.  The candidates, and so the survivor list as a set, are
// those k_tl_enum_a enumerates.
// Inner segments per module-pair tile: 32, or 16 for small batches, which have
// few tiles (enumeration of 128 dense events: 10.4 ms at 32, 10.6 at 24, 11.1 at
// 16; of one PU 200 event: 80 us at 32, 75 at 24, 72 at 16).
constexpr int kTileA = 32;
__device__ __forceinline__ int tile_shift(const BatchDev& b) { return b.hits_about <= kSmallBatch ? 4 : 5; }

__device__ __forceinline__ int64_t tile_count(const BatchDev& b, int64_t na, int64_t nb) {
    const int sh = tile_shift(b);
    return (na > 0 && nb > 0) ? ((na + (1 << sh) - 1) >> sh) * ((nb + kWarp - 1) / kWarp) : 0;
}

// the segments by their inner mini-doublet (joff scanned) and, for the
// module-map tracklets, by the global module of their outer one (eoff
// scanned) with the reference's candidate counters (Event.cc:635-663)
__global__ void k_sg_index(BatchDev b) {
    if (halted(b)) return;
    const int n_mod = b.geo.n_mod;
    const int64_t n = n_objects(b, kSG), C = b.obj[kSG].cap;
    const bool map = tl_variant(b) == 0;
    for (int64_t s = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; s - threadIdx.x < n; s += (int64_t)gridDim.x * blockDim.x) {
        const bool in = s < n;
        int64_t c = 0;
        int ev = 0, slot = 0;
        if (in) AT(b.jidx, AT(b.joff, OI(b, kSG, s), b.obj[kMD].cap + 1) + AT(b.jrank, s, C), C) = (int)s;
        if (!map) continue;
        if (in) {
            const int g2 = OG(b, kMD, OJ(b, kSG, s));
            AT(b.eidx, AT(b.eoff, g2, NG1(b)) + AT(b.erank, s, C), C) = (int)s;
            c = AT(b.conn_sum, g2, b.n_gm);
            const int g1 = OG(b, kSG, s);
            ev = ev_of(b, g1);
            slot = MOD(b, g1 - ev * n_mod).layer_slot;
        }
        const bool act = in && c != 0;
        warp_add(act ? counter_at(b, ev, kTL, 0, slot) : b.counters, (uint32_t)c, act);
    }
}
// the first segment of every segment's two mini-doublets (geometries whose
// connection lists repeat a module)
__global__ void k_sg_keys(BatchDev b) {
    if (halted(b)) return;
    const int64_t n = n_objects(b, kSG);
    for (int64_t s = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; s < n; s += (int64_t)gridDim.x * blockDim.x) {
        const int md = OI(b, kSG, s), om = OJ(b, kSG, s);
        int key = (int)s;
        const int64_t m = join_n(b, md);
        for (int64_t k = 0; k < m; ++k) {
            const int t = join_obj(b, md, k);
            if (t < key && OJ(b, kSG, t) == om) key = t;
        }
        AT(b.sgkey, s, b.obj[kSG].cap) = key;
    }
}

// the global module holding tile t: the largest g < n_gm with toff[g] <= t
// (toff[0] = 0 <= t), by a 32-way search; every lane calls it with the same t
__device__ __forceinline__ int tile_module(const BatchDev& b, int64_t t) {
    const int lane = threadIdx.x & 31;
    int lo = 0, hi = b.n_gm - 1;  // toff[lo] <= t, and the answer is in [lo, hi]
    while (hi - lo >= kWarp) {
        const int64_t span = (int64_t)(hi - lo) + 1;
        const int p = lo + (int)((span * lane) >> 5);  // probes lo = p_0 < p_1 < ... < p_31 <= hi
        const unsigned m = __ballot_sync(0xffffffffu, AT(b.toff, p, NG1(b)) <= t);
        const int j = 31 - __clz(m);  // bit 0 is set, and the set bits are a prefix
        if (j < 31) hi = lo + (int)((span * (j + 1)) >> 5) - 1;
        lo += (int)((span * j) >> 5);
    }
    const int p = lo + lane;
    const unsigned m = __ballot_sync(0xffffffffu, p <= hi && AT(b.toff, p, NG1(b)) <= t);
    return lo + 31 - __clz(m);
}

// The outer object of lane q - q0 of a tile whose outer block starts at entry
// q0 of global module g's outer list (the objects of g's connected modules in
// connection-list order; module m of event ev, connection entries [k0, k1)),
// from the entries' prefix sums and first objects (k_conn_sum).  While g has
// at most 32 connections, lane j loads entry k0 + j and each lane finds its
// entry among them (the last one whose prefix sum is <= its q); otherwise
// each lane searches.  Every lane of the warp calls it; lanes with has false
// get an unspecified value.
__device__ __forceinline__ int tile_outer(const BatchDev& b, int ev, int m, int k0, int k1, int64_t q0, bool has) {
    const int lane = threadIdx.x & 31;
    const int64_t q = q0 + lane;
    const int64_t pbase = (int64_t)ev * b.geo.n_conn;
    if (k1 - k0 <= kWarp) {
        int pj = 0x7fffffff, fj = 0;
        if (lane < k1 - k0) {
            pj = AT(b.conn_pref, pbase + k0 + lane, NCP(b));
            fj = AT(b.conn_first, pbase + k0 + lane, NCP(b));
        }
        // entry 0 has prefix sum 0 <= q0
        int j = 31 - __clz(__ballot_sync(0xffffffffu, pj <= q0));
        for (int jj = j + 1; jj < k1 - k0; ++jj) {
            const int pjj = __shfl_sync(0xffffffffu, pj, jj);
            if (pjj > q0 + (kWarp - 1)) break;
            if (pjj <= q) j = jj;
        }
        const int pref = __shfl_sync(0xffffffffu, pj, j);
        const int first = __shfl_sync(0xffffffffu, fj, j);
        return first + (int)(q - pref);
    }
    if (!has) return 0;
    int pref;
    const int k = conn_entry(b, ev, m, q, pref);
    return (int)(AT(b.conn_first, pbase + k, NCP(b)) + (q - pref));
}

// Each warp takes tiles from a shared counter (the next index is fetched
// while the current tile runs).  Per tile, the loads come in a few dependent
// rounds: the module (tile map), its offsets and connection-list range, the
// inner segments' indices with the connection entries' prefix sums and first
// segments (one entry per lane while the module has at most 32 connections),
// then the inner segments' records, a lane each, which it turns into the rows
// of the single-precision decisions (in shared memory, read there as
// warp-uniform values), with the lanes' outer-segment fields.  Bound by
// instruction issue: with the decisions on divisions, atan2 polynomials and
// asinf over the plain records the 128 dense events took 14.9 ms, 9.5 now.
// CTAs per SM it is compiled for (register budget): 9.5 ms at 4, 10.2 at 3,
// 10.3 at 5.
#ifndef SDLG_ENUM_MIN_BLOCKS
#define SDLG_ENUM_MIN_BLOCKS 4
#endif
__global__ void __launch_bounds__(kEnumThreads, SDLG_ENUM_MIN_BLOCKS) k_tl_enum_tiles(BatchDev b) {
    __shared__ TLRow srow[kEnumThreads / kWarp][kTileA];
    __shared__ int sidx[kEnumThreads / kWarp][kTileA];
    __shared__ int4 pbuf[kEnumThreads / kWarp][kPassBuf];
    __shared__ float4 sxy[kEnumThreads / kWarp][kWarp];  // the lanes' outer anchors (phase B1)
    if (halted(b) || b.n_gm <= 0) return;
    const int64_t ntile = AT(b.toff, b.n_gm, NG1(b));
    const bool mapped = ntile <= b.tile_cap;
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int n_mod = b.geo.n_mod;
    const int64_t sgcap = b.obj[kSG].cap;
    PassBuf pb{pbuf[w]};
    unsigned long long next = 0;
    if (lane == 0) next = atomicAdd(b.task + kTL * kLine, 1ull);
    for (;;) {
        const int64_t t = (int64_t)__shfl_sync(0xffffffffu, next, 0);
        if (t >= ntile) break;
        if (lane == 0) next = atomicAdd(b.task + kTL * kLine, 1ull);
        const int g = mapped ? AT(b.tile_gm, t, b.tile_cap) : tile_module(b, t);
        const int ev = ev_of(b, g), m2 = g - ev * n_mod;
        const int64_t a0 = AT(b.eoff, g, NG1(b));
        const int64_t na = AT(b.eoff, g + 1, NG1(b)) - a0;
        const int64_t nb = AT(b.conn_sum, g, b.n_gm);
        const int k0 = AT(b.geo.conn_off, m2, NM(b) + 1), k1 = AT(b.geo.conn_off, m2 + 1, NM(b) + 1);
        const int64_t nbb = (nb + kWarp - 1) / kWarp;
        const int64_t local = t - AT(b.toff, g, NG1(b));
        const int64_t ab = local / nbb, bb = local - ab * nbb;
        const int sh = tile_shift(b);
        const int64_t abase = ab << sh;
        const int nat = (int)min((int64_t)1 << sh, na - abase);
        // this lane's outer segment: entry q of g's outer list
        const int64_t q0 = bb * kWarp;
        const bool has = q0 + lane < nb;
        __syncwarp();  // the previous tile's rows have been read
        if (lane < nat) {
            const int sr = AT(b.eidx, a0 + abase + lane, sgcap);
            (void)IX(sr, sgcap);
            sidx[w][lane] = sr;
            srow[w][lane] = tl_row(load_sgv(b.sgpack, sr));
        }
        const int tt = tile_outer(b, ev, m2, k0, k1, q0, has);
        TLOut T{};
        if (has) {
            (void)IX(tt, sgcap);
            T = tl_out(load_sgo(b.sgouter, sgcap, tt));
            sxy[w][lane] = load_sgo_xy(b.sgouter, sgcap, tt);
        }
        __syncwarp();
        for (int r = 0; r < nat; ++r) {
            const int sr = sidx[w][r];
            int b1;
            bool exact;  // (a lane without an outer segment has no algorithm)
            const int algo = tl_ab1_decide<false>(srow[w][r], T, sxy[w][lane], b.sgpack, sr, tt, b1, exact);
            passbuf_add(b, pb, algo, sr, tt, b1);
        }
    }
    passbuf_flush(b, pb);
}

// CTAs per SM the segment second pass is compiled for (register budget: 64
// registers and no spill at 4, 40 and about 100 bytes of spills at 6).  With
// the pass split by algorithm, 4 measured fastest on the 128-event PU 150-300
// batch: segment stage 7.21 ms against 7.23 at 5 and 7.57 at 6
#ifndef SDLG_SGB_MIN_BLOCKS
#define SDLG_SGB_MIN_BLOCKS 4
#endif
constexpr int kSgbMinBlocks = SDLG_SGB_MIN_BLOCKS;

// Segment candidates in two passes (Event.cc:445-522 or 793-821 with
// Segment.cc:337-859): k_sg_enum_a takes tasks of consecutive candidates
// like k_tl_enum_a, gathers those the algorithm's first cuts do not certainly
// reject (40 % of them) to full warps, and lists those that the later cuts do
// not certainly reject either (7.7 %; 7.6 % are segments); k_sg_b runs the
// whole algorithm on the list and appends the segments.  Both are bound by
// instruction issue.  64 events: with the exact first cuts on 64-byte records
// the first pass took 547 us and the second, on the 40 %, 870; with
// sg_first_cuts alone 412 and 870; with the later cuts 437 and 257.
// A warp's segment first-pass survivors appended to the spare list pb:
// candidates with a barrel outer MD at its front (count n_pb[0]), the others
// at its back (n_pb[1]), so that the second pass runs each algorithm in its
// own kernel.  n_kept counts both and reserves their room: a batch that would
// take the two parts past kept_cap is not written and flags the overflow (the
// count keeps growing, so it holds the capacity needed).
__device__ __forceinline__ void sg_list_flush(const BatchDev& b, int4* buf, int& n, bool front) {
    __syncwarp();
    const int lane = threadIdx.x & 31;
    unsigned long long p0 = 0;
    int ok = 1;
    if (lane == 0 && n) {
        const unsigned long long tot = atomicAdd(b.n_kept, (unsigned long long)n);
        ok = tot + (unsigned long long)n <= (unsigned long long)b.kept_cap;
        if (ok) p0 = atomicAdd(b.n_pb + (front ? 0 : 1), (unsigned long long)n);
        else atomicOr(b.status, kStatusOverflowKept);
    }
    p0 = __shfl_sync(0xffffffffu, p0, 0);
    ok = __shfl_sync(0xffffffffu, ok, 0);
    if (ok)
        for (int k = lane; k < n; k += kWarp) {
            const int64_t q = (int64_t)p0 + k;
            AT(b.pb, front ? q : b.kept_cap - 1 - q, b.kept_cap) = buf[k];
        }
    __syncwarp();
    n = 0;
}

// kVar: 0 the module map, 1 the layer pairs, 2 the layer pairs with rows of any width
template <int kVar>
__global__ void __launch_bounds__(kEnumThreads) k_sg_enum_a(BatchDev b) {
    __shared__ int4 sbuf[kEnumThreads / kWarp][2][kPbBuf];
    __shared__ int2 mbuf[kEnumThreads / kWarp][2 * kWarp];
    if (halted(b)) return;
    const int64_t nobj = n_inner(b, kSG);
    if (nobj <= 0) return;
    const int64_t* off = b.cand[kSG];
    const int64_t offlim = b.cand_cap[kSG] + 1;
    const int64_t total = AT(off, nobj, offlim);
    const int task = b.task_size[kSG];
    const int64_t ntask = (total + task - 1) / task;
    const int lane = threadIdx.x & 31;
    int4* fb = sbuf[threadIdx.x >> 5][0];
    int4* bb = sbuf[threadIdx.x >> 5][1];
    int2* mb = mbuf[threadIdx.x >> 5];
    int nf = 0, nb = 0, nm = 0;
    const unsigned lt = (1u << lane) - 1u;
    // the later cuts on the last n of mb's pairs, one a lane
    auto later = [&](int n) {
        __syncwarp();
        int2 e = make_int2(0, 0);
        bool pass = false, ob = false;
        if (lane < n) {
            e = mb[nm - n + lane];
            const MDLite O = md_lite(b, e.y);
            ob = (O.fl & kMdBarrel) != 0;
            pass = sg_later_cuts(md_lite(b, e.x), O);
        }
        __syncwarp();
        nm -= n;
        const unsigned mf = __ballot_sync(0xffffffffu, pass && ob), mo = __ballot_sync(0xffffffffu, pass && !ob);
        if (nf + __popc(mf) > kPbBuf) sg_list_flush(b, fb, nf, true);
        if (nb + __popc(mo) > kPbBuf) sg_list_flush(b, bb, nb, false);
        if (pass && ob) fb[nf + __popc(mf & lt)] = make_int4(e.x, e.y, 1, 0);
        if (pass && !ob) bb[nb + __popc(mo & lt)] = make_int4(e.x, e.y, 2, 0);
        nf += __popc(mf);
        nb += __popc(mo);
    };
    for (;;) {
        unsigned long long t = 0;
        if (lane == 0) t = atomicAdd(b.task + kSG * kLine, 1ull);
        t = __shfl_sync(0xffffffffu, t, 0);
        if ((int64_t)t >= ntask) break;
        const int64_t base = (int64_t)t * task;
        const int64_t end = min(base + task, total);
        int ilo = 0;
        if (lane < 2) {
            int lo, hi;
            obj_bounds(b, nobj, total, base, end - 1, lo, hi);
            ilo = find_obj(b, off, offlim, lo, hi, lane == 0 ? base : end - 1);
        }
        const int i0 = __shfl_sync(0xffffffffu, ilo, 0);
        const int i1 = __shfl_sync(0xffffffffu, ilo, 1);
        for (int64_t cb = base; cb < end; cb += kWarp) {
            const int64_t c = cb + lane;
            int a = 0, bmd = 0;
            bool pass = false;
            if (c < end) {
                a = (i0 == i1) ? i0 : find_obj(b, off, offlim, i0, i1, c);
                const int64_t q = c - AT(off, a, offlim);
                bmd = kVar ? layer_md<kVar == 2>(b, layer_row<kVar == 2>(b, a), (int)q) : sg_outer_md(b, a, q);
                (void)IX(bmd, b.obj[kMD].cap);
                pass = sg_first_cuts(md_lite(b, a), md_lite(b, bmd));
            }
            const unsigned m = __ballot_sync(0xffffffffu, pass);
            if (pass) mb[nm + __popc(m & lt)] = make_int2(a, bmd);
            nm += __popc(m);
            if (nm >= kWarp) later(kWarp);
        }
    }
    later(nm);
    sg_list_flush(b, fb, nf, true);
    sg_list_flush(b, bb, nb, false);
}

template <int kOuter>
__device__ __forceinline__ void sg_b(const BatchDev& b, int (*rbuf)[3 + 6][kRecBuf]) {
    // kOuter 1: the barrel part of the first pass's list (front), 2: the endcap part (back)
    const int64_t nfront = min((int64_t)b.n_pb[0], b.kept_cap);
    const int64_t n = kOuter == 1 ? nfront : min((int64_t)b.n_pb[1], b.kept_cap - nfront);
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int64_t nwarp = (int64_t)gridDim.x * (kEnumThreads / 32);
    RecBuf<6> rb{rbuf[w]};
    for (int64_t base = ((int64_t)blockIdx.x * (kEnumThreads / 32) + w) * kWarp; base < n; base += nwarp * kWarp) {
        const int64_t i = base + lane;
        bool pass = false;
        int a = 0, bmd = 0;
        float fv[6];
        if (i < n) {
            const int4 e = AT(b.pb, kOuter == 1 ? i : b.kept_cap - 1 - i, b.kept_cap);
            a = e.x;
            bmd = e.y;
            const bool conn = kOuter == 1 || !(b.flags & kFlagSGLayers) || sg_connected(b, a, bmd);
            pass = sg_pair_rec<kOuter>(md_rec(b, a).v, md_rec(b, bmd), conn, fv);
        }
        const unsigned m = __ballot_sync(0xffffffffu, pass);
        if (!m) continue;
        if (rb.n + __popc(m) > kRecBuf) rec_flush<6>(b, kSG, rb);
        if (pass) {
            const int k = rb.n + __popc(m & ((1u << lane) - 1u));
            rb.e[0][k] = a;
            rb.e[1][k] = bmd;
            rb.e[2][k] = OG(b, kMD, a);
#pragma unroll
            for (int q = 0; q < 6; ++q) rb.e[3 + q][k] = __float_as_int(fv[q]);
        }
        rb.n += __popc(m);
    }
    rec_flush<6>(b, kSG, rb);
}
// kOuter 1: the barrel part of the list, 2: the endcap part, 0: both, by
// blockIdx.y (launch_pair)
template <int kOuter>
__global__ void __launch_bounds__(kEnumThreads, kSgbMinBlocks) k_sg_b(BatchDev b) {
    __shared__ int rbuf[kEnumThreads / kWarp][3 + 6][kRecBuf];
    if (halted(b)) return;
    if (kOuter == 1 || (kOuter == 0 && blockIdx.y == 0)) sg_b<1>(b, rbuf);
    else sg_b<2>(b, rbuf);
}

// Learned pre-filter of the tracklet candidates (no counterpart in the
// reference).  It scores the enumeration's survivor list (n_kept entries:
// through phase A, and through phase B1 or undecided there) in tiles of 128
// entries on the tensor cores; the entries whose logit reaches the threshold
// go to the kept list (n_kept2 entries), which k_tl_b1 and k_tl_b2 judge.  A
// candidate that fails phase A or B1 gives no tracklet, so the tracklets are
// those of the plain chain among the candidates the network keeps; the
// network only sees phase-A survivors, the candidates it was trained on.
// Each CTA takes every gridDim.x-th tile; while the tensor cores run a
// tile's first layer, the CTA loads the next tile's entries and features.
// Control flow around the tile is uniform over the CTA.

// one tile's kept entries: written once the atomic that reserved their
// positions (issued by lane `leader`, raw value there) has returned
struct PfPending {
    unsigned m = 0u;
    unsigned long long raw = 0ull;
    int leader = 0;
    int4 e = make_int4(0, 0, 0, 0);  // (inner, outer, algorithm, 0)
};

__device__ __forceinline__ void pf_flush(const BatchDev& b, const PfPending& p) {
    if (p.m == 0u) return;
    const unsigned long long p0 = __shfl_sync(0xffffffffu, p.raw, p.leader);
    const int lane = threadIdx.x & 31;
    if (!((p.m >> lane) & 1u)) return;
    const int64_t pos = (int64_t)p0 + __popc(p.m & ((1u << lane) - 1u));  // below the list length <= kept_cap
    AT(b.kept, pos, b.kept_cap) = p.e;
}

// CTAs per SM: shared memory (33.4 KB per CTA) leaves room for 6; 6 and 8
// CTAs measured the same before the second layer took b2 into its MMA
constexpr int kPfCtasPerSm = 6;
__global__ void __launch_bounds__(kMlpTile, kPfCtasPerSm) k_tl_prefilter(BatchDev b) {
    __shared__ MlpSmem sm;
    if (halted(b)) return;
    const int64_t n = min((int64_t)*b.n_kept, b.kept_cap);
    const int64_t ntile = (n + kMlpTile - 1) / kMlpTile;
    if (blockIdx.x == 0 && threadIdx.x == 0) atomicAdd(&b.mlp_stats->candidates, *b.n_cand_tl);
    if ((int64_t)blockIdx.x >= ntile) return;
    const int lane = threadIdx.x & 31;
    mlp_setup(sm, b.mlp_pack);
    const float thr = reinterpret_cast<const float*>(sm.w + kPackB3)[1];
    MlpThread st;
    if (b.flags & kFlagTestMlpGiveUp) st.polls = 0;
    unsigned n_scored = 0, n_kept = 0;
    // Three tiles in the pipeline of each thread: the list entry of tile
    // t + 2G (G = gridDim.x) is loaded, the two segment records of tile t + G
    // are loaded with the entry loaded one iteration earlier, and the features
    // of tile t are computed from the records loaded one iteration earlier,
    // so that every load has a tile's MMAs and epilogue to complete in.
    const int64_t G = gridDim.x;
    auto entry = [&](int64_t tt, int4& e) -> bool {
        const int64_t i = tt * kMlpTile + threadIdx.x;
        const bool valid = tt < ntile && i < n;
        if (valid) e = AT(b.passa, i, b.kept_cap);
        return valid;
    };
    int64_t t = blockIdx.x;
    PfPending cur, pend;
    int4 e1 = make_int4(0, 0, 0, 0), e2 = make_int4(0, 0, 0, 0);
    bool valid = entry(t, cur.e);
    bool v1 = entry(t + G, e1);
    FeatS rs{};
    FeatT rt{};
    if (valid) {
        rs = feat_s(b.sgfeat, b.obj[kSG].cap, cur.e.x);
        rt = feat_t(b.sgfeat, b.obj[kSG].cap, cur.e.y);
    }
    while (t < ntile) {
        float f[kMlpIn];
        if (valid) {
            tl_features(rs, rt, f);
        } else {
#pragma unroll
            for (int k = 0; k < kMlpIn; ++k) f[k] = 0.f;
        }
        mlp_tile_begin(sm, f, st);
        const bool v2 = entry(t + 2 * G, e2);
        if (v1) {
            rs = feat_s(b.sgfeat, b.obj[kSG].cap, e1.x);
            rt = feat_t(b.sgfeat, b.obj[kSG].cap, e1.y);
        }
        pf_flush(b, pend);
        const float z = mlp_tile_end(sm, st);
        const bool keep = valid && z >= thr;
        n_scored += valid;
        n_kept += keep;
        cur.m = __ballot_sync(0xffffffffu, keep);
        if (cur.m) {
            cur.leader = __ffs(cur.m) - 1;
            if (lane == cur.leader) cur.raw = atomicAdd(b.n_kept2, (unsigned long long)__popc(cur.m));
        }
        pend = cur;
        cur.e = e1;
        valid = v1;
        e1 = e2;
        v1 = v2;
        t += G;
    }
    pf_flush(b, pend);
    n_scored = __reduce_add_sync(0xffffffffu, n_scored);
    n_kept = __reduce_add_sync(0xffffffffu, n_kept);
    if (lane == 0) {
        atomicAdd(&b.mlp_stats->scored, (unsigned long long)n_scored);
        atomicAdd(&b.mlp_stats->kept, (unsigned long long)n_kept);
    }
    if (st.abort && threadIdx.x == 0) {
        atomicAdd(&b.mlp_stats->timeouts, 1ull);
        atomicOr(b.status, kStatusMlpTimeout);
    }
    mlp_teardown(sm, st);
}

// Self-check of tl_b2_quick (no counterpart in the reference): every entry of
// the last run's phase-A survivor list judged by the filter and by the exact
// phases B1 and B2.  out[10]: entries; through exact phase B1; through exact
// phases B1 and B2; rejected by the filter; rejected by the filter but
// through the exact phases (must be 0); rejected by the filter among those
// through exact phase B1; the largest |filter value - exact value| / the
// filter's bound for deltaBeta, dBetaCut2 and betaOut (float bits; below 1
// when the bounds hold); entries the filter left before reaching the cuts;
// entries it finds through phase B2; of those, entries through exact phase B1
// but not exact phase B2 (must be 0).
__global__ void __launch_bounds__(256) k_tl_b2q_check(BatchDev b, unsigned long long* out) {
    const int64_t n = min((int64_t)*b.n_kept, b.kept_cap);
    unsigned long long c[6] = {0, 0, 0, 0, 0, 0}, inc = 0, acc = 0, acc_bad = 0;
    float rmax[3] = {0.f, 0.f, 0.f};
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
        const int4 e = AT(b.passa, i, b.kept_cap);
        (void)IX(e.x, b.obj[kSG].cap);
        (void)IX(e.y, b.obj[kSG].cap);
        const SGV S = load_sgv(b.sgpack, e.x), T = load_sgv(b.sgpack, e.y);
        float cut, muls;
        tl_cut_values(e.z, S, T, cut, muls);
        const bool p1 = tl_phaseB1_sgv(e.z, S, T, cut);
        float rec[kTLVarN];
        rec[kTLVarDBeta] = __int_as_float(0x7fc00000);
        const bool p2 = p1 && tl_phaseB2_sgv<kB2All>(e.z, S, T, muls, false, rec);
        B2Quick q;
        const int full = tl_b2_quick(e.z, S, T, &q);
        const int f = b2_early(e.z, T.flags) && b2_reject_early(S, load_sgo_beta(b.sgouter, b.obj[kSG].cap, e.y)) ? 0 : full;
        c[0] += 1;
        c[1] += p1;
        c[2] += p2;
        c[3] += f == 0;
        c[4] += f == 0 && p2;
        c[5] += f == 0 && p1;
        inc += f != 0 && !q.complete;
        acc += f == 3;
        acc_bad += f == 3 && p1 && !p2;
        if (p1 && q.complete && rec[kTLVarDBeta] == rec[kTLVarDBeta]) {
            rmax[0] = fmaxf(rmax[0], fabsf(q.dbeta - rec[kTLVarDBeta]) / q.e_dbeta);
            rmax[1] = fmaxf(rmax[1], fabsf(q.cut2 - rec[kTLVarDBetaCut2]) / q.e_cut2);
            rmax[2] = fmaxf(rmax[2], fabsf(q.bout - rec[kTLVarBetaOut]) / q.e_bout);
        }
    }
    for (int k = 0; k < 6; ++k) atomicAdd(out + k, c[k]);
    for (int k = 0; k < 3; ++k) atomicMax(out + 6 + k, (unsigned long long)__float_as_uint(rmax[k]));
    atomicAdd(out + 9, inc);
    atomicAdd(out + 10, acc);
    atomicAdd(out + 11, acc_bad);
}

// Phase B1 on a survivor list of phase A (count entries of list/muls); the candidates
// through it go to the phase-B2 list, BBBB ones from the front and the others
// from the back, so that phase B2's warps mostly run one algorithm.  Front
// and back never meet: together they hold at most count <= kept_cap entries.
// Each warp collects its BBBB and its other survivors in two shared-memory
// buffers and appends each with one atomic per batch (as passbuf_add).
__device__ __forceinline__ void pb_flush(const BatchDev& b, int4* buf, int& n, bool front) {
    __syncwarp();
    const int lane = threadIdx.x & 31;
    unsigned long long p0 = 0;
    if (lane == 0 && n) p0 = atomicAdd(b.n_pb + (front ? 0 : 1), (unsigned long long)n);
    p0 = __shfl_sync(0xffffffffu, p0, 0);
    for (int k = lane; k < n; k += kWarp) {
        const int64_t q = (int64_t)p0 + k;  // below the list length <= kept_cap
        AT(b.pb, front ? q : b.kept_cap - 1 - q, b.kept_cap) = buf[k];
    }
    __syncwarp();
    n = 0;
}

// Phase B2's single-precision decision (tl_b2_quick, no counterpart in the
// reference) on a survivor list (in / n_in: the enumeration's, or the
// pre-filter's kept list): the entries it cannot reject go to the filtered
// list (n_keptf entries, same format), which phase B1 reads.  Exact phase B2
// passes about one in thirteen of the enumeration's entries, so the filter
// spares the exact phases (float-float arithmetic and the host libm's
// functions) most of their work; the tracklets do not change.  Each warp
// takes blocks of 32 consecutive entries (one tile's survivors are
// consecutive, so their segment records are shared in L1) and appends its
// kept entries in batches.  Pass 0 evaluates the common case (BBBB without a
// 2S endcap outer anchor) and defers the entries of the long branches to the
// phase-B2 list pb (unused until phase B1): BBEE entries to its front, EEEE
// and the 2S endcap BBBB entries to its back; passes 1 and 2 evaluate the
// front and the back, so that each pass's warps mostly run one branch.  An
// entry the filter finds through phase B2 by more than its bounds, whose
// phase B1 the enumeration decided already (passed), is a tracklet: it is
// appended here as k_tl_b2 would, and the exact phases skip it.
// kEarly (pass 0 on the enumeration's list): b2_reject_early drops most of the
// entries that fail, and the others wait in shared memory for a full warp of
// tl_b2_quick.  (PU 100-300: 85 % of the entries are dropped; 64 events, 52
// million entries: the filter 1.64 -> 1.10 ms.  The pre-filter's kept list has
// two passing entries in three and goes straight to tl_b2_quick.)
// The first pass is bound by the latency of its loads at 32 warps an SM: the
// next entry is loaded ahead and the fields of both segments together (64
// events: 936 -> 842 us).
template <int kPass, bool kEarly>
__device__ __forceinline__ void tl_b2f(const BatchDev& b, const int4* __restrict__ in, const unsigned long long* n_in,
                                       int4 (*fbuf)[kPassBuf], int4 (*dbuf)[2][kPbBuf], int (*tbuf)[3][kRecBuf],
                                       int4 (*qbuf)[2 * kWarp]) {
    constexpr bool kDefer = kPass == 0;
    int64_t n;
    if (kPass == 0) {
        n = min((int64_t)*n_in, b.kept_cap);
    } else {
        const int64_t nf = min((int64_t)b.n_pb[0], b.kept_cap);
        n = kPass == 1 ? nf : min((int64_t)b.n_pb[1], b.kept_cap - nf);
    }
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const unsigned lt = (1u << lane) - 1u;
    int4* buf = fbuf[w];
    int4* dfront = kDefer ? dbuf[w][0] : nullptr;
    int4* dback = kDefer ? dbuf[w][1] : nullptr;
    RecBuf<0> tl{tbuf[w]};
    int nb = 0, nf = 0, nk = 0, nq = 0;
    // p0 + nb <= the input length <= kept_cap: the filtered list cannot overflow
    auto flush = [&]() {
        __syncwarp();
        unsigned long long p0 = 0;
        if (lane == 0 && nb) p0 = atomicAdd(b.n_keptf, (unsigned long long)nb);
        p0 = __shfl_sync(0xffffffffu, p0, 0);
        for (int i = lane; i < nb; i += kWarp) AT(b.passf, (int64_t)p0 + i, b.kept_cap) = buf[i];
        __syncwarp();
        nb = 0;
    };
    // what tl_b2_quick says of the lanes' entries: 4 a tracklet, 1 undecided
    auto settle = [&](int4 e, int r) {
        const unsigned mt = __ballot_sync(0xffffffffu, r == 4);
        if (mt) {
            if (tl.n + __popc(mt) > kRecBuf) rec_flush<0>(b, kTL, tl);
            if (r == 4) {
                const int k = tl.n + __popc(mt & lt);
                tl.e[0][k] = e.x;
                tl.e[1][k] = e.y;
                tl.e[2][k] = OG(b, kSG, e.x);
            }
            tl.n += __popc(mt);
        }
        const unsigned m = __ballot_sync(0xffffffffu, r == 1);
        if (nb + __popc(m) > kPassBuf) flush();
        if (r == 1) buf[nb + __popc(m & lt)] = e;
        nb += __popc(m);
    };
    auto judge = [&](int4 e) {
        const int r = tl_b2_quick<kDefer>(e.z, load_sgv(b.sgpack, e.x), load_sgv(b.sgpack, e.y));
        return r == 3 ? (e.w ? 4 : 1) : r;  // (phase B1 undecided: both exact phases run)
    };
    // the entries in the queue, 32 at a time (the last ones with `all`)
    auto drain = [&](bool all) {
        while (nq >= kWarp || (all && nq > 0)) {
            __syncwarp();
            const int m = min(nq, kWarp);
            int r = 0;
            int4 e = make_int4(0, 0, 0, 0);
            if (lane < m) {
                e = qbuf[w][nq - m + lane];
                r = judge(e);
            }
            settle(e, r);
            nq -= m;
            __syncwarp();
        }
    };
    const int64_t warps = (int64_t)gridDim.x * (kEnumThreads / kWarp);
    auto entry = [&](int64_t i) {
        return i >= n ? make_int4(0, 0, 0, 0)
                      : kPass == 0 ? AT(in, i, b.kept_cap) : AT(b.pb, kPass == 1 ? i : b.kept_cap - 1 - i, b.kept_cap);
    };
    const int64_t first = ((int64_t)blockIdx.x * (kEnumThreads / kWarp) + w) * kWarp;
    // (the next entry is on its way while one is judged)
    int4 next = entry(first + lane);
    for (int64_t base = first; base < n; base += warps * kWarp) {
        const int64_t i = base + lane;
        int r = 0;
        bool queue = false;
        const int4 e = next;
        next = entry(i + warps * kWarp);
        if (i < n) {
            (void)IX(e.x, b.obj[kSG].cap);
            (void)IX(e.y, b.obj[kSG].cap);
            if (kEarly) {
                // (the outer segment's part from the per-field arrays: a tile's
                // entries are neighbours there, while the 128-byte records
                // cost a cache line per lane and load)
                const int64_t C = b.obj[kSG].cap;
                r = 2;
                if (e.z == kAlgoBBBB) {
                    // (all loads together: the flags decide afterwards)
                    const uint32_t flags = sgo_flags(b.sgouter, C, e.y);
                    const bool out = b2_reject_early(load_sgv(b.sgpack, e.x), load_sgo_beta(b.sgouter, C, e.y));
                    if (b2_early(e.z, flags)) {
                        r = 0;
                        queue = !out;
                    }
                }
            } else {
                r = judge(e);
            }
        }
        if (kEarly) {
            const unsigned m = __ballot_sync(0xffffffffu, queue);
            if (queue) qbuf[w][nq + __popc(m & lt)] = e;
            nq += __popc(m);
            drain(false);
        } else {
            settle(e, r);
        }
        if (kDefer) {
            // (the deferred entries fit: together at most the input length <= kept_cap)
            const bool front = e.z == kAlgoBBEE;
            const unsigned mf = __ballot_sync(0xffffffffu, r == 2 && front);
            const unsigned mk = __ballot_sync(0xffffffffu, r == 2 && !front);
            if (nf + __popc(mf) > kPbBuf) pb_flush(b, dfront, nf, true);
            if (nk + __popc(mk) > kPbBuf) pb_flush(b, dback, nk, false);
            if (r == 2 && front) dfront[nf + __popc(mf & lt)] = e;
            if (r == 2 && !front) dback[nk + __popc(mk & lt)] = e;
            nf += __popc(mf);
            nk += __popc(mk);
        }
    }
    if (kEarly) drain(true);
    flush();
    rec_flush<0>(b, kTL, tl);
    if (kDefer) {
        pb_flush(b, dfront, nf, true);
        pb_flush(b, dback, nk, false);
    }
}
// pass 0
template <bool kEarly>
__global__ void __launch_bounds__(kEnumThreads, 4) k_tl_b2f(BatchDev b, const int4* __restrict__ in, const unsigned long long* n_in) {
    __shared__ int4 fbuf[kEnumThreads / kWarp][kPassBuf];
    __shared__ int4 dbuf[kEnumThreads / kWarp][2][kPbBuf];
    __shared__ int tbuf[kEnumThreads / kWarp][3][kRecBuf];
    __shared__ int4 qbuf[kEarly ? kEnumThreads / kWarp : 1][2 * kWarp];
    if (halted(b)) return;
    tl_b2f<0, kEarly>(b, in, n_in, fbuf, dbuf, tbuf, qbuf);
}
// passes 1 and 2; 0: both, by blockIdx.y (launch_pair)
template <int kPass>
__global__ void __launch_bounds__(kEnumThreads, 4) k_tl_b2f_rest(BatchDev b) {
    __shared__ int4 fbuf[kEnumThreads / kWarp][kPassBuf];
    __shared__ int tbuf[kEnumThreads / kWarp][3][kRecBuf];
    if (halted(b)) return;
    if (kPass == 1 || (kPass == 0 && blockIdx.y == 0)) tl_b2f<1, false>(b, nullptr, nullptr, fbuf, nullptr, tbuf, nullptr);
    else tl_b2f<2, false>(b, nullptr, nullptr, fbuf, nullptr, tbuf, nullptr);
}

// Entries a warp takes at a time of a list of n: 32, or one where there are four
// warps for each.  The lanes of a warp part ways in the exact phases, so a short
// list (what the phase-B2 filter leaves of one event) takes as long as all their
// ways one after the other: phases B1 and B2 of one PU 200 event 36 us with 32
// entries a warp, 30 with one.  A longer list spread over all warps only fetches
// more instructions (64 events: 42 us with 32 entries a warp, 88 spread out).
__device__ __forceinline__ int entries_per_warp(int64_t n, int64_t nwarp) { return 4 * n <= nwarp ? 1 : kWarp; }

__global__ void __launch_bounds__(kEnumThreads) k_tl_b1(BatchDev b, const int4* __restrict__ list,
                                                         const unsigned long long* count) {
    __shared__ int4 fbuf[kEnumThreads / kWarp][kPbBuf], bbuf[kEnumThreads / kWarp][kPbBuf];
    if (halted(b)) return;
    const int64_t n = min((int64_t)*count, b.kept_cap);
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    int nfb = 0, nbb = 0;  // entries held in this warp's buffers
    const int64_t nwarp = (int64_t)gridDim.x * (kEnumThreads / 32);
    const int per = entries_per_warp(n, nwarp);
    for (int64_t base = ((int64_t)blockIdx.x * (kEnumThreads / 32) + w) * per; base < n; base += nwarp * per) {
        const int64_t i = base + lane;
        bool pass = false;
        int4 p = make_int4(0, 0, kAlgoNone, 0);
        float muls = 0.f;
        if (lane < per && i < n) {
            p = AT(list, i, b.kept_cap);
            if (p.w) {  // phase B1 passed in the enumeration
                pass = true;
                muls = tl_muls_entry(p.z, b.sgpack, p.x, p.y);
            } else {
                const B1Result r = tl_phaseB1_entry(p.z, b.sgpack, p.x, p.y);
                pass = r.pass;
                muls = r.muls;
            }
        }
        const bool front = pass && p.z == kAlgoBBBB;
        const unsigned mf = __ballot_sync(0xffffffffu, front);
        const unsigned mb = __ballot_sync(0xffffffffu, pass && !front);
        if (!(mf | mb)) continue;
        if (nfb + __popc(mf) > kPbBuf) pb_flush(b, fbuf[w], nfb, true);
        if (nbb + __popc(mb) > kPbBuf) pb_flush(b, bbuf[w], nbb, false);
        if (pass) {
            const unsigned below = (1u << lane) - 1u;
            const int4 e = make_int4(p.x, p.y, p.z, __float_as_int(muls));
            if (front) fbuf[w][nfb + __popc(mf & below)] = e;
            else bbuf[w][nbb + __popc(mb & below)] = e;
        }
        nfb += __popc(mf);
        nbb += __popc(mb);
    }
    pb_flush(b, fbuf[w], nfb, true);
    pb_flush(b, bbuf[w], nbb, false);
}

// CTAs per SM the phase-B2 kernels are compiled for (register budget; 4
// measured fastest on the 128-event PU 150-300 batch: phase B1+B2 8.1 ms
// against 9.7 ms at 1, plain chain's B2 54.9 ms against 58.5 ms)
#ifndef SDLG_B2_MIN_BLOCKS
#define SDLG_B2_MIN_BLOCKS 4
#endif
constexpr int kB2MinBlocks = SDLG_B2_MIN_BLOCKS;

// Phase B2 on one part of the phase-B2 list (kSet kB2BBBB: the front, BBBB
// entries; kB2Others: the back, BBEE and EEEE entries); appends the tracklets.
template <int kSet>
__device__ __forceinline__ void tl_b2(const BatchDev& b, int (*rbuf)[3][kRecBuf]) {
    const int64_t nf = min((int64_t)b.n_pb[0], b.kept_cap);
    const int64_t n = kSet == kB2BBBB ? nf : min((int64_t)b.n_pb[1], b.kept_cap - nf);
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const bool nm1 = (b.flags & kFlagTLNm1) != 0;
    const int64_t nwarp = (int64_t)gridDim.x * (kEnumThreads / 32);
    RecBuf<0> rb{rbuf[w]};
    const int per = entries_per_warp(n, nwarp);
    for (int64_t base = ((int64_t)blockIdx.x * (kEnumThreads / 32) + w) * per; base < n; base += nwarp * per) {
        const int64_t i = base + lane;
        bool pass = false;
        int s = 0, tt = 0;
        if (lane < per && i < n) {
            const int64_t k = kSet == kB2BBBB ? i : b.kept_cap - 1 - i;
            const int4 p = AT(b.pb, k, b.kept_cap);
            s = p.x;
            tt = p.y;
            pass = tl_phaseB2<kSet>(p.z, b.sgpack, s, tt, __int_as_float(p.w), nm1);
        }
        const unsigned m = __ballot_sync(0xffffffffu, pass);
        if (!m) continue;
        if (rb.n + __popc(m) > kRecBuf) rec_flush<0>(b, kTL, rb);
        if (pass) {
            const int k = rb.n + __popc(m & ((1u << lane) - 1u));
            rb.e[0][k] = s;
            rb.e[1][k] = tt;
            rb.e[2][k] = OG(b, kSG, s);
        }
        rb.n += __popc(m);
    }
    rec_flush<0>(b, kTL, rb);
}
// blockIdx.y 0: the list's front, 1: its back; an entry takes some 25 us from
// end to end, so the parts run side by side (phases B1 and B2 of one PU 200
// event: 55 -> 36 us)
__global__ void __launch_bounds__(kEnumThreads, kB2MinBlocks) k_tl_b2(BatchDev b) {
    __shared__ int rbuf[kEnumThreads / kWarp][3][kRecBuf];
    if (halted(b)) return;
    if (blockIdx.y == 0) tl_b2<kB2BBBB>(b, rbuf);
    else tl_b2<kB2Others>(b, rbuf);
}

__device__ __forceinline__ float hash_unit(unsigned long long c, unsigned long long seed) {
    // splitmix64 finaliser (Steele, Lea, Flood 2014)
    unsigned long long z = c + seed * 0x9E3779B97F4A7C15ull + 0x632BE59BD9B4E019ull;
    z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
    z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
    z ^= z >> 31;
    return (float)(z >> 40) * (1.0f / 16777216.0f);
}

// Training samples for the learned pre-filter: the features of every
// tracklet candidate of the last run that passes phase A, labelled by phase
// B (the plain chain's accept / reject); rejected ones are kept with
// probability neg_keep.
__global__ void k_tl_collect(BatchDev b, MlpCollect col) {
    if (halted(b)) return;
    const int64_t nobj = n_inner(b, kTL);
    if (nobj <= 0) return;
    const int64_t* off = b.cand[kTL];
    const int64_t offlim = b.cand_cap[kTL] + 1;
    const int64_t total = AT(off, nobj, offlim);
    const int lay = tl_variant(b);
    const int lane = threadIdx.x & 31;
    for (int64_t c0 = (int64_t)blockIdx.x * blockDim.x; c0 < total; c0 += (int64_t)gridDim.x * blockDim.x) {
        const int64_t c = c0 + threadIdx.x;
        bool keep = false;
        float label = 0.f;
        float f[kMlpIn];
        if (c < total) {
            int lo, hi;
            obj_bounds(b, nobj, total, c, c, lo, hi);
            const int s = find_obj(b, off, offlim, lo, hi, c);
            const int tt = tl_outer_of(b, lay, s, c - AT(off, s, offlim));
            const SGV S = load_sgv(b.sgpack, s);
            const SGV T = load_sgv(b.sgpack, tt);
            float cut = 0.f, muls = 0.f;
            const int algo = tl_phaseA(S, T, cut, muls);
            if (algo != kAlgoNone) {
                const bool pass = tl_phaseB(algo, b.sgpack, s, tt, cut, muls, false);
                label = pass ? 1.f : 0.f;
                keep = pass || hash_unit((unsigned long long)c, col.seed) < col.neg_keep;
                if (keep) tl_features(feat_s(b.sgfeat, b.obj[kSG].cap, s), feat_t(b.sgfeat, b.obj[kSG].cap, tt), f);
            }
        }
        const unsigned m = __ballot_sync(0xffffffffu, keep);
        if (!m) continue;
        const int leader = __ffs(m) - 1;
        unsigned long long p0 = 0;
        if (lane == leader) p0 = atomicAdd(col.n, (unsigned long long)__popc(m));
        p0 = __shfl_sync(0xffffffffu, p0, leader);
        const int64_t pos = (int64_t)p0 + __popc(m & ((1u << lane) - 1u));
        if (keep && pos < col.cap) {
#pragma unroll
            for (int k = 0; k < kMlpIn; ++k) col.x[pos * kMlpIn + k] = f[k];
            col.y[pos] = label;
        }
    }
}

// Self-check of the enumeration's single-precision decisions (tl_ab1_decide:
// phase A, then phase B1 for its survivors; tl_layer_out ahead of it) over the tracklet candidates of
// the last run, against the exact phase A and B1 on the packed records:
// out[0] candidates, out[1] settled by the approximations alone, out[2] that
// needed an exact evaluation, out[3] settled wrongly (0 when the margins
// hold): rejected although both phases pass, accepted with another
// algorithm or although phase A fails, or marked as through phase B1 although
// it fails.
__global__ void k_tl_quick_check(BatchDev b, unsigned long long* out) {
    if (halted(b)) return;
    const int64_t nobj = n_inner(b, kTL);
    if (nobj <= 0) return;
    const int64_t* off = b.cand[kTL];
    const int64_t offlim = b.cand_cap[kTL] + 1;
    const int64_t total = AT(off, nobj, offlim);
    const int lay = tl_variant(b);
    unsigned long long n[4] = {0ull, 0ull, 0ull, 0ull};
    for (int64_t c = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; c < total; c += (int64_t)gridDim.x * blockDim.x) {
        int lo, hi;
        obj_bounds(b, nobj, total, c, c, lo, hi);
        const int s = find_obj(b, off, offlim, lo, hi, c);
        const int tt = tl_outer_of(b, lay, s, c - AT(off, s, offlim));
        const SGV S = load_sgv(b.sgpack, s), Tv = load_sgv(b.sgpack, tt);
        const int64_t C = b.obj[kSG].cap;
        const SGOuter T = load_sgo(b.sgouter, C, tt);
        int b1 = 0, q = kAlgoNone;
        bool exact = false;
        if (lay != 1 || !tl_layer_out(b.sgpack, s, T))
            q = tl_ab1_decide<false>(tl_row(S), tl_out(T), load_sgo_xy(b.sgouter, C, tt), b.sgpack, s, tt, b1, exact);
        float cut, muls;
        const int e = tl_phaseA(S, Tv, cut, muls);
        const bool eb1 = e != kAlgoNone && tl_phaseB1_sgv(e, S, Tv, cut);
        const bool bad = q == kAlgoNone ? eb1 : (q != e || (b1 && !eb1));
        n[0] += 1;
        n[1] += !exact;
        n[2] += exact;
        n[3] += bad;
    }
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        unsigned long long v = n[k];
        for (int o = 16; o; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
        if ((threadIdx.x & 31) == 0 && v) atomicAdd(out + k, v);
    }
}

// Self-check of the first passes over the mini-doublet and segment candidates
// (md_first_cuts; sg_first_cuts and sg_later_cuts): every candidate of the last
// run judged by them and by the whole algorithm.  out[0..3] mini-doublets,
// out[4..7] segments: candidates, rejected by the first pass, of those accepted
// by the algorithm (must be 0), accepted by the algorithm.
__device__ __forceinline__ void first_cuts_count(unsigned long long* out, unsigned long long (&n)[4]) {
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        for (int o = 16; o; o >>= 1) n[k] += __shfl_down_sync(0xffffffffu, n[k], o);
        if ((threadIdx.x & 31) == 0 && n[k]) atomicAdd(out + k, n[k]);
    }
}
__global__ void k_md_first_check(BatchDev b, unsigned long long* out) {
    const int64_t* off = b.cand[kMD];
    const int64_t offlim = b.cand_cap[kMD] + 1;
    const int64_t total = b.n_gm > 0 ? AT(off, b.n_gm, offlim) : 0;
    unsigned long long n[4] = {0ull, 0ull, 0ull, 0ull};
    for (int64_t c = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; c < total; c += (int64_t)gridDim.x * blockDim.x) {
        const int g = find_obj(b, off, offlim, 0, b.n_gm - 1, c);
        int2 e;
        if (!md_candidate(b, g, c - AT(off, g, offlim), e)) continue;
        const ModDev& lm = MOD(b, mod_of(b, g));
        const MDCand d = md_cand(b, lm, e);
        const bool first = md_first_cuts(d.L, d.U, d.pixAsin, lm, d.sh);
        MDVals v;
        const bool pass = lm.subdet == kBarrel ? md_barrel(d.L, d.U, d.pixAsin, lm, d.sh, v) : md_endcap(d.L, d.U, d.pixAsin, lm, d.sh, v);
        n[0] += 1;
        n[1] += !first;
        n[2] += !first && pass;
        n[3] += pass;
    }
    first_cuts_count(out, n);
}
__global__ void k_sg_first_check(BatchDev b, unsigned long long* out) {
    const int64_t nobj = n_objects(b, kMD);
    const int64_t* off = b.cand[kSG];
    const int64_t offlim = b.cand_cap[kSG] + 1;
    const int64_t total = nobj > 0 ? AT(off, nobj, offlim) : 0;
    unsigned long long n[4] = {0ull, 0ull, 0ull, 0ull};
    for (int64_t c = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; c < total; c += (int64_t)gridDim.x * blockDim.x) {
        const int a = find_obj(b, off, offlim, 0, (int)nobj - 1, c);
        const int64_t q = c - AT(off, a, offlim);
        const int bmd = b.seg_layers ? layer_md<true>(b, layer_row<true>(b, a), (int)q) : sg_outer_conn(b, a, q);
        const MDLite I = md_lite(b, a), O = md_lite(b, bmd);
        const bool first = sg_first_cuts(I, O) && sg_later_cuts(I, O);
        float f6[6];
        const bool pass = sg_pair(b, a, bmd, !b.seg_layers || sg_connected(b, a, bmd), f6);
        n[0] += 1;
        n[1] += !first;
        n[2] += !first && pass;
        n[3] += pass;
    }
    first_cuts_count(out, n);
}

// per-module object counts of a stage -> offsets, and the layer counters
template <int st, bool kCounters>
struct ScanObj : ScanOp {
    static constexpr int kVals = 1, kSmall = 1, kBig = 8;
    __device__ static int64_t size(const BatchDev& b) { return b.n_gm; }
    __device__ static void load(const BatchDev& b, int64_t g, bool in, int64_t* v) {
        v[0] = in ? OFF(b, st, g) : 0;
        if (!kCounters) return;
        const bool act = v[0] != 0;
        int ev = 0, slot = 0;
        if (act) {
            ev = ev_of(b, g);
            slot = MOD(b, g - (int64_t)ev * b.geo.n_mod).layer_slot;
        }
        warp_add(act ? counter_at(b, ev, st, 1, slot) : b.counters, (uint32_t)v[0], act);
    }
    __device__ static void store(const BatchDev& b, int64_t g, const int64_t* e, const int64_t*) {
        AT(b.obj[st].mod_cnt, g, NG1(b)) = e[0];
    }
    __device__ static void total(const BatchDev& b, int64_t n, const int64_t* t) { AT(b.obj[st].mod_cnt, n, NG1(b)) = t[0]; }
};

// The tracklets that can be the outer one of a track candidate (g: the inner
// module): those starting in barrel layer 3 (Event.cc:835), or all for
// createTrackCandidatesFromTracklets.  Only these are indexed (128 dense events:
// the track-candidate stage took 0.80 ms with all of them, 0.59 now).
__device__ __forceinline__ bool tl_joins(const BatchDev& b, int g) {
    if (b.flags & kFlagTCFromTL) return true;
    const ModDev& m = MOD(b, mod_of(b, g));
    return m.subdet == kBarrel && m.layer == 3;
}
// a tracklet's place among those of its inner segment s (0 when not indexed)
__device__ __forceinline__ int tl_join_add(const BatchDev& b, int g, int s) {
    return tl_joins(b, g) ? (int)atomicAdd((unsigned long long*)&AT(b.joft, sg_key(b, s), b.obj[kSG].cap + 1), 1ull) : 0;
}
__global__ void k_tl_join_count(BatchDev b) {
    if (halted(b)) return;
    const int64_t n = n_objects(b, kTL);
    for (int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; t < n; t += (int64_t)gridDim.x * blockDim.x)
        AT(b.trank, t, b.obj[kTL].cap) = tl_join_add(b, OG(b, kTL, t), OI(b, kTL, t));
}

// The stage's records into the dense arrays grouped by inner module.  kJoin
// (tracklets): with each one's place among those of its inner segment, for the
// track candidates (when that stage is part of the run; otherwise it does that
// itself).  The counts that later stages accumulate per mini-doublet and per
// segment start at zero here, where their number is known.  (The packed
// records of mini-doublets and segments are not written here: in the records'
// order their writes and the hits' reads scatter, segment stage of 128 dense
// events 7.1 -> 11.9 ms, and one PU 200 event gained nothing either.)
template <int st, bool kJoin>
__global__ void __launch_bounds__(256) k_scatter(BatchDev b) {
    if (halted(b)) return;
    const Recs& R = b.rec[st];
    const Objs& O = b.obj[st];
    const int64_t n = min(b.n_rec[st * kLine], O.cap);
    const int64_t tid = (int64_t)blockIdx.x * blockDim.x + threadIdx.x, stride = (int64_t)gridDim.x * blockDim.x;
    constexpr int kNF = st == kMD ? 4 : (st == kSG ? 6 : 0);
    for (int64_t r = tid; r < n; r += stride) {
        const int g = AT(R.g, r, O.cap);
        const int64_t pos = OFF(b, st, g) + AT(R.rank, r, O.cap);
        if (pos >= O.cap) continue;
        const int i = AT(R.i, r, O.cap);
        AT(O.i, pos, O.cap) = i;
        AT(O.j, pos, O.cap) = AT(R.j, r, O.cap);
        AT(O.g, pos, O.cap) = g;
#pragma unroll
        for (int k = 0; k < kNF; ++k)
            AT(O.f, (int64_t)k * O.cap + pos, O.cap * kNF) = AT(R.f, (int64_t)k * O.cap + r, O.cap * kNF);
        if (kJoin) AT(b.trank, pos, O.cap) = tl_join_add(b, g, i);
    }
    if (st == kMD && b.joff)
        for (int64_t k = tid; k <= n; k += stride) AT(b.joff, k, O.cap + 1) = 0;
    if (st == kSG)
        for (int64_t k = tid; k <= n; k += stride) AT(b.joft, k, O.cap + 1) = 0;
}

// ------------------------------------------------------------------ counts
// mini-doublet candidates of a module: lower x upper hits (Event.cc:257-301)
struct ScanMdCand : ScanCand<kMD> {
    __device__ static void load(const BatchDev& b, int64_t g, bool in, int64_t* v) {
        int64_t c = 0;
        int ev = 0, slot = 0;
        if (in) {
            ev = ev_of(b, g);
            const ModDev& m = MOD(b, g - (int64_t)ev * b.geo.n_mod);
            if (m.lower && m.partner >= 0) {
                const int64_t pg = (int64_t)ev * b.geo.n_mod + m.partner;
                c = (AT(b.mod_hit, g + 1, NG1(b)) - AT(b.mod_hit, g, NG1(b))) *
                    (AT(b.mod_hit, pg + 1, NG1(b)) - AT(b.mod_hit, pg, NG1(b)));
            }
            slot = m.layer_slot;
        }
        const bool act = c != 0;
        warp_add(act ? counter_at(b, ev, kMD, 0, slot) : b.counters, (uint32_t)c, act);
        v[0] = c;
    }
};

// The connection entries of 32 consecutive modules (one per lane, g; `need`:
// the lane's sums are wanted): running sums of the connected modules' object
// counts (stage src) -> conn_pref and conn_first per entry, conn_sum per
// module (returned; 0 where not wanted).  Half a warp takes a module, an
// entry per lane: the lists have 15 entries on average and 33 at most.  Every
// lane of the warp calls it.
__device__ __forceinline__ int64_t conn_sums(const BatchDev& b, int64_t g, bool need, int src) {
    constexpr int kL = 16;
    const int n_mod = b.geo.n_mod;
    const int lane = threadIdx.x & 31, half = lane / kL, l = lane % kL;
    int ev = 0, k0 = 0, k1 = 0;
    if (need) {
        ev = ev_of(b, g);
        const int m = (int)(g - (int64_t)ev * n_mod);
        k0 = AT(b.geo.conn_off, m, NM(b) + 1);
        k1 = AT(b.geo.conn_off, m + 1, NM(b) + 1);
    }
    int64_t sum = 0;
    for (unsigned act = __ballot_sync(0xffffffffu, k1 > k0); act;) {
        const int j0 = __ffs(act) - 1;
        act &= act - 1u;
        const int j1 = act ? __ffs(act) - 1 : -1;
        act &= act - 1u;  // (0 stays 0)
        const int j = half ? j1 : j0, js = j < 0 ? 0 : j;
        const int64_t ej = __shfl_sync(0xffffffffu, ev, js);
        const int e0 = __shfl_sync(0xffffffffu, k0, js);
        const int e1s = __shfl_sync(0xffffffffu, k1, js), e1 = j < 0 ? e0 : e1s;
        const int64_t pbase = ej * b.geo.n_conn, ebase = ej * n_mod;
        int run = 0;
        for (int k = e0 + l; __any_sync(0xffffffffu, k < e1); k += kL) {
            int first = 0, x = 0, cnt = 0;
            if (k < e1) {
                const int64_t g2 = ebase + AT(b.geo.conn_idx, k, NC(b));
                first = (int)OFF(b, src, g2);
                x = cnt = (int)OFF(b, src, g2 + 1) - first;
            }
#pragma unroll
            for (int o = 1; o < kL; o <<= 1) {
                const int y = __shfl_up_sync(0xffffffffu, x, o, kL);
                if (l >= o) x += y;
            }
            if (k < e1) {
                AT(b.conn_pref, pbase + k, NCP(b)) = run + x - cnt;
                AT(b.conn_first, pbase + k, NCP(b)) = first;
            }
            run += __shfl_sync(0xffffffffu, x, kL - 1, kL);
        }
        const int r0 = __shfl_sync(0xffffffffu, run, 0), r1 = __shfl_sync(0xffffffffu, run, kL);
        if (lane == j0) sum = r0;
        if (lane == j1) sum = r1;
    }
    return sum;
}

// the reference's candidate counters of stage st get c for an object's
// (module's) candidates, by the layer of module g; every lane calls it
__device__ __forceinline__ void count_cand(const BatchDev& b, int st, int64_t g, int64_t c) {
    const bool act = c != 0;
    int ev = 0, slot = 0;
    if (act) {
        ev = ev_of(b, g);
        slot = MOD(b, g - (int64_t)ev * b.geo.n_mod).layer_slot;
    }
    warp_add(act ? counter_at(b, ev, st, 0, slot) : b.counters, (uint32_t)c, act);
}

// connection sums over the objects of stage src for every module, and the
// candidate counters of stage cst (none when negative): n_obj(g) * conn_sum(g)
__device__ __forceinline__ int64_t conn_sum_of(const BatchDev& b, int64_t g, bool in, bool need, int src, int cst) {
    const int64_t sum = conn_sums(b, g, in && need, src);
    if (in) AT(b.conn_sum, g, b.n_gm) = sum;
    if (cst >= 0) count_cand(b, cst, g, in && need ? (OFF(b, src, g + 1) - OFF(b, src, g)) * sum : 0);
    return sum;
}
// kEnds: only for the modules that hold objects or in which segments end
template <bool kNeeded>
__device__ __forceinline__ bool conn_needed(const BatchDev& b, int64_t g, bool in, int src, bool ends) {
    return !kNeeded || (in && (OFF(b, src, g + 1) > OFF(b, src, g) || (ends && AT(b.eoff, g, NG1(b)) > 0)));
}
template <bool kNeeded>
__global__ void k_conn_sum(BatchDev b, int src, int cst, bool ends) {
    if (halted(b)) return;
    for (int64_t g = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; g - (threadIdx.x & 31) < b.n_gm; g += (int64_t)gridDim.x * blockDim.x)
        (void)conn_sum_of(b, g, g < b.n_gm, conn_needed<kNeeded>(b, g, g < b.n_gm, src, ends), src, cst);
}

// The front of the module-map segment stage: the connection sums over the
// mini-doublets, the offsets of the outer lists (toff: for every global
// module holding mini-doublets, the mini-doublets of its connected modules)
// and of the modules' candidates (coff: mini-doublets x outer list).
// kFused: with the connection sums (for many modules k_conn_sum makes them).
template <bool kFused>
struct ScanSgFront : ScanCand<kSG> {
    static constexpr int kVals = 2, kSmall = kFused ? 1 : 4, kBig = kSmall;  // (kFused: few modules)
    __device__ static int64_t size(const BatchDev& b) { return b.n_gm; }
    __device__ static void load(const BatchDev& b, int64_t g, bool in, int64_t* v) {
        const int64_t n = in ? OFF(b, kMD, g + 1) - OFF(b, kMD, g) : 0;
        int64_t sum = 0;
        if (kFused) sum = conn_sum_of(b, g, in, n > 0, kMD, kSG);
        else if (n > 0) sum = AT(b.conn_sum, g, b.n_gm);
        v[0] = n > 0 ? sum : 0;
        v[1] = n * sum;
    }
    __device__ static void store(const BatchDev& b, int64_t g, const int64_t* e, const int64_t*) {
        AT(b.toff, g, NG1(b)) = e[0];
        AT(b.coff, g, NG1(b)) = e[1];
    }
    __device__ static void total(const BatchDev& b, int64_t n, const int64_t* t) {
        AT(b.toff, n, NG1(b)) = t[0];
        put_total(b, n_inner(b, kSG), t[1]);
    }
};

// Eight lanes per module: the candidate offsets and buckets of its
// mini-doublets (a module's mini-doublets have one outer list, so their
// offsets are multiples of its length), and the outer list, written out
// (entry q of g's list at olist[toff[g] + q]) so that a candidate finds its
// outer mini-doublet with one load: each lane writes the mini-doublets of
// every eighth connection.  The lists are not written when they exceed
// olist_cap (the candidates then search the connection list).
__global__ void k_sg_lists(BatchDev b) {
    if (halted(b)) return;
    constexpr int kL = 8;
    const bool lists = AT(b.toff, b.n_gm, NG1(b)) <= b.olist_cap;
    const int n_mod = b.geo.n_mod;
    const int l = threadIdx.x % kL;
    for (int64_t g = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) / kL; g < b.n_gm; g += (int64_t)gridDim.x * blockDim.x / kL) {
        const int64_t a0 = OFF(b, kMD, g), a1 = OFF(b, kMD, g + 1);
        if (a0 == a1) continue;
        const int64_t o = AT(b.toff, g, NG1(b)), c0 = AT(b.coff, g, NG1(b)), sum = AT(b.conn_sum, g, b.n_gm);
        for (int64_t a = a0 + l; a < a1; a += kL) ScanCand<kSG>::put(b, a, c0 + (a - a0) * sum, sum);
        if (!lists) continue;
        const int ev = ev_of(b, g), m = (int)(g - (int64_t)ev * n_mod);
        const int k0 = AT(b.geo.conn_off, m, NM(b) + 1), k1 = AT(b.geo.conn_off, m + 1, NM(b) + 1);
        const int64_t pbase = (int64_t)ev * b.geo.n_conn;
        for (int k = k0 + l; k < k1; k += kL) {
            const int64_t p = AT(b.conn_pref, pbase + k, NCP(b));
            const int64_t n = (k + 1 < k1 ? (int64_t)AT(b.conn_pref, pbase + k + 1, NCP(b)) : sum) - p;
            const int first = AT(b.conn_first, pbase + k, NCP(b));
            for (int64_t i = 0; i < n; ++i) AT(b.olist, o + p + i, b.olist_cap) = first + (int)i;
        }
    }
}

// layer-pair segment candidates of every MD (Event.cc:805-818 loops over
// inner-layer MDs x outer-layer MDs); the reference counts none of them
struct ScanSgLayers : ScanCand<kSG> {
    __device__ static void load(const BatchDev& b, int64_t a, bool in, int64_t* v) {
        v[0] = in ? layer_row<true>(b, (int)a)[2 * b.layer_width - 1] : 0;
    }
};

// The front of the module-map tracklet stage: the connection sums over the
// segments, the offsets of the segments by the module they end in (eoff, from
// the counts there), of the module-pair tiles (toff, with the tile -> module
// map while it fits tile_cap; the enumeration searches toff otherwise) and
// the candidates' total.  kFused as above.
template <bool kFused>
struct ScanTlFront : ScanOp {
    static constexpr int kVals = 3, kSmall = kFused ? 1 : 4, kBig = kSmall;
    __device__ static int64_t size(const BatchDev& b) { return b.n_gm; }
    __device__ static void load(const BatchDev& b, int64_t g, bool in, int64_t* v) {
        v[0] = in ? AT(b.eoff, g, NG1(b)) : 0;
        int64_t sum = 0;
        if (kFused) sum = conn_sum_of(b, g, in, conn_needed<true>(b, g, in, kSG, true), kSG, kTP);
        else if (v[0] > 0) sum = AT(b.conn_sum, g, b.n_gm);
        v[1] = tile_count(b, v[0], sum);
        v[2] = v[0] * sum;
    }
    __device__ static void store(const BatchDev& b, int64_t g, const int64_t* e, const int64_t* v) {
        AT(b.eoff, g, NG1(b)) = e[0];
        AT(b.toff, g, NG1(b)) = e[1];
        for (int64_t t = e[1]; t < e[1] + v[1]; ++t)
            if (t < b.tile_cap) AT(b.tile_gm, t, b.tile_cap) = (int)g;
    }
    __device__ static void total(const BatchDev& b, int64_t n, const int64_t* t) {
        AT(b.eoff, n, NG1(b)) = t[0];
        AT(b.toff, n, NG1(b)) = t[1];
        *b.n_cand_tl = (unsigned long long)t[2];
    }
};

// Tracklet candidates of every segment as a flat space, for the enumeration
// of the layer pairs (Event.cc:762-787), of navigation (Event.cc:694-751) and
// for the samples and self-checks of the module map; kCount: with the
// reference's candidate counters
template <bool kCount>
struct ScanTlCand : ScanCand<kTL> {
    __device__ static void load(const BatchDev& b, int64_t s, bool in, int64_t* v) {
        int64_t c = 0;
        int ev = 0, slot = 0;
        if (in) {
            const int g1 = OG(b, kSG, s);
            ev = ev_of(b, g1);
            slot = MOD(b, g1 - ev * b.geo.n_mod).layer_slot;
            const int var = tl_variant(b);
            if (var == 1) {
                const int so = tl_layer_outer(slot);
                c = so >= 0 ? layer_count(b, kSG, ev, so) : 0;
            } else if (var == 2) {
                const int m = OJ(b, kSG, s);
                const int64_t nc = join_n(b, m);
                for (int64_t k = 0; k < nc; ++k) c += join_n(b, OJ(b, kSG, join_obj(b, m, k)));
            } else {
                c = AT(b.conn_sum, OG(b, kMD, OJ(b, kSG, s)), b.n_gm);
            }
        }
        const bool act = kCount && c != 0;
        warp_add(act ? counter_at(b, ev, kTL, 0, slot) : b.counters, (uint32_t)c, act);
        v[0] = c;
    }
    __device__ static void total(const BatchDev& b, int64_t n, const int64_t* t) {
        put_total(b, n, t[0]);
        *b.n_cand_tl = (unsigned long long)t[0];
    }
};

// the triplets by their innermost mini-doublet (createTrackCandidatesFromTriplets)
__global__ void k_join2_count(BatchDev b) {
    if (halted(b)) return;
    const int64_t n = n_objects(b, kTP);
    for (int64_t o = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; o < n; o += (int64_t)gridDim.x * blockDim.x) {
        atomicAdd((unsigned long long*)&AT(b.joff2, join_key(b, kTP, o), b.obj[kMD].cap + 1), 1ull);
        AT(b.tpend, OJ(b, kSG, OJ(b, kTP, o)), b.obj[kMD].cap) = 1;
    }
}
__global__ void k_join2_scatter(BatchDev b) {
    if (halted(b)) return;
    const int64_t n = n_objects(b, kTP);
    for (int64_t o = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; o < n; o += (int64_t)gridDim.x * blockDim.x) {
        const int k = join_key(b, kTP, o);
        const int64_t pos = AT(b.joff2, k, b.obj[kMD].cap + 1) + atomicAdd(&AT(b.jcur2, k, b.obj[kMD].cap), 1);
        AT(b.jidx2, pos, b.obj[kTP].cap) = (int)o;
    }
}
// counts of a join index (0: segments by mini-doublet, 1: triplets by
// mini-doublet, 2: tracklets by segment, 3: k_tctp_b's pairs by mini-doublet)
// -> offsets
template <int kIndex>
struct ScanJoin : ScanOp {
    static constexpr int kVals = 1, kSmall = 2, kBig = 8, kKey = kIndex == 2 ? kSG : kMD;
    __device__ static int64_t* off(const BatchDev& b) { return kIndex == 0 ? b.joff : (kIndex == 1 ? b.joff2 : (kIndex == 2 ? b.joft : b.joff3)); }
    __device__ static int64_t size(const BatchDev& b) { return n_objects(b, kKey); }
    __device__ static void load(const BatchDev& b, int64_t i, bool in, int64_t* v) {
        v[0] = in ? AT(off(b), i, b.obj[kKey].cap + 1) : 0;
    }
    __device__ static void store(const BatchDev& b, int64_t i, const int64_t* e, const int64_t*) {
        AT(off(b), i, b.obj[kKey].cap + 1) = e[0];
    }
    __device__ static void total(const BatchDev& b, int64_t n, const int64_t* t) { AT(off(b), n, b.obj[kKey].cap + 1) = t[0]; }
};

// how often module m2 occurs in the connection list of module m1
__device__ __forceinline__ int conn_mult(const BatchDev& b, int m1, int m2) {
    int mult = 0;
    const int k0 = AT(b.geo.conn_off, m1, NM(b) + 1), k1 = AT(b.geo.conn_off, m1 + 1, NM(b) + 1);
    for (int k = k0; k < k1; ++k) mult += AT(b.geo.conn_idx, k, NC(b)) == m2;
    return mult;
}

// The triplets and track candidates of every inner object, each of which is
// made (k_expand): their offsets are the objects' places, and the total is
// known before any is written.
template <int st>
struct ScanJoined : ScanCand<st> {
    __device__ static void store(const BatchDev& b, int64_t i, const int64_t* e, const int64_t*) {
        AT(b.cand[st], i, b.cand_cap[st] + 1) = e[0];
    }
    __device__ static void total(const BatchDev& b, int64_t n, const int64_t* t) {
        AT(b.cand[st], n, b.cand_cap[st] + 1) = t[0];
        b.n_rec[st * kLine] = t[0];
        if (t[0] > b.obj[st].cap) atomicOr(b.status, 1u << st);
    }
};

// triplets of segment s (Event.cc:524-597 via Triplet.cc:55): the segments
// starting at its outer mini-doublet; the multiplicity of the outer module in
// the connection list repeats each, as the reference's nested loops do
struct ScanTp : ScanJoined<kTP> {
    __device__ static void load(const BatchDev& b, int64_t s, bool in, int64_t* v) {
        v[0] = 0;
        if (!in) return;
        const int md = OJ(b, kSG, s);
        const int64_t n = join_n(b, md);
        if (n == 0) return;
        v[0] = n;
        // (a module-map segment's outer module is in the list, once unless the
        // list repeats modules)
        if (!b.seg_layers && !b.geo.conn_dup) return;
        const int g1 = OG(b, kSG, s);
        const int ev = ev_of(b, g1);
        v[0] = (int64_t)conn_mult(b, g1 - ev * b.geo.n_mod, OG(b, kMD, md) - ev * b.geo.n_mod) * n;
    }
};

// tracklets whose inner segment has the mini-doublets of segment s
__device__ __forceinline__ int64_t tl_join_n(const BatchDev& b, int s) {
    const int k = sg_key(b, s);
    return AT(b.joft, k + 1, b.obj[kSG].cap + 1) - AT(b.joft, k, b.obj[kSG].cap + 1);
}
// tracklet t into the index of tracklets by inner segment (joft scanned)
__device__ __forceinline__ void tl_join_place(const BatchDev& b, int64_t t) {
    const int64_t at = AT(b.joft, sg_key(b, OI(b, kTL, t)), b.obj[kSG].cap + 1);
    AT(b.jidt, at + AT(b.trank, t, b.obj[kTL].cap), b.obj[kTL].cap) = (int)t;
}

// track candidates of tracklet t (Event.cc:823-872 via TrackCandidate.cc:161):
// the tracklets whose inner segment matches its outer one; Event.cc:835: the
// candidates in the counters are barrel-layer-1 x barrel-layer-3 tracklets
struct ScanTc : ScanJoined<kTC> {
    __device__ static void begin(const BatchDev& b) {
        for (int ev = blockIdx.x * blockDim.x + threadIdx.x; ev < b.n_ev; ev += gridDim.x * blockDim.x) {
            const uint32_t n1 = *counter_at(b, ev, kTL, 1, 0), n3 = *counter_at(b, ev, kTL, 1, 2);
            *counter_at(b, ev, kTC, 0, 0) += n1 * n3;
        }
    }
    __device__ static void load(const BatchDev& b, int64_t t, bool in, int64_t* v) {
        v[0] = 0;
        if (!in) return;
        const ModDev& m1 = MOD(b, mod_of(b, OG(b, kTL, t)));
        if (m1.subdet != kBarrel) return;
        if (m1.layer == 3) tl_join_place(b, t);
        if (m1.layer != 1) return;
        const int sB = OJ(b, kTL, t);
        const ModDev& m3 = MOD(b, mod_of(b, OG(b, kSG, sB)));
        if (m3.subdet == kBarrel && m3.layer == 3) v[0] = tl_join_n(b, sB);
    }
};

// createTrackCandidatesFromTracklets (Event.cc:984-1062): the reference's
// candidates of tracklet t are the tracklets of the modules connected to the
// module of its inner segment's outer MD (conn_sum over tracklet counts); the
// matching ones are the tracklets whose inner segment matches t's outer
// segment, which all lie in the module of that segment's inner MD and come
// once per occurrence of that module in the connection list.  Layer-pair
// tracklets are listed by no module (Event.cc:785 via
// addTrackletToLowerLayer), so after them there are no candidates.
struct ScanTcFromTl : ScanJoined<kTC> {
    __device__ static void load(const BatchDev& b, int64_t t, bool in, int64_t* v) {
        const int n_mod = b.geo.n_mod;
        int64_t cref = 0;
        int ev = 0, slot = 0;
        v[0] = 0;
        if (in) tl_join_place(b, t);
        if (in && !(b.flags & kFlagTLLayers)) {
            const int gA2 = OG(b, kMD, OJ(b, kSG, OI(b, kTL, t)));
            ev = ev_of(b, gA2);
            cref = AT(b.conn_sum, gA2, b.n_gm);
            const int sB = OJ(b, kTL, t);
            v[0] = (int64_t)conn_mult(b, gA2 - ev * n_mod, OG(b, kMD, OI(b, kSG, sB)) - ev * n_mod) * tl_join_n(b, sB);
            slot = MOD(b, OG(b, kTL, t) - ev * n_mod).layer_slot;
        }
        const bool act = cref != 0;
        warp_add(act ? counter_at(b, ev, kTC, 0, slot) : b.counters, (uint32_t)cref, act);
    }
};

// createTrackCandidatesFromTriplets (Event.cc:874-982): the reference's
// candidates of triplet p are the triplets of the modules connected to the
// module of its outermost MD (conn_sum over triplet counts)
__device__ __forceinline__ int64_t tctp_cand(const BatchDev& b, int64_t p, bool in) {
    int64_t c = 0;
    if (in) c = AT(b.conn_sum, OG(b, kMD, OJ(b, kSG, OJ(b, kTP, p))), b.n_gm);
    count_cand(b, kTC, c ? OG(b, kTP, p) : 0, c);
    return c;
}
// each evaluated with its trial segment (k_tctp_trial, after layer-pair segments)
struct ScanTcTrial : ScanCand<kTC> {
    __device__ static void load(const BatchDev& b, int64_t p, bool in, int64_t* v) { v[0] = tctp_cand(b, p, in); }
};

// After module-map segments: the trial segment from p1's outermost MD mdA to
// p2's innermost MD passes the segment algorithm exactly when the segment
// stage made it, and it made it once per occurrence of p2's module in the
// connection list of mdA's module, which is also how often the reference's
// loop (over that list) reaches p2.  So p1's track candidates are the pairs of
// a segment sx leaving mdA and a triplet p2 starting at sx's outer MD whose
// tracklet (sx, p2's outer segment) passes the default tracklet algorithm --
// the same pairs for every triplet that ends in mdA.  Each pair is judged
// once (six or seven triplets end in a mini-doublet at PU 200), in the tracklet
// stage's steps: ScanTctp counts the pairs of every segment that leaves a
// triplet's end, k_tctp_a lists those through the single-precision phases A and
// B1, k_tctp_b decides phase B2 where its bounds allow and k_tctp_c evaluates
// the rest exactly; the pairs that pass are indexed by mdA and expanded.  (Three
// events of PU 100-200: the stage took 1.72 ms with the exact phases on every
// triplet's every pair, 0.15 ms now.)
struct ScanTctp : ScanCand<kTL> {
    __device__ static void load(const BatchDev& b, int64_t s, bool in, int64_t* v) {
        v[0] = in && AT(b.tpend, OI(b, kSG, s), b.obj[kMD].cap) ? join2_n(b, OJ(b, kSG, s)) : 0;
    }
};
__global__ void __launch_bounds__(kEnumThreads) k_tctp_a(BatchDev b) {
    __shared__ int4 pbuf[kEnumThreads / kWarp][kPassBuf];
    if (halted(b)) return;
    const int64_t nobj = n_objects(b, kSG);
    if (nobj <= 0) return;
    const int64_t* off = b.cand[kTL];
    const int64_t offlim = b.cand_cap[kTL] + 1, C = b.obj[kSG].cap;
    const int64_t total = AT(off, nobj, offlim);
    const int task = b.task_size[kTL];
    const int64_t ntask = (total + task - 1) / task;
    const int lane = threadIdx.x & 31;
    PassBuf pb{pbuf[threadIdx.x >> 5]};
    for (;;) {
        unsigned long long t = 0;
        if (lane == 0) t = atomicAdd(b.task + kTC * kLine, 1ull);
        t = __shfl_sync(0xffffffffu, t, 0);
        if ((int64_t)t >= ntask) break;
        const int64_t base = (int64_t)t * task;
        const int64_t end = min(base + task, total);
        int ilo = 0;
        if (lane < 2) {
            int lo, hi;
            obj_bounds(b, nobj, total, base, end - 1, lo, hi);
            ilo = find_obj(b, off, offlim, lo, hi, lane == 0 ? base : end - 1);
        }
        const int i0 = __shfl_sync(0xffffffffu, ilo, 0);
        const int i1 = __shfl_sync(0xffffffffu, ilo, 1);
        for (int64_t cb = base; cb < end; cb += kWarp) {
            const int64_t c = cb + lane;
            int algo = kAlgoNone, s = 0, tt = 0, b1 = 0, p2 = 0;
            if (c < end) {
                s = (i0 == i1) ? i0 : find_obj(b, off, offlim, i0, i1, c);
                p2 = join2_obj(b, OJ(b, kSG, s), c - AT(off, s, offlim));
                tt = OJ(b, kTP, p2);
                bool exact;
                algo = tl_ab1_decide<true>(tl_row(load_sgv(b.sgpack, s)), tl_out(load_sgo(b.sgouter, C, tt)), load_sgo_xy(b.sgouter, C, tt),
                                     b.sgpack, s, tt, b1, exact);
            }
            passbuf_put(b, pb, algo != kAlgoNone, make_int4(s, tt, algo | (b1 << 8), p2));
        }
    }
    passbuf_flush(b, pb);
}
// pairs through all phases: (p2, sx's inner MD, place among that MD's pairs)
// to the kept list, a warp at a time
__device__ __forceinline__ void tctp_pass(const BatchDev& b, bool pass, int s, int p2) {
    const unsigned m = __ballot_sync(0xffffffffu, pass);
    if (!m) return;
    const int lane = threadIdx.x & 31, leader = __ffs(m) - 1;
    unsigned long long p0 = 0;
    if (lane == leader) p0 = atomicAdd(b.n_tc_pass, (unsigned long long)__popc(m));
    p0 = __shfl_sync(0xffffffffu, p0, leader);
    if (!pass) return;
    const int64_t pos = (int64_t)p0 + __popc(m & ((1u << lane) - 1u));  // below the list's length <= kept_cap
    const int md = OI(b, kSG, s);
    const int rank = (int)atomicAdd((unsigned long long*)&AT(b.joff3, md, b.obj[kMD].cap + 1), 1ull);
    AT(b.kept, pos, b.kept_cap) = make_int4(p2, md, rank, 0);
}
__global__ void __launch_bounds__(kEnumThreads) k_tctp_b(BatchDev b) {
    __shared__ int4 pbuf[kEnumThreads / kWarp][kPassBuf];
    if (halted(b)) return;
    const int64_t n = min((int64_t)*b.n_tc_list, b.kept_cap);
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    // the undecided pairs go to the filtered list
    BatchDev u = b;
    u.passa = b.passf;
    u.n_kept = b.n_tc_open;
    PassBuf pb{pbuf[w]};
    const int64_t warps = (int64_t)gridDim.x * (kEnumThreads / kWarp);
    for (int64_t base = ((int64_t)blockIdx.x * (kEnumThreads / kWarp) + w) * kWarp; base < n; base += warps * kWarp) {
        int r = 0;
        int4 e = make_int4(0, 0, 0, 0);
        if (base + lane < n) {
            e = AT(b.pb, base + lane, b.kept_cap);
            r = tl_b2_quick<false>(e.z & 0xff, load_sgv(b.sgpack, e.x), load_sgv(b.sgpack, e.y));
            if (r == 3 && !(e.z >> 8)) r = 1;  // phase B1 undecided
        }
        tctp_pass(b, r == 3, e.x, e.w);
        passbuf_put(u, pb, r == 1, e);
    }
    passbuf_flush(u, pb);
}
__global__ void __launch_bounds__(kEnumThreads) k_tctp_c(BatchDev b) {
    if (halted(b)) return;
    const int64_t n = min((int64_t)*b.n_tc_open, b.kept_cap);
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int64_t warps = (int64_t)gridDim.x * (kEnumThreads / kWarp);
    const int per = entries_per_warp(n, warps);  // (3 events: 57 -> 25 us)
    for (int64_t base = ((int64_t)blockIdx.x * (kEnumThreads / kWarp) + w) * per; base < n; base += warps * per) {
        bool pass = false;
        int4 e = make_int4(0, 0, 0, 0);
        if (lane < per && base + lane < n) {
            e = AT(b.passf, base + lane, b.kept_cap);
            float cut, muls;
            const int algo = tl_phaseA(load_sgv(b.sgpack, e.x), load_sgv(b.sgpack, e.y), cut, muls);
            pass = algo != kAlgoNone && tl_phaseB1(algo, b.sgpack, e.x, e.y, cut) &&
                   tl_phaseB2<kB2All>(algo, b.sgpack, e.x, e.y, muls, false);
        }
        tctp_pass(b, pass, e.x, e.w);
    }
}
__global__ void k_tctp_place(BatchDev b) {
    if (halted(b)) return;
    const int64_t n = min((int64_t)*b.n_tc_pass, b.kept_cap);
    for (int64_t k = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; k < n; k += (int64_t)gridDim.x * blockDim.x) {
        const int4 e = AT(b.kept, k, b.kept_cap);
        AT(b.jidx3, AT(b.joff3, e.y, b.obj[kMD].cap + 1) + e.z, b.kept_cap) = e.x;
    }
}
// track candidates of triplet p: the passing pairs of its outermost MD
struct ScanTcFromTp : ScanJoined<kTC> {
    __device__ static void load(const BatchDev& b, int64_t p, bool in, int64_t* v) {
        (void)tctp_cand(b, p, in);
        v[0] = 0;
        if (!in) return;
        const int md = OJ(b, kSG, OJ(b, kTP, p));
        v[0] = AT(b.joff3, md + 1, b.obj[kMD].cap + 1) - AT(b.joff3, md, b.obj[kMD].cap + 1);
    }
};

// The triplets (st kTP) and track candidates (kTC) from their scanned counts:
// every candidate is an object and its offset its place, so there is nothing
// to evaluate, rank or regroup.  A warp takes 32 consecutive inner objects and
// writes their objects 32 at a time, coalesced; each lane finds the inner
// object of its output among the lanes' offsets.  blockIdx.y 1: the objects'
// offsets per module and the layer counters.  (64 events: the triplet stage 480 -> 142 us,
// the track-candidate stage 354 -> 166 us against enumerating, ranking and
// scattering.)
template <int st, bool kFromTp>
__global__ void __launch_bounds__(256) k_expand(BatchDev b) {
    if (halted(b)) return;
    constexpr int ist = st == kTP ? kSG : (kFromTp ? kTP : kTL);
    const int64_t* off = b.cand[st];
    const int64_t offlim = b.cand_cap[st] + 1;
    const int64_t n = n_inner(b, st);
    if (blockIdx.y == 1) {
        for (int64_t g = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; g - (threadIdx.x & 31) <= b.n_gm;
             g += (int64_t)gridDim.x * blockDim.x) {
            int64_t c = 0;
            if (g <= b.n_gm) {
                const int64_t o = AT(off, min(OFF(b, ist, g), n), offlim);
                AT(b.obj[st].mod_cnt, g, NG1(b)) = o;
                if (g < b.n_gm) c = AT(off, min(OFF(b, ist, g + 1), n), offlim) - o;
            }
            const bool act = c != 0;
            int ev = 0, slot = 0;
            if (act) {
                ev = ev_of(b, g);
                slot = MOD(b, g - (int64_t)ev * b.geo.n_mod).layer_slot;
            }
            warp_add(act ? counter_at(b, ev, st, 1, slot) : b.counters, (uint32_t)c, act);
        }
        return;
    }
    const Objs& O = b.obj[st];
    const int lane = threadIdx.x & 31;
    const int64_t warps = (int64_t)gridDim.x * (blockDim.x / kWarp);
    for (int64_t base = ((int64_t)blockIdx.x * (blockDim.x / kWarp) + (threadIdx.x >> 5)) * kWarp; base < n; base += warps * kWarp) {
        const int64_t i = base + lane;
        const int64_t e0 = AT(off, base, offlim);
        const int64_t mine = AT(off, min(i, n), offlim);
        const int total = (int)(AT(off, min(base + kWarp, n), offlim) - e0);  // (below the capacity, an int's range)
        const int lo = (int)(mine - e0);
        int64_t list = 0;
        int len = 0, g = 0;
        if (i < n && AT(off, i + 1, offlim) > mine) {
            g = OG(b, ist, i);
            if (st == kTP) {
                const int md = OJ(b, kSG, i);
                list = AT(b.joff, md, b.obj[kMD].cap + 1);
                len = (int)(AT(b.joff, md + 1, b.obj[kMD].cap + 1) - list);
            } else if (kFromTp) {
                const int md = OJ(b, kSG, OJ(b, kTP, i));
                list = AT(b.joff3, md, b.obj[kMD].cap + 1);
                len = (int)(AT(b.joff3, md + 1, b.obj[kMD].cap + 1) - list);
            } else {
                const int k = sg_key(b, OJ(b, kTL, i));
                list = AT(b.joft, k, b.obj[kSG].cap + 1);
                len = (int)(AT(b.joft, k + 1, b.obj[kSG].cap + 1) - list);
            }
        }
        for (int t0 = 0; t0 < total; t0 += kWarp) {
            const int t = t0 + lane;
            int src = 0;  // the last lane with lo <= t
#pragma unroll
            for (int o = 16; o; o >>= 1) {
                const int x = __shfl_sync(0xffffffffu, lo, src + o);
                if (x <= t) src += o;
            }
            const int q = t - __shfl_sync(0xffffffffu, lo, src);
            const int64_t l = __shfl_sync(0xffffffffu, list, src);
            const int m = __shfl_sync(0xffffffffu, len, src);
            const int gs = __shfl_sync(0xffffffffu, g, src);
            if (t < total) {
                const int64_t pos = e0 + t;
                const int64_t k = l + (q < m ? q : q % m);
                AT(O.i, pos, O.cap) = (int)base + src;
                AT(O.j, pos, O.cap) = st == kTP ? AT(b.jidx, k, b.obj[kSG].cap)
                                                : (kFromTp ? AT(b.jidx3, k, b.kept_cap) : AT(b.jidt, k, b.obj[kTL].cap));
                AT(O.g, pos, O.cap) = gs;
            }
        }
    }
}

// ------------------------------------------------------------------ output
__device__ __forceinline__ void put_md(const BatchDev& b, int a, int32_t* o) {
    o[0] = AT(b.hidx, OI(b, kMD, a), H(b));
    o[1] = AT(b.hidx, OJ(b, kMD, a), H(b));
}
__device__ __forceinline__ void put_sg(const BatchDev& b, int s, int32_t* o) {
    put_md(b, OI(b, kSG, s), o);
    put_md(b, OJ(b, kSG, s), o + 2);
}
__device__ __forceinline__ void put_tl(const BatchDev& b, int st, int t, int32_t* o) {
    put_sg(b, OI(b, st, t), o);
    put_sg(b, OJ(b, st, t), o + 4);
}

// one row of W hit indices, built in registers, stored with 8- or 16-byte
// stores when the output is 16-byte aligned
template <int W>
__device__ __forceinline__ void store_row(int32_t* o, const int32_t* v, bool vec) {
    if (vec) {
        if constexpr (W == 2) {
            *reinterpret_cast<int2*>(o) = make_int2(v[0], v[1]);
        } else {
#pragma unroll
            for (int i = 0; i < W; i += 4) *reinterpret_cast<int4*>(o + i) = make_int4(v[i], v[i + 1], v[i + 2], v[i + 3]);
        }
    } else {
#pragma unroll
        for (int i = 0; i < W; ++i) o[i] = v[i];
    }
}

template <int kSt>
__global__ void k_materialize(BatchDev b, int64_t first, int64_t n, int32_t* out) {
    constexpr int W = kSt == kMD ? 2 : kSt == kSG ? 4 : kSt == kTC ? 16 : 8;
    const bool vec = (reinterpret_cast<uintptr_t>(out) & 15) == 0;
    const int ist = (b.flags & kFlagTCFromTP) ? kTP : kTL;  // track candidates: two tracklets or two triplets
    for (int64_t k = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; k < n; k += (int64_t)gridDim.x * blockDim.x) {
        const int o = (int)(first + k);
        int32_t v[W];
        if constexpr (kSt == kMD) {
            put_md(b, o, v);
        } else if constexpr (kSt == kSG) {
            put_sg(b, o, v);
        } else if constexpr (kSt == kTC) {
            put_tl(b, ist, OI(b, kTC, o), v);
            put_tl(b, ist, OJ(b, kTC, o), v + 8);
        } else {
            put_tl(b, kSt, o, v);
        }
        store_row<W>(out + (int64_t)W * k, v, vec);
    }
}

// The object graph of stage st for objects [first, first + n) of one event:
// constituents as indices into the event's lists of the stage below (hits:
// their position in the event's input order), the inner lower module within
// the event, and the floats the stage keeps per object.  lo_first: the
// event's first object of the stage below (its first input hit for
// mini-doublets); gm0: the event's first global module.
__global__ void k_links(BatchDev b, int st, int64_t first, int64_t n, int64_t lo_first, int64_t gm0, int32_t* links,
                        int32_t* module, float* vals) {
    const int nf = b.obj[st].nf;
    for (int64_t k = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; k < n; k += (int64_t)gridDim.x * blockDim.x) {
        const int64_t o = first + k;
        int64_t a = OI(b, st, o), c = OJ(b, st, o);
        if (st == kMD) {  // sorted hit positions -> input hits
            a = AT(b.hit_perm, a, H(b));
            c = AT(b.hit_perm, c, H(b));
        }
        if (links) {
            links[2 * k] = (int32_t)(a - lo_first);
            links[2 * k + 1] = (int32_t)(c - lo_first);
        }
        if (module) module[k] = (int32_t)(OG(b, st, o) - gm0);
        if (vals)
            for (int f = 0; f < nf; ++f) vals[k * nf + f] = OF(b, st, f, o);
    }
}

// the host libm's float functions as the chain evaluates them, on the float
// bit patterns start .. start + n - 1 (the self-check of the libm tables)
__global__ void k_libm_eval(int fn, uint32_t start, int64_t n, float* out) {
    for (int64_t k = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; k < n; k += (int64_t)gridDim.x * blockDim.x) {
        const float x = __uint_as_float(start + (uint32_t)k);
        float v;
        switch (fn) {
            case kLmAsin: v = g_asin(x); break;
            case kLmAtan: v = g_atan(x); break;
            case kLmSin: v = g_sin(x); break;
            case kLmCos: v = g_cos(x); break;
            default: v = g_tan(x); break;
        }
        out[k] = v;
    }
}

unsigned grid_for(int64_t n, int threads, int cap_blocks) {
    int64_t g = (n + threads - 1) / threads;
    if (g < 1) g = 1;
    if (g > cap_blocks) g = cap_blocks;
    return (unsigned)g;
}

// the argument of the next launch: b with the stamps set since the last
// one, which this launch takes
BatchDev take(const BatchDev& b, Hooks* h) {
    BatchDev c = b;
    c.ts = 0;
    if (h) {
        c.ts = h->ts;
        h->ts = 0;
        h->launches += 1;
    }
    return c;
}
inline void mark(Hooks* h, int s) {
    if (h) h->ts |= stamp_bit(s);
}

__global__ void __launch_bounds__(256) k_clear(BatchDev b, ClearJobs j) {
    if (b.ts && blockIdx.x == 0 && blockIdx.y == 0 && threadIdx.x == 0)
        for (int k = 0; k < j.stamps; ++k) b.stamps[k] = 0ull;
    stamp(b);
    const int q = blockIdx.y;
    const int64_t w = j.words[q], n = w * j.rows[q];
    uint32_t* p = j.p[q];
    const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x, stride = (int64_t)gridDim.x * blockDim.x;
    if (j.rows[q] > 1) {
        for (int64_t i = t; i < n; i += stride) p[i / w * j.pitch[q] + i % w] = 0u;
        return;
    }
    int64_t done = 0;
    if ((reinterpret_cast<uintptr_t>(p) & 15u) == 0) {
        for (int64_t i = t; i < n / 4; i += stride) reinterpret_cast<uint4*>(p)[i] = make_uint4(0u, 0u, 0u, 0u);
        done = n / 4 * 4;
    }
    for (int64_t i = done + t; i < n; i += stride) p[i] = 0u;
}

__global__ void __launch_bounds__(256) k_finish(BatchDev b, int64_t* host) {
    stamp(b);
    const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x, stride = (int64_t)gridDim.x * blockDim.x;
    if (t < kNumStages) host[kRunRec + t] = b.n_rec[t * kLine];
    if (t == kNumStages) host[kRunStatus] = (int64_t)*b.status;
    if (t == kNumStages + 1) host[kRunKept] = (int64_t)max(max(*b.n_kept, *b.n_kept_sg), *b.n_tc_list);
    // (this kernel's own stamp is written by the thread that copies it)
    if (blockIdx.x == 0 && threadIdx.x == 0)
        for (int k = 0; k < kNumStamps; ++k) host[kRunStamps + k] = (int64_t)b.stamps[k];
    const int64_t per = b.n_ev + 1;
    for (int64_t i = t; i < kNumStages * per; i += stride) {
        const int st = (int)(i / per);
        host[kRunOffsets + i] = b.obj[st].mod_cnt[(i - st * per) * b.geo.n_mod];
    }
    uint32_t* c = reinterpret_cast<uint32_t*>(host + kRunOffsets + kNumStages * per);
    for (int64_t i = t; i < (int64_t)b.n_ev * 110; i += stride) c[i] = b.counters[i];
}

// n: about the number of elements (the grid loops over the tiles).  A round of tiles (about 300
// CTAs in flight) takes around ten microseconds whatever its size, so the
// tiles are large where there would be several rounds of small ones (objects
// per module of 64 events, 2.2M modules: 46 us at 4 per thread, 35 at 8; of
// one event, 22k modules: 11 us at 4, 8 at 1).  The connection sums of many
// modules are a kernel of their own for the same reason (64 events: 62 + 43 us
// against 300 us within the scan; one event: 15 us within it).
constexpr int64_t kScanSmall = (int64_t)1 << 18;
// an object array's capacity is about three times what a batch that fills the
// hits' capacity puts there
inline int64_t objects_about(const BatchDev& b, int64_t cap) {
    return b.hits_about == b.n_hit_cap ? cap / 3 : (int64_t)((double)cap / 3 * (double)b.hits_about / (double)b.n_hit_cap);
}
template <class Op>
void scan(const BatchDev& b, int slot, int64_t n, cudaStream_t s, Hooks* h) {
    const int items = n <= kScanSmall ? Op::kSmall : Op::kBig;
    auto* k = n <= kScanSmall ? k_scan<Op, Op::kSmall> : k_scan<Op, Op::kBig>;
    k<<<grid_for(n, kScanThreads * items, b.n_sm * 4), kScanThreads, 0, s>>>(take(b, h), slot);
}

int enum_grid(const BatchDev& b, int st) { return b.enum_grid[st] > 0 ? b.enum_grid[st] : kGridDefault; }

// The two parts of a list: one kernel for both where neither fills the GPU
// (one PU 200 event: segments 106 -> 100 us, phase-B2 filter 66 -> 60), one
// after the other where each does and the other part's code would only take
// room in the instruction caches (128 dense events: segments 7.15 ms apart,
// 7.30 together).
void launch_pair(const BatchDev& b, void (*both)(BatchDev), void (*one)(BatchDev), void (*two)(BatchDev), int grid,
                 cudaStream_t s, Hooks* h) {
    if (b.hits_about <= kSmallBatch) {
        both<<<dim3((unsigned)grid, 2), kEnumThreads, 0, s>>>(take(b, h));
    } else {
        one<<<grid, kEnumThreads, 0, s>>>(take(b, h));
        two<<<grid, kEnumThreads, 0, s>>>(take(b, h));
    }
}

template <int st>
void scatter(const BatchDev& b, cudaStream_t s, Hooks* h) {
    if (st == kTL && b.last >= kTC) k_scatter<st, st == kTL><<<b.n_sm * 8, 256, 0, s>>>(take(b, h));
    else k_scatter<st, false><<<b.n_sm * 8, 256, 0, s>>>(take(b, h));
}

// triplets or track candidates: counts scanned by Count -> objects
template <int st, class Count, bool kFromTp = false>
void expand(const BatchDev& b, cudaStream_t s, Hooks* h) {
    scan<Count>(b, kScanCand + st, objects_about(b, b.cand_cap[st]), s, h);
    if (!kFromTp) mark(h, kStampEnum + st);
    k_expand<st, kFromTp><<<dim3((unsigned)b.n_sm * 8, 2), 256, 0, s>>>(take(b, h));
    mark(h, kStampEnumEnd + st);
}

// device-to-device copies of 4-byte words (job blockIdx.y), 16 bytes at a
// time where both buffers are 16-byte aligned
__global__ void __launch_bounds__(256) k_copy_words(CopyJobs j) {
    const int q = blockIdx.y;
    if (q >= j.count) return;
    const uint32_t* __restrict__ src = j.src[q];
    uint32_t* __restrict__ dst = j.dst[q];
    const int64_t n = j.n[q];
    const int64_t stride = (int64_t)gridDim.x * blockDim.x;
    const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    int64_t done = 0;
    if (((reinterpret_cast<uintptr_t>(src) | reinterpret_cast<uintptr_t>(dst)) & 15u) == 0) {
        const int64_t n4 = n / 4;
        const uint4* s4 = reinterpret_cast<const uint4*>(src);
        uint4* d4 = reinterpret_cast<uint4*>(dst);
        for (int64_t i = t; i < n4; i += stride) d4[i] = __ldg(s4 + i);
        done = n4 * 4;
    }
    for (int64_t i = done + t; i < n; i += stride) dst[i] = __ldg(src + i);
}

}  // namespace

void launch_ingest(const BatchDev& b, cudaStream_t s, Hooks* h) {
    const unsigned g = grid_for(b.hits_about, 256, b.n_sm * 16);
    k_hit_map<<<g, 256, 0, s>>>(take(b, h));
    scan<ScanHits>(b, kScanHit, b.n_gm, s, h);
    k_hit_perm<<<g, 256, 0, s>>>(take(b, h));
    k_hit_scatter<<<dim3(g, 2), 256, 0, s>>>(take(b, h));
}

void launch_md(const BatchDev& b, cudaStream_t s, Hooks* h) {
    scan<ScanMdCand>(b, kScanCand + kMD, b.n_gm, s, h);
    mark(h, kStampEnum + kMD);
    k_md_enum<<<b.n_sm * enum_grid(b, kMD), kEnumThreads, 0, s>>>(take(b, h));
    mark(h, kStampEnumEnd + kMD);
    scan<ScanObj<kMD, true>>(b, kScanObj + kMD, b.n_gm, s, h);
    scatter<kMD>(b, s, h);
}

void launch_sg(const BatchDev& b, cudaStream_t s, Hooks* h) {
    k_md_pack<<<dim3((unsigned)b.n_sm * 8, 2), 256, 0, s>>>(take(b, h));
    const bool layers = (b.flags & kFlagSGLayers) != 0;
    if (layers) {
        k_layer_runs<<<grid_for((int64_t)b.n_ev * kNumSlots, 64, b.n_sm), 64, 0, s>>>(take(b, h));
        scan<ScanSgLayers>(b, kScanCand + kSG, objects_about(b, b.cand_cap[kSG]), s, h);
    } else if (b.n_gm <= kScanSmall) {
        scan<ScanSgFront<true>>(b, kScanCand + kSG, b.n_gm, s, h);
    } else {
        k_conn_sum<true><<<grid_for(b.n_gm, 256, b.n_sm * 32), 256, 0, s>>>(take(b, h), kMD, kSG, false);
        scan<ScanSgFront<false>>(b, kScanCand + kSG, b.n_gm, s, h);
    }
    if (!layers) k_sg_lists<<<grid_for(8 * (int64_t)b.n_gm, 256, b.n_sm * 32), 256, 0, s>>>(take(b, h));
    // first cuts -> survivor list -> whole algorithm (k_sg_enum_a, k_sg_b)
    mark(h, kStampEnum + kSG);
    BatchDev l = b;  // with this list's own counts
    l.n_kept = b.n_kept_sg;
    l.n_pb = b.n_pb_sg;
    auto* enum_a = !layers ? k_sg_enum_a<0> : b.layer_width == kLayerRuns ? k_sg_enum_a<1> : k_sg_enum_a<2>;
    enum_a<<<b.n_sm * enum_grid(b, kSG), kEnumThreads, 0, s>>>(take(l, h));
    launch_pair(l, k_sg_b<0>, k_sg_b<1>, k_sg_b<2>, b.n_sm * enum_grid(b, kSG), s, h);
    mark(h, kStampEnumEnd + kSG);
    // (Event.cc:793-821, the layer pairs, increments no per-layer counter)
    if (layers) scan<ScanObj<kSG, false>>(b, kScanObj + kSG, b.n_gm, s, h);
    else scan<ScanObj<kSG, true>>(b, kScanObj + kSG, b.n_gm, s, h);
    scatter<kSG>(b, s, h);
}

void launch_tl(const BatchDev& b, cudaStream_t s, Hooks* h) {
    // conn sums over segment counts serve the tracklet enumeration and the
    // triplet candidate counters (Event.cc:547-596 loops over the same lists)
    k_sg_pack<<<b.n_sm * 8, 256, 0, s>>>(take(b, h));
    // module-map candidates: the module-pair tiles (k_tl_enum_tiles)
    const bool tiles = !(b.flags & (kFlagTLLayers | kFlagTLNav));
    const unsigned gconn = grid_for(b.n_gm, 256, b.n_sm * 32);
    if (!tiles) {
        k_conn_sum<true><<<gconn, 256, 0, s>>>(take(b, h), kSG, kTP, false);
    } else if (b.n_gm <= kScanSmall) {
        scan<ScanTlFront<true>>(b, kScanTlFront, b.n_gm, s, h);
    } else {
        k_conn_sum<true><<<gconn, 256, 0, s>>>(take(b, h), kSG, kTP, true);
        scan<ScanTlFront<false>>(b, kScanTlFront, b.n_gm, s, h);
    }
    // the segments by inner mini-doublet, for navigation and the triplets
    scan<ScanJoin<0>>(b, kScanJoinSg, objects_about(b, b.obj[kMD].cap), s, h);
    k_sg_index<<<b.n_sm * 8, 256, 0, s>>>(take(b, h));
    if (b.geo.conn_dup) k_sg_keys<<<b.n_sm * 8, 256, 0, s>>>(take(b, h));
    if (!tiles) scan<ScanTlCand<true>>(b, kScanCand + kTL, objects_about(b, b.cand_cap[kTL]), s, h);
    mark(h, kStampEnum + kTL);
    // enumeration + phase A -> survivor list (-> the pre-filter -> kept list)
    // -> phase B1 -> phase B2
    if (tiles) k_tl_enum_tiles<<<b.n_sm * enum_grid(b, kTL), kEnumThreads, 0, s>>>(take(b, h));
    else k_tl_enum_a<<<b.n_sm * enum_grid(b, kTL), kEnumThreads, 0, s>>>(take(b, h));
    mark(h, kStampTlMid + 0);
    // the list phase B1 reads: the enumeration's, the pre-filter's kept
    // entries, then what phase B2's single-precision filter leaves of it (not
    // with DefaultNm1, whose phase B2 keeps what fails the deltaBeta cut)
    int4* list = b.passa;
    unsigned long long* count = b.n_kept;
    const bool mlp = (b.flags & kFlagMLP) != 0;
    if (mlp) {
        k_tl_prefilter<<<b.n_sm * kPfCtasPerSm, kMlpTile, 0, s>>>(take(b, h));
        list = b.kept;
        count = b.n_kept2;
    }
    mark(h, kStampTlMid + 1);
    const bool filt = !(b.flags & (kFlagTLNm1 | kFlagNoB2Filter));
    if (filt) {
        BatchDev l = b;  // with the deferred entries' own counts
        l.n_pb = b.n_pb_f;
        auto* first = mlp ? k_tl_b2f<false> : k_tl_b2f<true>;
        first<<<b.n_sm * enum_grid(b, kTL), kEnumThreads, 0, s>>>(take(l, h), list, count);
        launch_pair(l, k_tl_b2f_rest<0>, k_tl_b2f_rest<1>, k_tl_b2f_rest<2>, b.n_sm * enum_grid(b, kTL), s, h);
        list = b.passf;
        count = b.n_keptf;
    }
    mark(h, kStampTlMid + 2);
    k_tl_b1<<<b.n_sm * enum_grid(b, kTL), kEnumThreads, 0, s>>>(take(b, h), list, count);
    k_tl_b2<<<dim3((unsigned)(b.n_sm * enum_grid(b, kTL)), 2), kEnumThreads, 0, s>>>(take(b, h));
    mark(h, kStampEnumEnd + kTL);
    scan<ScanObj<kTL, true>>(b, kScanObj + kTL, b.n_gm, s, h);
    scatter<kTL>(b, s, h);
}


void launch_tp(const BatchDev& b, cudaStream_t s, Hooks* h) { expand<kTP, ScanTp>(b, s, h); }

void launch_tc(const BatchDev& b, cudaStream_t s, Hooks* h) {
    if (b.flags & kFlagTCFromTP) {
        const unsigned gconn = grid_for(b.n_gm, 256, b.n_sm * 32);
        k_conn_sum<false><<<gconn, 256, 0, s>>>(take(b, h), kTP, -1, false);
        if (b.flags & kFlagSGLayers) {
            scan<ScanTcTrial>(b, kScanCand + kTC, objects_about(b, b.cand_cap[kTC]), s, h);
            mark(h, kStampEnum + kTC);
            k_tctp_trial<<<b.n_sm * enum_grid(b, kTC), kEnumThreads, 0, s>>>(take(b, h));
            mark(h, kStampEnumEnd + kTC);
            scan<ScanObj<kTC, true>>(b, kScanObj + kTC, b.n_gm, s, h);
            scatter<kTC>(b, s, h);
            return;
        }
        ClearJobs j{};
        j.add(b.joff2, 2 * (b.obj[kMD].cap + 1));
        j.add(b.jcur2, b.obj[kMD].cap);
        j.add(b.tpend, b.obj[kMD].cap);
        j.add(b.joff3, 2 * (b.obj[kMD].cap + 1));
        static_assert(kClearJobs >= 4, "the jobs fit");
        (void)launch_clear(b, j, s, h);
        const unsigned g = b.n_sm * 8, ge = b.n_sm * enum_grid(b, kTL);
        k_join2_count<<<g, 256, 0, s>>>(take(b, h));
        scan<ScanJoin<1>>(b, kScanJoinTc, objects_about(b, b.obj[kMD].cap), s, h);
        k_join2_scatter<<<g, 256, 0, s>>>(take(b, h));
        scan<ScanTctp>(b, kScanTctp, objects_about(b, b.cand_cap[kTL]), s, h);
        mark(h, kStampEnum + kTC);
        BatchDev l = b;  // the pairs' list is the tracklets' spare one, with a count of its own
        l.passa = b.pb;
        l.n_kept = b.n_tc_list;
        k_tctp_a<<<ge, kEnumThreads, 0, s>>>(take(l, h));
        k_tctp_b<<<ge, kEnumThreads, 0, s>>>(take(b, h));
        k_tctp_c<<<ge, kEnumThreads, 0, s>>>(take(b, h));
        scan<ScanJoin<3>>(b, kScanTctpJoin, objects_about(b, b.obj[kMD].cap), s, h);
        k_tctp_place<<<g, 256, 0, s>>>(take(b, h));
        expand<kTC, ScanTcFromTp, true>(b, s, h);
        return;
    }
    // the tracklets by inner segment
    if (b.first > kTL) k_tl_join_count<<<b.n_sm * 8, 256, 0, s>>>(take(b, h));  // (else in k_scatter)
    scan<ScanJoin<2>>(b, kScanJoinTc, objects_about(b, b.obj[kSG].cap), s, h);
    if (b.flags & kFlagTCFromTL) {
        k_conn_sum<false><<<grid_for(b.n_gm, 256, b.n_sm * 32), 256, 0, s>>>(take(b, h), kTL, -1, false);
        expand<kTC, ScanTcFromTl>(b, s, h);
    } else {
        expand<kTC, ScanTc>(b, s, h);
    }
}

// ------------------------------------------------------------------ self-check
// The float-float fast paths of the cut arithmetic against the double
// evaluation they stand for: every input whose fast path succeeds must give
// the same float bit for bit.  Inputs are either all float bit patterns of a
// range (unary functions) or hashed pseudo-random values.
__device__ __forceinline__ float hash_log(unsigned long long h, float lo_exp, float hi_exp) {
    const float u = (float)((h >> 11) & 0xffffffull) * (1.f / 16777216.f);
    const float m = 1.f + (float)((h >> 35) & 0x7fffffull) * (1.f / 8388608.f);
    return ldexpf(m, (int)floorf(lo_exp + u * (hi_exp - lo_exp)));
}
__device__ __forceinline__ unsigned long long mix64(unsigned long long z) {
    z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
    z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
    return z ^ (z >> 31);
}

__global__ void k_math_check(int fn, int exhaustive, unsigned long long start, long long n, unsigned long long seed,
                             unsigned long long* out) {
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
        float a = 0.f, b = 0.f, c = 0.f, d = 0.f;
        if (exhaustive) {
            a = __uint_as_float((unsigned)(start + (unsigned long long)i));
        } else {
            const unsigned long long h1 = mix64(seed * 0x9E3779B97F4A7C15ull + (unsigned long long)i);
            const unsigned long long h2 = mix64(h1 + 0x632BE59BD9B4E019ull);
            const unsigned long long h3 = mix64(h2 + 0x632BE59BD9B4E019ull);
            const unsigned long long h4 = mix64(h3 + 0x632BE59BD9B4E019ull);
            const float sa = (h1 & 1) ? -1.f : 1.f, sb = (h2 & 1) ? -1.f : 1.f;
            switch (fn) {
                case 1: case 2: case 16: case 20:  // coordinates: magnitudes 2^-12..2^9, a fraction on axes and diagonals
                    a = sa * hash_log(h1, -12.f, 9.f);
                    b = sb * hash_log(h2, -12.f, 9.f);
                    if ((h3 & 15) == 0) b = sb * fabsf(a) * (1.f + (float)((h4 >> 40) & 0xff) * 0x1p-20f);
                    if ((h3 & 15) == 1) b = a * 0x1p-20f;
                    break;
                case 3:
                    a = sa * hash_log(h1, -20.f, 4.f);
                    b = hash_log(h2, -40.f, 6.f);
                    break;
                case 7:  // (dr k, beta): |beta| below 0.5
                    a = hash_log(h1, -8.f, 1.f);
                    b = sa * hash_log(h2, -24.f, -1.f);
                    break;
                case 8: case 15:  // (rtOut - rtIn, r3/rt)
                    a = hash_log(h1, -10.f, 8.f);
                    b = 1.f + hash_log(h2, -12.f, 2.f);
                    break;
                case 9:  // (head, t)
                    a = hash_log(h1, -30.f, 2.f);
                    b = hash_log(h2, -16.f, 2.f);
                    break;
                case 13:  // coordinate differences
                    a = sa * hash_log(h1, -12.f, 8.f);
                    b = sb * hash_log(h2, -12.f, 8.f);
                    break;
                case 14:  // (dphi, dz)
                    a = sa * hash_log(h1, -24.f, 1.f);
                    b = sb * hash_log(h2, -8.f, 4.f);
                    break;
                case 4:
                    a = hash_log(h1, -10.f, 1.f);
                    b = hash_log(h2, -14.f, 1.f);
                    c = hash_log(h3, -14.f, 1.f);
                    d = (h4 & 3) == 0 ? 0.f : hash_log(h4, -14.f, 3.f);
                    break;
                default:
                    a = sa * hash_log(h1, -30.f, 0.f);
            }
        }
        float f = 0.f, ref = 0.f;
        bool ok = false;
        switch (fn) {
            case 0: ok = f_asin_fast(a, f); if (ok) ref = f_asin_d(a); break;
            case 1: ok = atan2_fast(a, b, f); if (ok) ref = atan2_d(a, b); break;
            case 2: {
                f = phi_of(a, b);
                ref = phi_of_d(a, b);
                ok = true;
                break;
            }
            case 3: ok = add_dsqrt_fast(a, b, f); if (ok) ref = add_dsqrt_d(a, b); break;
            case 4: ok = add_dsqrt3_fast(a, b, c, d, f); if (ok) ref = add_dsqrt3_d(a, b, c, d); break;
            case 5: ok = phi_mpi_pi_fast(a, f); if (ok) ref = phi_mpi_pi_d(a); break;
            case 6: ok = add_pi_fast(a, f); if (ok) ref = (float)(kPi + (double)a); break;
            case 7: ok = pt_from_fast(a, b, f); if (ok) ref = pt_from_d(a, b); break;
            case 8: ok = muls_fast(a, b, true, f); if (ok) ref = muls_d(a, b, true); break;
            case 9: ok = add_quarter_sq_fast(a, b, f); if (ok) ref = add_quarter_sq_d(a, b); break;
            case 10: ok = f_sincos_fast(a, 0, f); if (ok) ref = f_sin_d(a); break;
            case 11: ok = f_sincos_fast(a, 1, f); if (ok) ref = f_cos_d(a); break;
            case 12: ok = f_atan_fast(a, f); if (ok) ref = f_atan_d(a); break;
            case 13: ok = hypot_fast(a, b, f); if (ok) ref = hypot_d(a, b); break;
            case 14: ok = times15_over_fast(a, b, f); if (ok) ref = times15_over_d(a, b); break;
            case 15: ok = muls_fast(a, b, false, f); if (ok) ref = muls_d(a, b, false); break;
            case 16: ok = phi_approx(a, b, f); if (ok) ref = phi_of(a, b); break;
            case 17: ok = fabsf(a) <= kSinAlphaMax; if (ok) { f = asinf(a); ref = f_asin(a); } break;
            case 18: ok = f_tan_fast(a, false, f); if (ok) ref = f_tan(a); break;
            case 19: ok = f_tan_fast(a, true, f); if (ok) ref = f_tan_over_d(a); break;
            case 20: ok = phi_fast(a, b, f); if (ok) ref = phi_of(a, b); break;
            default: break;
        }
        // functions 16, 17 and 20 are the approximations of phase B1: within
        // 2e-6 (16, 17) and 2.5e-6 (20) of the exact value (directions compared
        // modulo 2 pi); the others must match the double evaluation bit for bit
        const bool approx = fn == 16 || fn == 17 || fn == 20;
        const float tol = fn == 20 ? 2.5e-6f : 2e-6f;
        const bool bad = approx ? ok && !(fabsf(fn == 17 ? f - ref : wrap_approx(f - ref)) <= tol)
                                : ok && __float_as_uint(f) != __float_as_uint(ref) && !(isnan(f) && isnan(ref));
        const unsigned m_ok = __ballot_sync(__activemask(), ok);
        const unsigned m_bad = __ballot_sync(__activemask(), bad);
        if ((threadIdx.x & 31) == 0) {
            atomicAdd(out + 0, (unsigned long long)__popc(m_ok));
            if (m_bad) atomicAdd(out + 1, (unsigned long long)__popc(m_bad));
        }
        if (bad && atomicCAS(out + 2, 0ull, 1ull) == 0ull) {
            out[3] = __float_as_uint(a);
            out[4] = __float_as_uint(b);
            out[5] = __float_as_uint(c);
            out[6] = __float_as_uint(f);
            out[7] = __float_as_uint(ref);
        }
    }
}

void launch_math_check(int fn, int exhaustive, unsigned long long start, long long n, unsigned long long seed,
                       unsigned long long* out, int n_sm, cudaStream_t s) {
    k_math_check<<<n_sm * 16, 256, 0, s>>>(fn, exhaustive, start, n, seed, out);
}

// the tracklet candidates as a flat space, after a run: the module map's
// enumeration needs none, the bucket table holds the last stage's, and the
// connection sums may be those over tracklets or triplets
// (createTrackCandidatesFromTracklets / FromTriplets)
static void tl_cand_space(const BatchDev& b, cudaStream_t s) {
    if (!(b.flags & (kFlagTLLayers | kFlagTLNav)))
        k_conn_sum<false><<<grid_for(b.n_gm, 256, b.n_sm * 32), 256, 0, s>>>(b, kSG, -1, false);
    ClearJobs j{};
    j.add(b.scan_state + (int64_t)(kScanCand + kTL) * b.scan_cap, 2 * b.scan_cap);
    (void)launch_clear(b, j, s, nullptr);
    scan<ScanTlCand<false>>(b, kScanCand + kTL, objects_about(b, b.cand_cap[kTL]), s, nullptr);
}

void launch_tl_collect(const BatchDev& b, const MlpCollect& c, cudaStream_t s) {
    tl_cand_space(b, s);
    k_tl_collect<<<b.n_sm * 8, 256, 0, s>>>(b, c);
}

void launch_first_cuts_check(const BatchDev& b, unsigned long long* out, cudaStream_t s) {
    // (the connection sums are those of a later stage)
    if (!b.seg_layers) k_conn_sum<false><<<grid_for(b.n_gm, 256, b.n_sm * 32), 256, 0, s>>>(b, kMD, -1, false);
    k_md_first_check<<<b.n_sm * 8, 256, 0, s>>>(b, out);
    k_sg_first_check<<<b.n_sm * 8, 256, 0, s>>>(b, out + 4);
}

void launch_tl_b2q_check(const BatchDev& b, unsigned long long* out, cudaStream_t s) {
    k_tl_b2q_check<<<b.n_sm * 8, 256, 0, s>>>(b, out);
}

void launch_tl_quick_check(const BatchDev& b, unsigned long long* out, cudaStream_t s) {
    tl_cand_space(b, s);
    k_tl_quick_check<<<b.n_sm * 8, 256, 0, s>>>(b, out);
}

// the final cut variables of tracklets [first, first + n) (kTLVarN floats
// each, NaN for a pair phase A does not accept): phase A for the algorithm
// and the factors, then phase B2 with its record.  The reference's BBEE
// algorithm records none of them (Tracklet.cc:1540-2016 only resets them to
// -999 at its start), so BBEE tracklets report -999 as the reference does.
__global__ void k_tl_vars(BatchDev b, int64_t first, int64_t n, float* out) {
    const bool nm1 = (b.flags & kFlagTLNm1) != 0;
    for (int64_t k = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; k < n; k += (int64_t)gridDim.x * blockDim.x) {
        const int64_t o = first + k;
        const SGV S = load_sgv(b.sgpack, OI(b, kTL, o));
        const SGV T = load_sgv(b.sgpack, OJ(b, kTL, o));
        float cut, muls, rec[kTLVarN];
#pragma unroll
        for (int j = 0; j < kTLVarN; ++j) rec[j] = __int_as_float(0x7fc00000);
        const int algo = tl_phaseA(S, T, cut, muls);
        if (algo == kAlgoBBEE) {
#pragma unroll
            for (int j = 0; j < kTLVarN; ++j) rec[j] = -999.f;
        } else if (algo != kAlgoNone) {
            (void)tl_phaseB2_sgv<kB2All>(algo, S, T, muls, nm1, rec);
        }
#pragma unroll
        for (int j = 0; j < kTLVarN; ++j) out[k * kTLVarN + j] = rec[j];
    }
}

void launch_tl_vars(const BatchDev& b, int64_t first, int64_t n, float* out, cudaStream_t s) {
    if (n <= 0) return;
    k_tl_vars<<<grid_for(n, 128, b.n_sm * 8), 128, 0, s>>>(b, first, n, out);
}

void launch_links(const BatchDev& b, int st, int64_t first, int64_t n, int64_t lo_first, int64_t gm0, int32_t* links,
                  int32_t* module, float* vals, cudaStream_t s) {
    if (n <= 0) return;
    k_links<<<grid_for(n, 256, b.n_sm * 16), 256, 0, s>>>(b, st, first, n, lo_first, gm0, links, module, vals);
}

cudaError_t set_libm_tables(const LibmTab* t) { return cudaMemcpyToSymbol(c_libm, t, sizeof(LibmTab) * kLmCount); }

void launch_libm_eval(int fn, uint32_t start, int64_t n, float* out, int n_sm, cudaStream_t s) {
    if (n <= 0) return;
    k_libm_eval<<<grid_for(n, 256, n_sm * 16), 256, 0, s>>>(fn, start, n, out);
}

cudaError_t launch_clear(const BatchDev& b, const ClearJobs& j, cudaStream_t s, Hooks* h) {
    if (j.full) return cudaErrorInvalidValue;
    int64_t most = 1;
    for (int k = 0; k < j.count; ++k) most = most > j.words[k] * j.rows[k] ? most : j.words[k] * j.rows[k];
    k_clear<<<dim3(grid_for((most + 3) / 4, 256, b.n_sm * 4), (unsigned)j.count), 256, 0, s>>>(take(b, h), j);
    return cudaSuccess;
}

void launch_finish(const BatchDev& b, int64_t* host, cudaStream_t s, Hooks* h) {
    k_finish<<<grid_for((int64_t)b.n_ev * 110, 256, b.n_sm), 256, 0, s>>>(take(b, h), host);
}

cudaError_t launch_copy_words(const CopyJobs& j, int n_sm, cudaStream_t s) {
    if (j.full) return cudaErrorInvalidValue;
    if (j.count <= 0) return cudaSuccess;
    k_copy_words<<<dim3((unsigned)(n_sm * 2), (unsigned)j.count), 256, 0, s>>>(j);
    return cudaSuccess;
}

void launch_materialize(const BatchDev& b, int st, int64_t first, int64_t n, int32_t* out, cudaStream_t s) {
    if (n <= 0) return;
    const unsigned g = grid_for(n, 256, b.n_sm * 16);
    switch (st) {
        case kMD: k_materialize<kMD><<<g, 256, 0, s>>>(b, first, n, out); break;
        case kSG: k_materialize<kSG><<<g, 256, 0, s>>>(b, first, n, out); break;
        case kTL: k_materialize<kTL><<<g, 256, 0, s>>>(b, first, n, out); break;
        case kTP: k_materialize<kTP><<<g, 256, 0, s>>>(b, first, n, out); break;
        default: k_materialize<kTC><<<g, 256, 0, s>>>(b, first, n, out);
    }
}

}  // namespace sdlg
