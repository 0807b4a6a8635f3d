// Launchers for the segment-linking kernels (sm_103a).  The host code in
// sdl_capi.cu owns the buffers and calls these in stage order on one stream.
#pragma once
#include <cuda_runtime.h>

#include "sdl_mlp.cuh"
#include "sdl_types.h"

namespace sdlg {

// Layer.cc:32-50: the outer layer slots paired with inner slot si (barrel
// layers 1-5 -> the next barrel layer and endcap layer 1; endcap 1 -> 2;
// endcap 2 -> 3, 4, 5; endcap 3 -> 4; endcap 4 -> 5); -1 past the last
__host__ __device__ inline int sg_layer_outer(int si, int k) {
    if (si <= 4) return k == 0 ? si + 1 : (k == 1 ? 6 : -1);
    if (si == 6) return k == 0 ? 7 : -1;
    if (si == 7) return k < 3 ? 8 + k : -1;
    if (si == 8 || si == 9) return k == 0 ? si + 1 : -1;
    return -1;
}

constexpr int kLayerRuns = 12;

constexpr int kTaskDefault = 256;  // candidates per warp task unless tuned
constexpr int kGridDefault = 8;    // CTAs per SM of an enumeration unless tuned

// Batches of up to so many hits take the launch shapes of small ones: tiles of
// 16 rows, both parts of a list in one launch, small scan tiles (each measured
// where it is chosen).
constexpr int64_t kSmallBatch = (int64_t)1 << 18;
// The hits that a batch's launch shapes are made for: the buffers' capacity,
// or, for a small batch in larger buffers (a context that once held a large
// batch), half the limit.  So two figures per set of buffers, and two graphs,
// serve any order of batches.
constexpr int64_t batch_hits(int64_t n_hit, int64_t cap) {
    return n_hit <= kSmallBatch && cap > kSmallBatch ? kSmallBatch / 2 : cap;
}

// Counters that kernels update atomically at the same time lie 256 bytes
// apart (8-byte words): atomics on one line take turns at its L2 slice.
constexpr int64_t kLine = 32;

struct BatchDev {
    Geometry geo;
    int n_ev;
    int n_gm;          // n_ev * n_mod
    int64_t n_hit_cap;
    int64_t hits_about;     // the hits that the launch shapes are made for (batch_hits)
    const int64_t* n_hit;   // device scalar
    // inputs (concatenated events)
    const float *in_x, *in_y, *in_z;
    const int32_t* in_idx;
    const uint32_t* in_det;
    const int64_t* ev_off;   // n_ev + 1
    // ingest
    int32_t* hit_gm;
    int32_t* hit_rank;
    int32_t* hit_perm;       // sorted position -> input hit
    int64_t* mod_hit;        // n_gm + 1: counts -> offsets
    // sorted hits (SoA)
    float *hx, *hy, *hz, *hrt, *hphi, *hr3, *ha1;
    float *hsx, *hsy, *hsz;  // the strip-shift anchor point of an anchoring hit (shift_anchor)
    int32_t *hidx, *hgm;
    // stages
    Objs obj[kNumStages];
    Recs rec[kNumStages];
    int64_t* cand[kNumStages];     // per inner object candidate counts -> offsets (cap_inner + 1)
    int64_t cand_cap[kNumStages];
    int64_t* n_rec;                // per stage (kLine apart): attempted appends
    // connection-list prefix sums of per-module object counts
    int32_t* conn_pref;            // n_ev * n_conn
    int32_t* conn_first;           // n_ev * n_conn: offset of the entry's module's first object
    int64_t* conn_sum;             // n_gm
    float* sgpack;                 // segment cap * PK_N packed records for the tracklet stage
    float* sgouter;                // segment cap * kSgOuter, one array per field: what the enumeration and the
                                   //   B2 filter read of an outer segment (lrt, lz, ltd, la1, uphi, flags,
                                   //   0.1/lrt: SGOuter; lx, ly, ux, uy: load_sgo_xy; alphaup, rtseg,
                                   //   urt - lrt: load_sgo_beta)
    float* sgfeat;                 // [kFeatN / 4][segment cap] 16-byte words: what the pre-filter reads of a segment
    float* mdpack;                 // mini-doublet cap * kMdPack: packed records for the segment stage
    float* mdbend;                 // mini-doublet cap * 2: tan over the asin angle, and the third-layer asin, of the anchor
    float* mdlite;                 // mini-doublet cap * kMdLite: what its first pass reads
    uint32_t* counters;            // n_ev * 110
    uint32_t* status;
    unsigned long long* task;      // per stage (kLine apart): work counter
    unsigned long long* scan_state;  // kScanSlots x scan_cap: per scan the tile counter and a word per tile and value
    int64_t scan_cap;
    int32_t* bucket;               // first inner object of every 256 consecutive candidates of the running stage
    int64_t bucket_cap;
    int flags;                     // kFlag* bits
    int first, last;               // the stages being enqueued
    bool seg_layers;               // the segments are (or will be) those of the layer pairs
    // launch shape of each stage's candidate-evaluation kernel (autotuned):
    // candidates per warp task (a multiple of 32) and CTAs per SM
    int enum_task[kNumStages];
    int enum_grid[kNumStages];
    int* task_size;                // per stage: candidates per warp task of this run (ScanCand)
    const unsigned char* mlp_pack; // packed pre-filter weights and threshold (kPackBytes)
    MlpStats* mlp_stats;           // pre-filter counts of the last run
    int4* passa;                   // tracklet candidates through phase A: (inner, outer, algorithm, 1 when
                                   //   phase B1 passed already, else 0)
    int64_t kept_cap;              // entries of each survivor list
    unsigned long long* n_kept;    // phase-A survivors found (can exceed kept_cap: overflow)
    int4* kept;                    // the phase-A survivors the pre-filter kept, as passa
    unsigned long long* n_kept2;
    int4* passf;                   // what phase B2's single-precision decision (tl_b2_quick) left of
                                   //   the enumeration's or the pre-filter's list, as passa
    unsigned long long* n_keptf;
    unsigned long long* n_cand_tl;   // tracklet candidates
    // join indices: the segments by their inner mini-doublet (navigation,
    // triplets), the triplets by theirs (createTrackCandidatesFromTriplets), the
    // tracklets by their inner segment (track candidates)
    int64_t* joff;                 // mini-doublet cap + 1: counts -> offsets
    int32_t* jrank;                // segment cap: place among its mini-doublet's
    int32_t* jidx;                 // segment cap: segment indices
    int64_t* joff2;                // mini-doublet cap + 1
    int32_t* jcur2;                // mini-doublet cap: fill cursors
    int32_t* jidx2;                // triplet cap
    // createTrackCandidatesFromTriplets: mini-doublets in which a triplet ends,
    // and the passing pairs by the segment's inner mini-doublet
    uint32_t* tpend;               // mini-doublet cap
    int64_t* joff3;                // mini-doublet cap + 1
    int32_t* jidx3;                // kept_cap: triplet indices
    unsigned long long* n_tc_list; // pairs through phases A and B1 (in pb; can exceed kept_cap: overflow)
    unsigned long long* n_tc_open; // of those, undecided in phase B2 (in passf)
    unsigned long long* n_tc_pass; // pairs through all phases (in kept)
    int64_t* joft;                 // segment cap + 1
    int32_t* trank;                // tracklet cap: place among its inner segment's
    int32_t* jidt;                 // tracklet cap: tracklet indices
    int32_t* sgkey;                // segment cap: first segment of the same mini-doublets (when geo.conn_dup)
    // module-pair tiles of the module-map tracklet candidates: the segments by
    // the global module of their outer mini-doublet, and the tiles per module
    int64_t* eoff;                 // n_gm + 1: counts -> offsets
    int32_t* erank;                // segment cap: place among its module's
    int32_t* eidx;                 // segment cap: segment indices
    int64_t* toff;                 // n_gm + 1: tile counts -> offsets
    int32_t* tile_gm;              // tile_cap: the global module of each tile (when the tiles fit)
    int64_t tile_cap;
    int* layer_runs;               // n_ev x kNumSlots rows of 2 * layer_width: the layer-pair segments' outer runs (k_layer_runs)
    int layer_width;               // the most outer runs of one inner layer slot, at least kLayerRuns
    int64_t* coff;                 // n_gm + 1: offsets of the modules' segment candidates
    int32_t* olist;                // olist_cap: the segment candidates' outer lists (k_sg_lists; offsets in toff)
    int64_t olist_cap;
    int4* pb;                      // candidates through phase B1: (inner, outer, algorithm, muls bits), BBBB
                                   //   from the front, the others from the back
    unsigned long long* n_pb;      // [2]: BBBB entries, other entries (kept_cap in all)
    // the segment first pass's counts (as n_kept, n_pb) and the B2 filter's
    // deferred entries (as n_pb): each use has its own, cleared with the rest
    // of the run's counts (launch_clear)
    unsigned long long* n_kept_sg;
    unsigned long long* n_pb_sg;
    unsigned long long* n_pb_f;
    int n_sm;
    unsigned long long* dbg;       // bounds-check record (debug builds): count, line, index, limit
    // device clock (%globaltimer, ns) at the start of chosen kernels: a
    // launch's ts is a mask of the stamps its first thread writes
    unsigned long long* stamps;    // kNumStamps
    uint32_t ts;
};

// The scans of a run, one slot of scan_state each (k_scan)
enum ScanSlot : int {
    kScanHit = 0,
    kScanCand = 1,                        // + st: candidate offsets (module-map segments: with the outer lists')
    kScanObj = kScanCand + kNumStages,    // + st: objects per module
    kScanTlFront = kScanObj + kNumStages,
    kScanJoinSg,
    kScanJoinTc,
    kScanTctp,
    kScanTctpJoin,
    kScanSlots
};
// words of one slot for scans over up to n_gm global modules (up to 3 values
// each) and objects, in tiles of at least 512
constexpr int64_t scan_words(int64_t n_gm, int64_t objects) {
    return 1 + (3 * (n_gm / 512 + 1) > objects / 512 + 1 ? 3 * (n_gm / 512 + 1) : objects / 512 + 1);
}

// Device time stamps of a run.  An event node in a CUDA graph costs about
// 4.5 us (a kernel node 0.8 us), so the stage and pass boundaries are stamps
// that the kernels behind them write; only the whole run is between events.
enum Stamp : int {
    kStampStart = 0,                                 // the run's first kernel
    kStampStage = 1,                                 // + st: the first kernel of stage st
    kStampEnd = kStampStage + kNumStages,            // the run's last kernel
    kStampEnum = kStampEnd + 1,                      // + st: stage st's candidate evaluation
    kStampEnumEnd = kStampEnum + kNumStages,         // + st: the kernel after it
    kStampTlMid = kStampEnumEnd + kNumStages,        // + 0..2: after phase A, after the pre-filter, after the B2 filter
    kNumStamps = kStampTlMid + 3
};
constexpr uint32_t stamp_bit(int s) { return 1u << s; }

// Host-side record of the launches: kernels launched, and the stamps the
// next one takes.
struct Hooks {
    int launches = 0;
    uint32_t ts = 0;
};

// Buffers set to zero at the start of a run (4-byte words; rows > 1: a
// column block of a matrix), all by one kernel: a memset node in a CUDA graph
// costs 4.6 us.
constexpr int kClearJobs = 24;  // (a run takes 18 at most)
struct ClearJobs {
    uint32_t* p[kClearJobs];
    int64_t words[kClearJobs];
    int64_t rows[kClearJobs];
    int64_t pitch[kClearJobs];
    int count;
    int stamps;  // the first so many stamps too
    bool full;   // a job did not fit: the launch is refused
    void add(void* q, int64_t n_words, int64_t n_rows = 1, int64_t n_pitch = 0) {
        if (count == kClearJobs) {
            full = true;
            return;
        }
        p[count] = static_cast<uint32_t*>(q);
        words[count] = n_words;
        rows[count] = n_rows;
        pitch[count++] = n_pitch;
    }
};
cudaError_t launch_clear(const BatchDev& b, const ClearJobs& j, cudaStream_t s, Hooks* h);

// What the host reads after a run, written by the run's last kernel to
// pinned memory (8-byte words): the appends attempted per stage, the status
// word, the longest survivor list, the stamps, the object offsets of every
// event (n_ev + 1 per stage), the per-layer counters (110 x n_ev 4-byte words).
enum RunWord : int {
    kRunRec = 0,
    kRunStatus = kNumStages,
    kRunKept = kNumStages + 1,
    kRunStamps = kNumStages + 2,
    kRunOffsets = kRunStamps + kNumStamps
};
constexpr int64_t run_words(int64_t n_ev) { return kRunOffsets + kNumStages * (n_ev + 1) + 55 * n_ev; }
void launch_finish(const BatchDev& b, int64_t* host, cudaStream_t s, Hooks* h);

// stage launchers (each enqueues its kernels on stream s)
void launch_ingest(const BatchDev& b, cudaStream_t s, Hooks* h);
void launch_md(const BatchDev& b, cudaStream_t s, Hooks* h);
void launch_sg(const BatchDev& b, cudaStream_t s, Hooks* h);
void launch_tl(const BatchDev& b, cudaStream_t s, Hooks* h);
void launch_tp(const BatchDev& b, cudaStream_t s, Hooks* h);
void launch_tc(const BatchDev& b, cudaStream_t s, Hooks* h);
// Training samples for the pre-filter from the last run's tracklet step
struct MlpCollect {
    float* x;                  // cap x kMlpIn features
    float* y;                  // cap labels (1: the tracklet cuts accept)
    int64_t cap;
    unsigned long long* n;     // samples found (can exceed cap; nothing past cap is written)
    float neg_keep;            // probability of keeping a rejected candidate
    unsigned long long seed;
};
void launch_tl_collect(const BatchDev& b, const MlpCollect& c, cudaStream_t s);
// self-check of the float-float fast paths (out[8]: see k_math_check)
void launch_math_check(int fn, int exhaustive, unsigned long long start, long long n, unsigned long long seed,
                       unsigned long long* out, int n_sm, cudaStream_t s);
// self-check of the mini-doublets' and segments' first passes (out[8]: see k_md_first_check)
void launch_first_cuts_check(const BatchDev& b, unsigned long long* out, cudaStream_t s);
// self-check of phase A's single-precision decision (out[4]: see k_tl_quick_check)
void launch_tl_b2q_check(const BatchDev& b, unsigned long long* out, cudaStream_t s);
void launch_tl_quick_check(const BatchDev& b, unsigned long long* out, cudaStream_t s);
// final cut variables of tracklets [first, first + n) (15 floats each, the kTLVar* order)
void launch_tl_vars(const BatchDev& b, int64_t first, int64_t n, float* out, cudaStream_t s);
// the host libm's float functions on the device (sdl_libm.cu): build the
// tables once per process, upload them once per device and point this
// module's kernels at them (call with the device current); the host tables'
// size, moved entries and exceptions of function fn; the device's values on
// consecutive float bit patterns; the constant-memory setter
int libm_setup(int device, const char** err);
void libm_stats(int fn, uint64_t* out3);
void launch_libm_eval(int fn, uint32_t start, int64_t n, float* out, int n_sm, cudaStream_t s);
cudaError_t set_libm_tables(const LibmTab* t);
// object graph of stage st for objects [first, first + n) of one event (see k_links)
void launch_links(const BatchDev& b, int st, int64_t first, int64_t n, int64_t lo_first, int64_t gm0, int32_t* links,
                  int32_t* module, float* vals, cudaStream_t s);
// hit-index tuples of stage st for objects [first, first + n) into out (width 2/4/8/8/16)
void launch_materialize(const BatchDev& b, int st, int64_t first, int64_t n, int32_t* out, cudaStream_t s);

// copies of 4-byte words to the device on the SMs, one kernel for up to
// kCopyJobs buffers in device or pinned host memory (the copy engines may be
// busy with readbacks, and each of their copies costs a few microseconds)
constexpr int kCopyJobs = 8;
struct CopyJobs {
    const uint32_t* src[kCopyJobs];
    uint32_t* dst[kCopyJobs];
    int64_t n[kCopyJobs];  // words
    int count;
    bool full;  // a job did not fit: the launch is refused
    void add(const void* from, void* to, int64_t words) {
        if (count == kCopyJobs) {
            full = true;
            return;
        }
        src[count] = static_cast<const uint32_t*>(from);
        dst[count] = static_cast<uint32_t*>(to);
        n[count++] = words;
    }
};
cudaError_t launch_copy_words(const CopyJobs& j, int n_sm, cudaStream_t s);

}  // namespace sdlg
