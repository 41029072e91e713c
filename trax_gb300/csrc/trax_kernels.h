// trax_kernels.h -- host-side launchers of the sm_103a kernels.  Each
// launcher enqueues work on its Queue's stream (or `st`) and counts the
// kernels it launched.  Counts that are only known on the device are passed as
// device pointers together with a host-side capacity that sizes the grid.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include "trax_device.cuh"

struct trax_ctx;

namespace trax {

// Where the launchers enqueue: a stream, the number of kernels launched so
// far, and the time marks the next kernel writes as it starts.
struct Queue {
  cudaStream_t st = nullptr;
  uint32_t launches = 0;
  Stamp marks;
};

// Every kernel of the chain takes its Stamp first.
template <class... P, class... A>
cudaError_t launch(Queue& q, void (*kernel)(Stamp, P...), dim3 blocks, unsigned threads, size_t smem,
                   A&&... args) {
  cudaLaunchConfig_t c = {};
  c.gridDim = blocks;
  c.blockDim = dim3(threads);
  c.dynamicSmemBytes = smem;
  c.stream = q.st;
  const Stamp marks = q.marks;
  q.marks.which = 0;
  ++q.launches;
  return cudaLaunchKernelEx(&c, kernel, marks, static_cast<P>(args)...);
}

// ---------------------------------------------------------------- scans
size_t scan_scratch_bytes(uint64_t maxN);
// One array to scan, in place allowed; scratch holds scan_scratch_bytes.
struct ScanJob {
  const uint32_t* in;
  uint32_t* out;
  void* scratch;
  ScanTotal total;
};
// Exclusive scans of one or two arrays of n elements (or *nDev + nAdd when
// nDev != nullptr, with maxN bounding the launch).  Outputs wrap modulo 2^32;
// with flagOverflow a total of 2^32 or more sets TRAX_EBIT_OVERFLOW.  `ctl`
// bounds the look-back waits (and may name a tile that never publishes).
// `cleared`: the scratch is zero already and used by no other scan since
// (otherwise it is cleared here).
cudaError_t scan_exclusive(const ScanJob* jobs, int nJobs, uint64_t n, const uint32_t* nDev, uint32_t nAdd,
                           uint64_t maxN, bool cleared, uint32_t* err, Queue& q, bool flagOverflow, WaitCtl ctl);
// one array of n elements
cudaError_t scan_exclusive(const uint32_t* in, uint32_t* out, uint64_t n, void* scratch, uint32_t* err, Queue& q,
                           bool flagOverflow, WaitCtl ctl);

// ------------------------------------------------------ event bucketing
// The hits of a group of events as their file holds them, with the host's
// bucketing keys (trax_events.h); scratchOffsets[e]: the event's global
// sort scratch (events too large for shared memory).
struct RawEventHits {
  const float* x;
  const float* y;
  const float* z;
  const uint32_t* layer;
  const uint32_t* det;
  const uint32_t* tid;
  const unsigned long long* key;
  const uint32_t* rawOffsets;      // [E+1]
  const uint32_t* scratchOffsets;  // [E]
};
// the context's input hit columns and the first kept hit of each event
struct HitColumns {
  float* x;
  float* y;
  float* z;
  uint32_t* layer;
  uint32_t* det;
  uint32_t* hid;
  uint32_t* evt;
  const uint32_t* eventOffsets;  // [E]
};
// global scratch keys an event of this many hits needs (0: shared memory)
uint32_t bucket_scratch_keys(uint32_t hitsInEvent);
// every event's kept hits, sorted by key, into the columns at its offset
cudaError_t bucket_events(const RawEventHits& in, unsigned long long* scratch, uint32_t nEvents, uint32_t nKept,
                          HitColumns out, cudaStream_t st, uint32_t* launches);

// per (event, layer triplet) segment of the triplet offsets [S+1]: fake
// triplets, real
// triplets of findable tracks, distinct findable tracks found; findIds are
// each event's findable track ids, sorted, from findOff[e]; foundFlags
// [nLT * n_findable] zeroed by the caller, as are fakes and realFindable
cudaError_t physics_counts(const uint32_t* h1, const uint32_t* h2, const uint32_t* h3, const uint32_t* nTDev,
                           uint64_t maxT, const uint32_t* offsets, const uint32_t* hitTrack, uint32_t nEvents,
                           uint32_t nLT, const uint32_t* findOff,
                           const uint32_t* findIds, uint32_t* fakes, uint32_t* realFindable, uint32_t* foundFlags,
                           uint32_t* found, cudaStream_t st, uint32_t* launches);

// ------------------------------------------------------ track evaluation
// The tracks of the CA output (k_tracks.cu): [nTracks] hit-list start and
// size, real flag, first hit's simulated track id, union-find parent,
// component size / start / cursor (nTracks + 1 for the scan), members and
// the filtered list per component; [entries] hits and their track; [hits]
// the smallest track holding each hit.
struct TrackLists {
  uint32_t* start;
  uint32_t* size;
  uint32_t* real;
  uint32_t* firstId;
  uint32_t* parent;
  uint32_t* compSize;
  uint32_t* compStart;
  uint32_t* cursor;
  uint32_t* members;
  uint32_t* filtered;
  uint32_t* hits;
  uint32_t* entryTrack;
  uint32_t* owner;
};
// isTrack[i], hitsOf[i] for i <= nT (the +1 slots zero): chains of three or
// more triplets and their hit counts
cudaError_t track_sizes(const uint32_t* off, uint32_t nT, uint32_t* isTrack, uint32_t* hitsOf, cudaStream_t st);
// with isTrack / hitsOf scanned into trackOf / hitStart
cudaError_t track_extract(const uint32_t* off, const uint32_t* chain, uint32_t nT, const uint32_t* h1,
                          const uint32_t* h2, const uint32_t* h3, const uint32_t* hitTrack, const uint32_t* trackOf,
                          const uint32_t* hitStart, TrackLists t, cudaStream_t st);
// one union-find round (hook, compress); *changed set when a root moved
cudaError_t track_union_step(TrackLists t, uint32_t nTracks, uint32_t nEntries, uint32_t* changed, cudaStream_t st);
// place == false: component sizes; true: members at the scanned starts
cudaError_t track_members(TrackLists t, uint32_t nTracks, bool place, cudaStream_t st);
// per component the greedy clone removal; counts[0..2]: filtered, real,
// distinct real simulated track ids (table: 2^k zeroed slots, mask 2^k - 1)
cudaError_t track_greedy(TrackLists t, uint32_t nTracks, unsigned long long* table, uint32_t tableMask,
                         unsigned long long* counts, cudaStream_t st);

// ------------------------------------------------------------ grid build
struct GridInput {  // the seven columns first, in DevHits' order
  const float* x;
  const float* y;
  const float* z;
  const uint32_t* layer;
  const uint32_t* det;
  const uint32_t* hid;
  const uint32_t* evt;
  const uint32_t* eventOffsets;  // [E]
  const uint32_t* layerHits;     // [E*L]
  const uint32_t* layerOffsets;  // [E*L]
};

struct GridScratch {
  uint32_t* cell;    // [n]
  float* phi;        // [n]
  uint32_t* perm;    // [n]
  uint32_t* counts;  // [E*L*C] used when the cell counters do not fit in shared memory
  uint4* clear;      // scan scratch of the chain, zeroed by the grid build (clearWords of 16 bytes)
  uint32_t clearWords;
};

cudaError_t grid_build(const DevConfig& cfg, const GridInput& in, uint32_t* grid, DevHits out,
                       GridScratch scratch, uint32_t maxLayerHits, uint32_t* err, Queue& q);
cudaError_t grid_prepare(int device);  // one-time kernel attributes
// Layer size a grid build captured for layers of up to maxLayerHits hits can
// be laid out for at no cost: a quarter more, as far as the CTAs per SM stay.
uint32_t grid_layer_room(const DevConfig& cfg, uint32_t maxLayerHits);

// The fine z grid the prediction count walks when cfg.fineRows > 0: the
// grid-ordered hits of every (event, layer) sorted again by fine cell (fine
// row = fine_row of the hit's z inside its z row's block of fineRows rows,
// the same phi column), ties by grid order.  grid[E*L*fineC] holds the
// cell starts like the grid's, hits[n] each hit in fine order as (z, phi,
// its grid-order index as the bits of a float, 0): one 16-byte load gives
// a visit its test and its candidate.  Built from the grid and the
// grid-ordered packed hits (xyzp) after grid_build; `counters` (global
// scratch of fine_counter_cells(cfg) words) is used only when one z row's
// fine cells do not fit in shared memory.
struct FineGrid {
  uint32_t* grid;
  float4* hits;
};
// dynamic shared memory the grid builds give one CTA
#define TRAX_GRID_SMEM_BYTES (227u * 1024u - 256u)
inline uint32_t fine_row_cells(const DevConfig& cfg) { return cfg.fineRows * (cfg.nP + 1); }
inline uint64_t fine_counter_cells(const DevConfig& cfg) {
  return (uint64_t)fine_row_cells(cfg) * sizeof(uint32_t) > TRAX_GRID_SMEM_BYTES
             ? (uint64_t)cfg.E * cfg.L * cfg.nZ * fine_row_cells(cfg)
             : 0;
}
cudaError_t fine_grid_build(const DevConfig& cfg, const uint32_t* grid, const float4* xyzp, FineGrid fine,
                            uint32_t* counters, Queue& q);
// hit collection = uploaded hits in input order (plus the packed xyz-phi array)
cudaError_t identity_hits(const GridInput& in, uint32_t n, DevHits out, Queue& q);

// ----------------------------------------------------------------- pairs
// Per (event, layer triplet) segment: its first outer hit, and the exclusive
// scan of the segments' outer hits in taskBase[S+1] with its total published
// (S up to TRAX_SEGMENT_SCAN; above, the counts are left for scan_exclusive).
#define TRAX_SEGMENT_SCAN 32767u
cudaError_t pair_segments(const DevConfig& cfg, const uint32_t* grid, uint32_t* segOuter, uint32_t* taskBase,
                          ScanTotal total, uint32_t* err, Queue& q);
// What the count pass leaves for the store pass per outer-hit task k, so
// that the store pass neither searches the task's segment nor recomputes
// its window: bounds[k] = (zLow, zHigh, phiLow, phiHigh);
// secs[k] = (zLowSector | ordered << 31, zHighSector | wrap << 31, pL, pH),
// `ordered` when the task's visit ranges are disjoint and ascending
// (zLowSector <= INT32_MAX, zHighSector <= nZ < 2^22); ids[k] = (outer hit,
// segment).  pair_task_state_bytes(n) bytes hold the arrays of n tasks.
struct PairTaskState {
  float4* bounds;
  uint4* secs;
  uint2* ids;
};
inline size_t pair_task_state_bytes(uint64_t n) { return (size_t)n * 40u; }
inline PairTaskState pair_task_state(void* base, uint64_t n) {
  char* b = static_cast<char*>(base);
  return PairTaskState{reinterpret_cast<float4*>(b), reinterpret_cast<uint4*>(b + 16 * n),
                       reinterpret_cast<uint2*>(b + 32 * n)};
}

// Count (emit == false) or store (emit == true) pairs of every outer-hit task.
// taskBase[S+1] is the exclusive scan of segCount; nTasksDev = &taskBase[S].
// The count pass writes `state`, the store pass reads it and also writes
// pairOffsets[s] = first pair of segment s (Pairing::pairingOffsets).
cudaError_t pair_tasks(const DevConfig& cfg, bool emit, const uint32_t* grid, DevHits hits,
                       const uint32_t* segOuter, const uint32_t* taskBase, const uint32_t* nTasksDev,
                       uint64_t maxTasks, uint32_t* taskCount, PairTaskState state, uint2* pairs,
                       uint64_t capPairs, uint32_t* pairOffsets, uint32_t* sentinelCount, uint32_t* err, Queue& q);

// ------------------------------------------------------------ prediction
// Count pass (emit == false): per pair the exclusive offset of its
// candidates within its warp of 32 pairs (candCount[nPairs]), the sum of
// each warp's counts in warpSums[ceil(nPairs/32) + 1] (+1 slot zeroed; the
// number of sums goes to *nWarpsOut) and up to cfg.predKeep captured
// candidates per pair in keep[nPairs * cfg.predKeep]; store pass
// (emit == true): with warpSums exclusively scanned, candidates at
// warpSums[gid / 32] + candCount[gid].  predKeep is 4 (TRAX_PRED_KEEP,
// the default) to TRAX_PRED_KEEP_MAX.
#define TRAX_PRED_KEEP 4
#define TRAX_PRED_KEEP_MAX 32
// words of the captured candidates of `pairs` pairs, whole warps of 32
// pairs; the slots of a warp's pairs are interleaved (keep_slots) with 16 or
// more slots per pair or with the fine z grid
inline uint64_t pred_keep_words(uint64_t pairs, uint32_t keep) { return (pairs + 31) / 32 * 32 * keep; }
inline bool keep_interleaved(const DevConfig& cfg) { return cfg.predKeep >= 16u || cfg.fineRows > 0u; }

// grids of up to this many cells per layer are built with shared-memory
// counters (4 bytes per cell)
#define TRAX_GRID_SMEM_CELLS 53248u
// With cfg.fineRows > 0 the count pass, and the store pass's re-walks of
// pairs with more candidates than slots, walk `fine` (same outputs).  The
// store pass also writes candOffsets[s] = first candidate of segment s.
cudaError_t predict_pairs(const DevConfig& cfg, bool emit, const uint32_t* grid, DevHits hits, const uint2* pairs,
                          const uint32_t* nPairsDev, uint64_t maxPairs, uint32_t* candCount, uint32_t* warpSums,
                          uint32_t* nWarpsOut, uint32_t* keep, uint2* cands, uint64_t capCands,
                          uint32_t* sentinelCount, uint32_t* err, Queue& q,
                          FineGrid fine, const uint32_t* pairOffsets, uint32_t* candOffsets);

// ---------------------------------------------------------------- filter
// the flags of 32 consecutive candidates as one word masks[g / 32] (bit
// g % 32), the number of flags set per word in warpSums[ceil(n/32) + 1]
// (+1 slot zeroed; the number of words goes to *nWordsOut)
cudaError_t filter_candidates(const DevConfig& cfg, DevHits hits, const uint2* pairs, const uint2* cands,
                              const uint32_t* nCandsDev, uint64_t maxCands, uint32_t* masks, uint32_t* warpSums,
                              uint32_t* nWordsOut, Queue& q);
// Segments of the triplets: segStart[s] = first triplet of segment s or later,
// offsets = trackletOffsets, both S + 1 entries.
struct TripletSegments {
  uint32_t S;
  const uint32_t* candOffsets;  // first candidate of every segment
  const uint32_t* nTDev;
  uint32_t* segStart;
  uint32_t* offsets;
};
// with warpSums exclusively scanned into wordStart: the triplets of the
// flagged candidates at wordStart[g / 32] + (flags below g in its word)
cudaError_t filter_store(const uint2* pairs, const uint2* cands, const uint32_t* nCandsDev, uint64_t maxCands,
                         const uint32_t* masks, const uint32_t* wordStart, uint32_t* h1, uint32_t* h2, uint32_t* h3,
                         uint64_t capT, TripletSegments seg, Queue& q);
// ---------------------------------------------------------- connectivity
struct TripletView {
  const uint32_t* h1;
  const uint32_t* h2;
  const uint32_t* h3;
  const uint32_t* nDev;
  uint64_t maxN;
};

// What connectivity starts from: eta, inDeg / inCursor zeroed, and the runs.
struct LinkStart {
  float* eta;
  uint32_t* inDeg;     // [nT+1]
  uint32_t* inCursor;  // [nT]
  // [nHits] or null: (first, end) of the triplets whose second hit it is.
  // Only hits that are some triplet's second hit have theirs written, so an
  // entry counts when its first triplet is there and has that second hit.
  // Given where every layer is the second of one layer triplet at most.
  uint2* runs;
};
// A caller's triplets: segStart and offsets as TripletSegments, and segOf[t].
cudaError_t triplet_segments(const DevConfig& cfg, DevHits hits, TripletView t, uint32_t* segStart, uint32_t* segOf,
                             uint32_t* offsets, Queue& q);
cudaError_t triplet_link_start(const DevConfig& cfg, DevHits hits, TripletView t, LinkStart link, Queue& q);
// links per basis triplet (linkCount, +1 slot zeroed) and per follower
// (inDeg); runStart[t]: where the store pass starts looking for t's followers
cudaError_t connectivity_count(const DevConfig& cfg, DevHits hits, TripletView t, const float* eta,
                               const uint32_t* offsets, const uint32_t* segStart, const uint2* runs,
                               uint32_t* linkCount, uint32_t* inDeg, uint32_t* runStart, bool sortedSegments,
                               Queue& q);
// With linkCount and inDeg scanned (the latter into inStart): the links, the
// bases of each follower's links in inList (any order), and the words of 32
// connectable flags with the number set per word (+1 slot zeroed, the number
// of words to *nWordsOut)
struct LinkStore {
  const uint32_t* linkStart;
  const uint32_t* runStart;
  const uint32_t* inStart;
  uint32_t* inCursor;
  uint32_t* basis;
  uint32_t* follower;
  uint32_t* inList;
  uint32_t capLinks;
  bool sortedSegments;
  uint32_t* connWords;
  uint32_t* connSums;
  uint32_t* nWordsOut;
};
cudaError_t connectivity_store(const DevConfig& cfg, TripletView t, const float* eta, LinkStore ls, Queue& q);
// With connSums scanned into wordStart: the connectable and non-connectable
// triplets among the first nT - 1
struct ConnLists {
  const uint32_t* wordStart;
  uint32_t* conn;
  uint32_t* nonConn;
};
cudaError_t connectable_lists(TripletView t, const uint32_t* connWords, ConnLists lists, Queue& q);
// the context's slots and the time marks after them to page-locked host memory
cudaError_t slots_to_host(const uint32_t* slots, uint32_t* host, uint32_t words, Queue& q);

// ---------------------------------------------------- circle fit and CA
cudaError_t circle_fit(DevHits hits, TripletView t, const uint32_t* connectable, const uint32_t* nConnDev,
                       uint64_t maxConn, float* pt, Queue& q);

// pt[t] of every triplet: the circle fit of the connectable ones, 0 for the others
cudaError_t circle_fit_words(DevHits hits, TripletView t, const uint32_t* connWords, float* pt,
                             const ConnLists* lists, Queue& q);

struct CABuffers {
  uint32_t* states;    // [nT]
  uint32_t* inStart;   // [nT+1]
  uint32_t* inCursor;  // [nT]
  uint32_t* inList;    // [nLinks] bases of the incoming links, grouped by follower, any order
  uint32_t* best;      // [nT]
  uint32_t* isBest;    // [nT]
  uint32_t* handlers;  // [nT+1]
  uint32_t* segOf;     // [nT] layer-triplet segment of each triplet
};

cudaError_t ca_in_degree(const uint32_t* follower, const uint32_t* nLinksDev, uint64_t maxLinks, CABuffers b,
                         const uint32_t* nTDev, uint64_t maxT, Queue& q);
cudaError_t ca_fill(const uint32_t* basis, const uint32_t* follower, const uint32_t* nLinksDev, uint64_t maxLinks,
                    CABuffers b, Queue& q);
// Triplets per event (on average) up to which one CTA per event runs the
// chain's CA (ca_event_kernel); above, a CTA would take too many steps and a
// launch per level over the whole chip is faster.
#define TRAX_CA_EVENT_TRIPLETS 16384u
// The chain's forward and backward phases and handlers (inStart and inList
// given).  perEvent: one CTA per event; segStart null: levels by segOf.
cudaError_t ca_chain(const DevConfig& cfg, const float* pt, CABuffers b, const uint32_t* segStart, bool perEvent,
                     const uint32_t* nTDev, uint64_t maxT, const uint32_t* nLinksDev, Queue& q);
// One forward iteration of the reference's CA over any link set
// (CellularAutomaton.h:52-100); *living is set when a cell lives.
cudaError_t ca_iteration(const uint32_t* basis, const uint32_t* follower, uint32_t nLinks, const uint32_t* cur,
                         uint32_t* next, uint32_t* living, Queue& q);
cudaError_t fill_u32(uint32_t* p, uint32_t v, uint32_t n, Queue& q);
cudaError_t ca_backward(const float* pt, CABuffers b, const uint32_t* nTDev, uint64_t maxT,
                        const uint32_t* nLinksDev, const uint32_t* err, Queue& q);
cudaError_t ca_tracks(CABuffers b, const uint32_t* nTDev, uint64_t maxT, uint32_t* tracks, uint64_t maxTracks,
                      uint32_t* err, Queue& q);

// ------------------------------------------- differentiable triplet fit
// Fit rows are the selected triplets ordered by layer triplet; rows of layer
// triplet k are [ltBase[k], ltBase[k+1]) and are reduced by the blocks
// [blkStart[k], blkStart[k+1]), each taking `chunk` rows, so that every
// sum is taken in a fixed order.
// Rows per block: two blocks of the gradient fit in an SM at a time, and about
// four blocks per SM give two full waves of equal blocks, each thread with as
// many rows as possible before the block's sums; at least one row per thread.
// (Blocks of a fixed 4096 rows kept 17 of 152 SMs busy for 66 k rows, and
// blocks of 512 spent a seventh of their instructions on the sums.)
#define TRAX_FIT_CHUNK_MIN 256u
inline uint32_t fit_chunk(uint64_t rows, uint32_t nLT, int sms) {
  const uint64_t blocks = (uint64_t)sms * 4 - nLT;  // a layer triplet's last block is not full
  const uint64_t c = (rows / blocks + TRAX_FIT_CHUNK_MIN) / TRAX_FIT_CHUNK_MIN * TRAX_FIT_CHUNK_MIN;
  return (uint32_t)(c > 0x40000000ull ? 0x40000000ull : c);
}

// per block: chi2, d chi2 / d(dr, dz, dphi) of the three hit layers, and an
// approximate Gauss-Newton diagonal for the same nine (a preconditioner)
#define TRAX_FIT_SLOTS 19

struct FitConfig {
  uint32_t L, nLT, nBlocks, chunk;
  uint32_t layer[3][TRAX_MAX_LT];  // 0-based layer of each hit slot of a layer triplet
  float wTip[TRAX_MAX_LT];         // 1 / sigma_tip^2 per layer triplet
  float wZ;                        // 1 / sigma_z^2
  // per-layer correction: r -> r + dr, z -> z + dz, rotation by dphi given
  // as sin(dphi) and cos(dphi) - 1 (both from double precision on the host)
  float dr[TRAX_MAX_LAYERS], dz[TRAX_MAX_LAYERS], sn[TRAX_MAX_LAYERS], cm1[TRAX_MAX_LAYERS];
  uint32_t ltBase[TRAX_MAX_LT + 1];
  uint32_t blkStart[TRAX_MAX_LT + 1];
};

// ok[t] = 1 for triplets whose hits lie on their layer triplet's layers, whose
// three hits share a nonzero hit id when truthOnly, and whose fit at the
// configured alignment is finite; segCount[s] counts them per segment
cudaError_t fit_select(const FitConfig& fc, const DevConfig& cfg, DevHits hits, TripletView t, uint64_t nT,
                       int truthOnly, uint32_t* ok, uint32_t* segCount, cudaStream_t st, uint32_t* launches);
// rows[okScan[t] + segDelta[seg(t)]] = t for the selected triplets
cudaError_t fit_scatter(const DevConfig& cfg, DevHits hits, TripletView t, uint64_t nT, const uint32_t* okScan,
                        const int32_t* segDelta, uint32_t* rows, cudaStream_t st, uint32_t* launches);
// chi2 (and with grad: alignment and hit gradients) of the fit rows.
// partials[b * TRAX_FIT_SLOTS + k]; params[row * 4] = (curvature, d0, z0,
// cot theta) when not null; dHits (double, grid order, 3 per hit) is added to
// when not null.
cudaError_t fit_eval(const FitConfig& fc, bool grad, DevHits hits, TripletView t, const uint32_t* rows,
                     double* partials, float* params, double* dHits, cudaStream_t st, uint32_t* launches);
// out[0] = chi2, out[1 + 3 l + p] = d chi2 / d(dr, dz, dphi)_l, and
// out[1 + 3 L + 3 l + p] = the approximate Gauss-Newton diagonal; fixed-order sums
cudaError_t fit_reduce(const FitConfig& fc, const double* partials, double* out, cudaStream_t st,
                       uint32_t* launches);
// uploaded (input-order) hits corrected in place by fc's per-layer shifts
cudaError_t fit_apply(const FitConfig& fc, float* x, float* y, float* z, const uint32_t* layer, uint64_t n,
                      cudaStream_t st, uint32_t* launches);
// float gradient per input hit from the double grid-order sums
cudaError_t fit_hits_out(const double* dHits, const uint32_t* orig, uint64_t nHits, float* out, cudaStream_t st,
                         uint32_t* launches);

// number of SMs of the current device (cached)
int sm_count();

// context hooks for the autotuner (capi.cu)
uint64_t workload_hash(const trax_ctx* c);
int ctx_device(const trax_ctx* c);
bool ctx_ready(const trax_ctx* c);
void ctx_set_error(trax_ctx* c, const char* msg);

}  // namespace trax
