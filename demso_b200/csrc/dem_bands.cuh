// The step in bands: a layout of the sorted state that a step leaves in place.
//
// The reference sorts all particles by cell on every step, although between
// two steps of a granular scene only a few in a hundred thousand change cell.
// In a densely packed order each of them shifts every particle behind it, so
// even an incremental sort rewrites the whole state.  Here the order is kept
// in bands of whole cell rows with free slots at the end of each: a particle
// that changes cell shifts only the particles between the two places of its
// own band, or those behind it in the two bands it left and entered; every
// other band stays where it is, in every array.  A step is two kernels:
//
//   fix   one block per band that a particle left or entered in the last
//         step: the band's particles in the stable order of their new cells
//         ([arrivals from lower cells][stayers][arrivals from higher cells],
//         each in the previous order), in place;
//   step  collide + integrate + new cell, a thread per slot, from one dynamic
//         set into the other; radius, mass, id and type stay in place.  A
//         particle whose cell changed writes an event (its whole state) for
//         the band it enters and a note for the band it leaves.
//
// When a band's events or free slots run out (or there is no band layout yet)
// the next step first lays the bands out again: the state is packed, sorted
// with the radix sort and spread into bands.  At the end of a call the state
// is packed into the context's sorted arrays, so that every reader finds it
// as after a packed sort: the concatenation of the bands is the reference's
// sorted order, and the bits are its own.
//
// Against the packed incremental sort (six kernels a step, 40 B moved per
// particle in the sort phase and 88 B in the step; here two kernels, 68 B in
// the step), with the kept candidates below: a call of 20 steps of 4,194,304
// disks 4,669 -> 2,988 us, of 1,000,003 dense disks 1,503 -> 1,116 us, 50 steps of
// 65,536 1,229 -> 834 us, 20 steps of a fast gas of 131,071 584 -> 365 us, of 256
// specimens of two materials 1,243 -> 784 us.  A batch's specimens keep their
// own bands, so a slot never changes specimen.
//
// The two dynamic sets alternate with the steps (kBandCur: the one that holds
// the state; a new layout keeps it, so the host knows it from the step count).
// A kernel of set q does nothing unless kBandCur is q: when a step of the loop
// below is skipped for a new layout, the next one of its set takes its place.
#pragma once

#include <cstdint>
#include <cuda_runtime.h>
#include <vector>

#include "dem_kernels.cuh"

namespace dem {

constexpr uint32_t kBandEmpty = 0xffffffffu;  // key of a free slot
// Events (particles that left or entered) a band takes in one step.
constexpr uint32_t kBandEvents = 128;
// Free slots of a band: at least this, and a sixteenth of its share of n.
constexpr uint32_t kBandMinSlack = 64;
// Cells of a band: a whole row and at least kBandMinCells (a batch's, whose
// bands do not span specimens, kBandBatchCells where a specimen has them);
// scenes with wider rows than kBandMaxRow cells take the packed path (one block
// rewrites a band).
constexpr uint32_t kBandMinCells = 256, kBandBatchCells = 1024;
constexpr uint32_t kBandMaxRow = 4096, kBandMaxBands = 4096;

// Words of BandArgs::ctrl.
constexpr uint32_t kBandLeft = 0;   // steps left of the call
constexpr uint32_t kBandDone = 1;   // steps of the call done (the row block of the followed particles)
constexpr uint32_t kBandFull = 2;   // the next step needs a new layout
constexpr uint32_t kBandCur = 3;    // dynamic set holding the state
constexpr uint32_t kBandLaid = 4;   // the bands hold the state (0: only the packed arrays do)
constexpr uint32_t kBandAct = 5;    // [2] step of set q: 0 skipped, 1 runs, 2 runs as the call's last
constexpr uint32_t kBandDirty = 7;  // [2] bands with events, by the set the fix of which takes them
constexpr uint32_t kBandStep = 9;   // steps since the context was made
constexpr uint32_t kBandNow = 10;   // [2] kBandStep as the step of set q sees it
constexpr uint32_t kBandDirtySum = 12;  // bands the call's fixes rewrote (of more than kFixBlocks)
constexpr uint32_t kBandLayouts = 13;   // the call's layouts of a state that was in bands already
constexpr uint32_t kBandCtrlWords = 16;
// Blocks of the fix: that many bands are rewritten at once (two blocks to a
// multiprocessor).
constexpr uint32_t kFixBlocks = 296;

// Kept candidates.  The search for neighbours (row intervals, radii and
// distances of some twenty candidates) finds almost the same few pairs step
// after step.  Every slot keeps a bit for each candidate within reach plus a
// skin of kSkin * rmax, counted from the first slot of its row interval, 21
// bits for each of the three rows; a step then meets only those.  (A skin of
// 0.05 / 0.07 / 0.1: 144.7 / 145.8 / 148.3 us a step at 4,194,304 disks, 51.8 / 53.5 /
// 54.5 at 1,000,003 dense ones, 18.8 / 18.6 / 18.4 for a fast gas of 131,071.)  The bits
// are a superset of the contacts until a pair of the band or its neighbour
// bands may have closed the skin -- the sum over the steps since of the
// largest displacement of the band and of the largest of the three bands --
// or a particle enters or leaves a cell of the slot's 3 x 3, which stamps the
// cells around it for the next step.  Then the slot searches again.  Slots
// whose bits do not fit search on every step.
constexpr float kSkin = 0.07f;
constexpr uint32_t kCandBits = 21;
constexpr unsigned long long kCandNone = 1ull << 63;  // no bits kept: search

// A particle that changed cell: its slot and cells, and its state.
struct __align__(16) BandEvent {
    uint4 a;   // slot, new cell, old cell, id
    float4 b;  // position, velocity
    float4 c;  // angle, spin, radius, mass
    uint4 d;   // type
};

// A band: its cells, its first row in the first-slot array, the bands and packed
// slots of its scene or specimen before it, and in a batch the free slots before
// it.  kBandWhole in `free`: the band is its whole specimen; nothing leaves or
// enters it, so it has no free slots (20,000 specimens of 28 disks with 64 each
// stepped at 68.7 us, without at 34.2).
struct BandGeo {
    uint32_t cell0, cells, first, log2gx;
    uint32_t sceneBand, scenePart, spec, free;
};
constexpr uint32_t kBandWhole = 0x80000000u;

// Words in host memory that the device writes for the host to read whenever they
// arrive.
struct BandLoad {
    uint32_t busy;  // set by a call whose steps lost to the packed path (band_overload)
    // the last estimate (launch_band_estimate); kBandUnknown until it arrives
    uint32_t estDirty, estMovers;
};
constexpr uint32_t kBandUnknown = 0xffffffffu;

struct BandArgs {
    uint32_t bands = 0, shift = 0;  // band of a cell of a single scene: cell >> shift
    uint32_t cells = 0, firstWords = 0;
    uint32_t batchFree = 0;  // a batch's free slots in all
    const BandGeo* geo = nullptr;
    uint32_t* cellBand = nullptr;  // batches: band of a cell
    // batches: the specimens' parameters, the specimen of every slot
    const KParams* table = nullptr;
    uint32_t* slotSpec = nullptr;
    uint32_t n = 0, slots = 0, slack = 0;
    DynSet dyn[2] = {};  // slot-indexed
    StatSet stat = {};
    uint32_t* key = nullptr;  // cell of every slot's particle (kBandEmpty: free)
    uint32_t* loc = nullptr;  // slot by id
    uint32_t* first = nullptr;  // first slot of every cell, gx + 1 words a row (the last: row end)
    uint32_t* base = nullptr;   // bands + 1
    uint32_t* count = nullptr;  // particles of each band
    uint32_t* gap = nullptr;    // slots less packed places of each band (launch_band_gaps)
    uint32_t* evCnt = nullptr;
    BandEvent* ev = nullptr;
    uint32_t* dirty[2] = {};
    unsigned long long* cand = nullptr;  // kept candidates of every slot
    float skin = 0.0f;
    uint32_t* stamp = nullptr;      // per cell: the step that searches anew there
    uint32_t* moved[2] = {};        // per band: largest |dx| + |dy| of a step (float bits)
    float* grown = nullptr;         // per band: bound on a pair's approach since the search
    uint32_t* search = nullptr;     // per band: this step searches anew
    uint32_t* ctrl = nullptr;
    uint32_t* mark = nullptr;  // per band: the last estimate (launch_band_estimate) that met it
    BandLoad* load = nullptr;  // may be null: `busy`, set by a call's pack
    float* pressure = nullptr;  // slot-indexed, null when not kept
    float2* acc = nullptr;
    float* alpha = nullptr;
    uint32_t* errFlag = nullptr;
};

// The packed arrays: the context's state in sorted order.
struct PackedState {
    DynSet dyn;
    StatSet stat;
    uint32_t* loc;
    float* pressure;
    float2* acc;
    float* alpha;
};

// The bands of the `grids` grids P (one scene, partOff null, or a batch's specimens
// of partOff[s + 1] - partOff[s] particles), whose firstOff it sets; false when a
// grid takes the packed path.
bool band_shape(KParams* P, uint32_t grids, const uint32_t* partOff, BandArgs& b,
                std::vector<BandGeo>& geo);
// Free slots per band of a single scene, and slots in all, for n particles.
uint32_t band_slack(const BandArgs& b, uint32_t n);
size_t band_slots(const BandArgs& b, uint32_t n, bool batch);
// Bytes of the band arrays of `capacity` particles, and their addresses.
size_t band_bytes(const BandArgs& b, uint32_t capacity, bool typed, bool pressure, bool accel,
                  bool batch);
void carve_bands(BandArgs& b, void* base, uint32_t capacity, bool typed, bool pressure, bool accel,
                 bool batch);

// Band of every cell of a batch (once, after the arrays are made).
cudaError_t launch_band_cell_table(const BandArgs& b, cudaStream_t st);

// Adds to out[0] the bands that particles would leave or enter if all moved on
// by a step at their velocities, to out[1] the particles; `serial`: another
// number each time.  spec: a batch's specimen of every packed slot.  Of many
// particles a part is looked at, one block of 256 in band_estimate_stride.
inline uint32_t band_estimate_stride(uint32_t n) { return n >> 20 ? n >> 20 : 1u; }
cudaError_t launch_band_estimate(const KParams& P, const BandArgs& b, const float2* pos,
                                 const float2* vel, const uint32_t* spec, uint32_t n,
                                 uint32_t serial, uint32_t* out, cudaStream_t st);

// The kernels; `q` is the dynamic set they step from.
cudaError_t launch_band_fix(const BandArgs& b, int q, cudaStream_t st);
// everyStep: pressure and accelerations are stored on every step, not only on
// the call's last one.
cudaError_t launch_band_step(const KParams& P, const BandArgs& b, int q, bool everyStep,
                             int variant, ControlArgs ctl, cudaStream_t st);
// Before a step with a control particle, whose reactions are stored in packed
// order: the bands' gaps.
cudaError_t launch_band_gaps(const BandArgs& b, cudaStream_t st);
cudaError_t launch_band_followed(const BandArgs& b, int q, const uint32_t* ids,
                                 const uint32_t* countWord, float* ring, cudaStream_t st);
// The record of the step of set q (adj_record_step's, packed) at record block
// kBandDone - 1 from recBase, records `stride` bytes apart.
cudaError_t launch_band_record(const BandArgs& b, int q, void* recBase, size_t stride,
                               cudaStream_t st);
// The state into the packed arrays (with pressure and accelerations unless
// stateOnly); nothing when the bands hold no state.
cudaError_t launch_band_pack(const BandArgs& b, const PackedState& out, bool stateOnly,
                             cudaStream_t st);
// Whether nearly all bands are rewritten on every step (see too_many_movers).
__host__ __device__ inline bool band_overload(uint32_t bands, uint32_t dirty) {
    return bands > kFixBlocks && dirty > bands - bands / (bands < 2048u ? 10u : 25u);
}
// New layout from the packed arrays, sorted by `keys` (their particles in
// order `from`); cellFirst: numCells + 1 words of scratch.
cudaError_t launch_band_layout(const BandArgs& b, const PackedState& in, const uint32_t* keys,
                               const uint32_t* from, uint32_t* cellFirst, cudaStream_t st);
// Packed cell ranges and first-particle array of the current state.
cudaError_t launch_band_cells(const BandArgs& b, uint2* cells, uint32_t* first, cudaStream_t st);

// Conditions of the step loop's graph nodes.
cudaError_t launch_band_head(const BandArgs& b, cudaGraphConditionalHandle full,
                             cudaGraphConditionalHandle loop, bool setLoop, cudaStream_t st);
cudaError_t launch_band_next(const BandArgs& b, cudaGraphConditionalHandle loop, bool whileFull,
                             cudaStream_t st);

}  // namespace dem
