// The step in bands (see dem_bands.cuh).
#include "dem_bands.cuh"

#include <algorithm>

#include "dem_collide.cuh"
#include "dem_sort.cuh"

namespace dem {
namespace {

inline unsigned blocks_for(size_t n, int t) { return (unsigned)((n + (size_t)t - 1) / (size_t)t); }
inline size_t al256(size_t b) { return (b + 255u) & ~(size_t)255u; }

// Entries of the sorted a[0, n) below v.
__device__ __forceinline__ uint32_t lower_count(const uint32_t* a, uint32_t n, uint32_t v) {
    uint32_t lo = 0, hi = n;
    while (lo < hi) {
        const uint32_t mid = (lo + hi) >> 1;
        if (a[mid] < v) lo = mid + 1u;
        else hi = mid;
    }
    return lo;
}

__device__ __forceinline__ uint32_t band_of(const BandArgs& B, uint32_t cell) {
    return B.cellBand ? __ldg(B.cellBand + cell) : cell >> B.shift;
}

// Free slots before band b.
__device__ __forceinline__ uint32_t free_before(const BandArgs& B, uint32_t b) {
    return B.table ? B.geo[b].free & ~kBandWhole : b * B.slack;
}

// ------------------------------------------------------------------ fix
// Bound by latency: four rounds of loads (the control words; the band's words
// and events; its cells' first slots; its fields), each begun together: 153.8 ->
// 150.4 us a step at 4,194,304 disks, 18.1 -> 17.4 at 131,071 fast ones, against
// a load at a time.  512 threads hold a run of 512 particles in registers while the
// next run loads, so a band of any length is rewritten in place: a particle
// moves by at most kBandEvents slots, so the places a run is stored to have
// been read by then.  Two such blocks fit on a multiprocessor, so 296 bands
// are rewritten at once; runs of 1,024 (one block) measured 162 against 154 us
// a step at 4,194,304 disks, 256 threads 165.
constexpr int kFixThreads = 512;
constexpr int kFixItems = 1;
constexpr uint32_t kFixRun = kFixThreads * kFixItems;
static_assert(kBandEvents <= kFixRun && kBandEvents <= (uint32_t)kFixThreads,
              "an event per thread; moves stay within the next run");

template <bool TYPED>
struct Held {
    float2 p, v;
    float th, om, r, m;
    uint32_t id, key, type, dst;
    unsigned long long cand;
};

struct FixShared {
    uint4 ev[kBandEvents];           // slot, new cell, old cell
    uint32_t leave[kBandEvents];     // leavers' places in the band, sorted
    uint32_t leaveCell[kBandEvents]; // their old cells (sorted too)
    uint32_t arrive[kBandEvents];    // arrivals' 2 * cell + (from a higher cell), sorted
    uint32_t arriveEv[kBandEvents];
    uint32_t arriveDst[kBandEvents];  // by event
    uint32_t arriveAt[kBandEvents];   // the old place they go in front of
    uint32_t nl, na;
};

template <bool TYPED>
__device__ __forceinline__ void fix_load(const BandArgs& B, const DynSet& d, const FixShared& S,
                                         uint32_t base, uint32_t cell0, uint32_t from,
                                         uint32_t end, uint32_t nl, uint32_t na,
                                         Held<TYPED> (&h)[kFixItems]) {
#pragma unroll
    for (int u = 0; u < kFixItems; ++u) {
        const uint32_t j = from + (uint32_t)u * kFixThreads + threadIdx.x;
        h[u].dst = kBandEmpty;
        if (j >= end) continue;
        const uint32_t s = base + j;
        h[u].key = B.key[s];
        h[u].p = d.pos[s];
        h[u].v = d.vel[s];
        h[u].th = d.theta[s];
        h[u].om = d.omega[s];
        h[u].r = B.stat.radius[s];
        h[u].m = B.stat.mass[s];
        h[u].id = B.stat.id[s];
        h[u].cand = B.cand[s];
        if (TYPED) h[u].type = B.stat.type[s];
        const uint32_t rl = lower_count(S.leave, nl, j);
        if (rl < nl && S.leave[rl] == j) continue;  // it left
        const uint32_t to = j - rl + lower_count(S.arrive, na, 2u * (h[u].key - cell0) + 1u);
        if (to != j) h[u].dst = to;
    }
}

template <bool TYPED>
__device__ __forceinline__ void put(const BandArgs& B, const DynSet& d, uint32_t s, float2 p,
                                    float2 v, float th, float om, float r, float m, uint32_t id,
                                    uint32_t type, uint32_t key, unsigned long long cand) {
    d.pos[s] = p;
    d.vel[s] = v;
    d.theta[s] = th;
    d.omega[s] = om;
    B.stat.radius[s] = r;
    B.stat.mass[s] = m;
    B.stat.id[s] = id;
    if (TYPED) B.stat.type[s] = type;
    B.key[s] = key;
    B.cand[s] = cand;
    B.loc[id] = s;
}

template <bool TYPED>
__device__ void fix_band(const BandArgs& B, const DynSet& d, FixShared& S, uint32_t b) {
    const uint32_t tid = threadIdx.x;
    // the band's words and the events, whether or not there are that many, in
    // one round of loads
    const BandGeo geo = B.geo[b];
    const uint32_t cell0 = geo.cell0, gx = 1u << geo.log2gx;
    const uint32_t base = B.base[b], cnt = B.count[b];
    const uint32_t ne = min(B.evCnt[b], kBandEvents);
    BandEvent e{};
    if (tid < kBandEvents) {
        e = B.ev[(size_t)b * kBandEvents + tid];
        S.ev[tid] = e.a;
    }
    if (tid == 0) S.nl = S.na = 0u;
    __syncthreads();
    const bool mine = tid < ne;
    const bool enters = mine && e.a.y - cell0 < geo.cells;
    if (mine) {
        const bool leaves = e.a.z - cell0 < geo.cells;
        const uint32_t k2 = 2u * e.a.y + (e.a.z < e.a.y ? 0u : 1u);
        uint32_t rl = 0, ra = 0;
        for (uint32_t f = 0; f < ne; ++f) {
            const uint4 o = S.ev[f];
            const uint32_t o2 = 2u * o.y + (o.z < o.y ? 0u : 1u);
            if (o.z - cell0 < geo.cells && o.x < e.a.x) ++rl;
            if (o.y - cell0 < geo.cells && (o2 < k2 || (o2 == k2 && o.x < e.a.x))) ++ra;
        }
        if (leaves) {
            S.leave[rl] = e.a.x - base;
            S.leaveCell[rl] = e.a.z - cell0;
            atomicAdd(&S.nl, 1u);
        }
        if (enters) {
            S.arrive[ra] = k2 - 2u * cell0;
            S.arriveEv[ra] = tid;
            atomicAdd(&S.na, 1u);
        }
    }
    __syncthreads();
    const uint32_t nl = S.nl, na = S.na;
    if (tid < na) {
        const uint32_t k2 = S.arrive[tid], c = k2 >> 1;
        // in front of its cell's stayers, or behind them
        const uint32_t at = B.first[geo.first + (c >> geo.log2gx) * (gx + 1u) + (c & (gx - 1u)) +
                                    (k2 & 1u)] - base;
        S.arriveAt[tid] = at;
        S.arriveDst[S.arriveEv[tid]] = at - lower_count(S.leave, nl, at) + tid;
    }
    __syncthreads();
    // places outside [from, end) keep their particles
    const uint32_t from = min(nl ? S.leave[0] : cnt, na ? S.arriveAt[0] : cnt);
    const uint32_t end = nl != na ? cnt
                                  : max(nl ? S.leave[nl - 1] + 1u : 0u, na ? S.arriveAt[na - 1] : 0u);
    Held<TYPED> now[kFixItems], next[kFixItems];
    fix_load<TYPED>(B, d, S, base, cell0, from, end, nl, na, now);
    // first slots (beside the loads): one more for every arrival in a lower
    // cell, one fewer for every leaver of one
    const uint32_t words = (geo.cells >> geo.log2gx) * (gx + 1u);
    for (uint32_t k = tid; k < words; k += kFixThreads) {
        const uint32_t row = k / (gx + 1u), c = k - row;  // row * gx + column
        const uint32_t up = lower_count(S.arrive, na, 2u * c);
        const uint32_t down = lower_count(S.leaveCell, nl, c);
        if (up != down) B.first[geo.first + k] += up - down;
    }
    for (uint32_t run = from; run < end; run += kFixRun) {
        fix_load<TYPED>(B, d, S, base, cell0, run + kFixRun, end, nl, na, next);
        __syncthreads();  // this run and the next are read
#pragma unroll
        for (int u = 0; u < kFixItems; ++u) {
            const Held<TYPED>& h = now[u];
            if (h.dst != kBandEmpty && B.slotSpec) B.slotSpec[base + h.dst] = geo.spec;
            if (h.dst != kBandEmpty)
                put<TYPED>(B, d, base + h.dst, h.p, h.v, h.th, h.om, h.r, h.m, h.id, h.type, h.key,
                           h.cand);
        }
#pragma unroll
        for (int u = 0; u < kFixItems; ++u) now[u] = next[u];
    }
    __syncthreads();
    if (enters && B.slotSpec) B.slotSpec[base + S.arriveDst[tid]] = geo.spec;
    if (enters)
        put<TYPED>(B, d, base + S.arriveDst[tid], make_float2(e.b.x, e.b.y),
                   make_float2(e.b.z, e.b.w), e.c.x, e.c.y, e.c.z, e.c.w, e.a.w, e.d.x, e.a.y,
                   kCandNone);
    const uint32_t newCnt = cnt - nl + na;
    for (uint32_t j = newCnt + tid; j < cnt; j += kFixThreads) B.key[base + j] = kBandEmpty;
    if (tid == 0) {
        B.count[b] = newCnt;
        B.evCnt[b] = 0u;
    }
}

template <bool TYPED>
__global__ void __launch_bounds__(kFixThreads, 2)
band_fix_kernel(const __grid_constant__ BandArgs B, const __grid_constant__ DynSet d, uint32_t q) {
    __shared__ FixShared S;
    // left, done, full, cur; the first band of this block, if there is one
    const uint4 c = *reinterpret_cast<const uint4*>(B.ctrl);
    const uint32_t nd = min(B.ctrl[kBandDirty + q], B.bands);
    uint32_t band = blockIdx.x < B.bands ? B.dirty[q][blockIdx.x] : 0u;
    static_assert(kBandLeft == 0 && kBandFull == 2 && kBandCur == 3, "one load of 16 bytes");
    const bool active = c.x != 0u && c.w == q && c.z == 0u;
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        B.ctrl[kBandAct + q] = active ? (c.x == 1u ? 2u : 1u) : 0u;
        B.ctrl[kBandNow + q] = B.ctrl[kBandStep];
        if (active && B.bands > kFixBlocks) atomicAdd(B.ctrl + kBandDirtySum, nd);
    }
    if (!active) return;
    for (uint32_t k = blockIdx.x; k < nd; k += gridDim.x) {
        if (k != blockIdx.x) band = B.dirty[q][k];
        fix_band<TYPED>(B, d, S, band);
        __syncthreads();
    }
    // how far pairs may have approached since their bands searched, by the
    // blocks from the last on (the first ones have the events).  A pair's bands
    // are the same or beside each other, the first and the last one of a scene
    // too: a disk that left a window of rows is met across the grid's wrap, and
    // so is one pushed against the top wall whose radius the wall's height
    // swallows (Ly - r == Ly is in the row behind the last).
    for (uint32_t b = (gridDim.x - 1u - blockIdx.x) * kFixThreads + threadIdx.x; b < B.bands;
         b += gridDim.x * kFixThreads) {
        uint32_t lo = (b ? b : B.bands) - 1u, hi = b + 1u < B.bands ? b + 1u : 0u;
        if (B.table) {
            const BandGeo g = B.geo[b];
            if (b == g.sceneBand) {
                const KParams& P = B.table[g.spec];
                lo = b + (P.gx * P.gy) / g.cells - 1u;
            }
            if (hi == 0u || B.geo[hi].sceneBand == hi) hi = g.sceneBand;
        }
        const float own = __uint_as_float(B.moved[q][b]);
        // as bits, so that a NaN is the largest
        const float any = __uint_as_float(max(B.moved[q][b], max(B.moved[q][lo], B.moved[q][hi])));
        const float grown = B.grown[b] + (own + any) * 1.0001f;
        const bool keep = grown <= 0.99f * B.skin;
        B.grown[b] = keep ? grown : 0.0f;
        B.search[b] = keep ? 0u : 1u;
        B.moved[q ^ 1u][b] = 0u;  // the step of this set collects it
    }
}

// ----------------------------------------------------------------- step
// An event into band b's list; the band's first one puts it on the list of
// the next step's fix.  A full list, or no free slot for every event, asks
// for a new layout.
__device__ __forceinline__ BandEvent* push_event(const BandArgs& B, uint32_t b, uint32_t nextSet) {
    const uint32_t k = atomicAdd(B.evCnt + b, 1u);
    if (k == 0u) {
        const uint32_t w = atomicAdd(B.ctrl + kBandDirty + nextSet, 1u);
        if (w < B.bands) B.dirty[nextSet][w] = b;
    }
    uint32_t room = B.base[b + 1u] - B.base[b] - B.count[b];
    if (B.table && (B.geo[b].free & kBandWhole)) room = kBandEvents;
    if (k >= min(kBandEvents, room)) {
        B.ctrl[kBandFull] = 1u;
        return nullptr;
    }
    return B.ev + (size_t)b * kBandEvents + k;
}

// Reach of a particle's search: contacts (or attraction) plus the skin.
template <bool ATTRACT>
__device__ __forceinline__ float search_bound(float r, float rj, float skin) {
    const float d = (ATTRACT ? kAttractReach * fmaxf(r, rj) : r + rj) + skin;
    return d * d * 1.00001f;
}

// The kept candidates of a particle (see kCandNone): one bit for every
// candidate within reach plus the skin, row by row.  A cell met across the
// wrap of the grid's columns is only checked: a candidate there, as a row
// interval of more than kCandBits, keeps none.
template <bool ATTRACT>
__device__ __noinline__ unsigned long long
search_candidates(const KParams& P, uint32_t i, uint32_t key, float2 p, float r, float skin,
                  const float2* __restrict__ pos, const float* __restrict__ radius,
                  const uint32_t* __restrict__ first) {
    if (!P.cull || (ATTRACT && !(r > 0.0f))) return kCandNone;
    key -= P.cellOff;
    first += P.firstOff;
    const int gx = (int)(key & (P.gx - 1u)), gy = (int)(key >> P.log2gx);
    int y0 = -1, y1 = 1;
    if (p.y > P.cullMargin && p.y < P.Ly - P.cullMargin && p.x > P.cullMargin &&
        p.x < P.Lx - P.cullMargin) {
        const float reach =
            (ATTRACT ? kAttractReach * P.rmax : r + P.rmax) * 1.0001f + P.cullMargin + skin;
        const float Y0 = (float)(gy + P.rowOff) * P.cellH;
        if (p.y - Y0 > reach) y0 = 0;
        if (Y0 + P.cellH - p.y > reach) y1 = 0;
    }
    const int xb = max(gx - 1, 0), xe = min(gx + 1, (int)P.gx - 1);
    unsigned long long kept = 0ull;
#pragma unroll 1
    for (int dy = y0; dy <= y1; ++dy) {
        const uint32_t* __restrict__ f =
            first + (size_t)((gy + dy) & (int)(P.gy - 1u)) * (P.gx + 1u);
        const uint32_t a = __ldg(f + xb), n = __ldg(f + xe + 1) - a;
        if (n > kCandBits) return kCandNone;
        uint32_t bits = 0u;
#pragma unroll 1
        for (uint32_t k0 = 0; k0 < n; k0 += 4u) {
            float2 q[4];
            float rq[4];
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                q[k] = __ldg(pos + (a + k0 + k));
                rq[k] = __ldg(radius + (a + k0 + k));
            }
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                const float dx = q[k].x - p.x, dy2 = q[k].y - p.y;
                if (dx * dx + dy2 * dy2 <= search_bound<ATTRACT>(r, rq[k], skin))
                    bits |= 1u << (k0 + k);
            }
        }
        bits &= (1u << n) - 1u;  // groups are read whole
        if (i - a < n) bits &= ~(1u << (i - a));
        kept |= (unsigned long long)bits << (kCandBits * (uint32_t)(dy + 1));
        if (xe - xb != 2) {
            const int w = gx == 0 ? (int)P.gx - 1 : 0;
            for (uint32_t j = __ldg(f + w), e = __ldg(f + w + 1); j < e; ++j) {
                const float2 q = __ldg(pos + j);
                const float dx = q.x - p.x, dy2 = q.y - p.y;
                if (dx * dx + dy2 * dy2 <= search_bound<ATTRACT>(r, __ldg(radius + j), skin))
                    return kCandNone;
            }
        }
    }
    return kept;
}

// The search and the law together, for slots that keep no candidates.
template <bool TYPED, bool ATTRACT, bool CULL>
__device__ __noinline__ Pull collide_slot(const KParams& P, const BandArgs& B, const DynSet& in,
                                          uint32_t i, uint32_t key, float2 p, float2 v, float w,
                                          float r, uint32_t mat) {
    key -= P.cellOff;
    const int2 g = make_int2((int)(key & (P.gx - 1u)), (int)(key >> P.log2gx));
    // collide_rows counts a row's words from cellOff
    const uint32_t* __restrict__ first = B.first + P.firstOff;
    Pull o;
    if (!CULL || !P.cull ||
        !collide_rows<TYPED, ATTRACT>(P, i, g, p, v, w, r, mat, in.pos, in.vel, in.omega,
                                      B.stat.radius, B.stat.type, nullptr, first - P.cellOff,
                                      P.gx + 1u, o.f, o.moment, o.pr)) {
        const RowCells cells{first, P.gx, P.log2gx, P.cellOff};
        if (CULL && !ATTRACT && P.cull)
            collide_one<TYPED, ATTRACT, CULL && !ATTRACT>(P, i, g, p, v, w, r, mat, in.pos, in.vel,
                                                          in.omega, B.stat.radius, B.stat.type,
                                                          nullptr, cells, o.f, o.moment, o.pr);
        else
            collide_one<TYPED, ATTRACT, false>(P, i, g, p, v, w, r, mat, in.pos, in.vel, in.omega,
                                               B.stat.radius, B.stat.type, nullptr, cells, o.f,
                                               o.moment, o.pr);
    }
    return o;
}

// First slot of each of the three row intervals around the cell of `key`, for
// the rows with candidates in `cand`.
struct RowBase {
    uint32_t a[3];
};
__device__ __forceinline__ const uint32_t* row_first(const KParams& P, const BandArgs& B,
                                                     uint32_t key, uint32_t row) {
    key -= P.cellOff;
    const uint32_t x = key & (P.gx - 1u), y = (key >> P.log2gx) + row - 1u;
    return B.first + P.firstOff + (size_t)(y & (P.gy - 1u)) * (P.gx + 1u) + (x ? x - 1u : 0u);
}
__device__ __forceinline__ RowBase row_bases(const KParams& P, const BandArgs& B, uint32_t key,
                                             unsigned long long cand) {
    RowBase o;
#pragma unroll
    for (uint32_t k = 0; k < 3u; ++k) {
        const uint32_t bits = (uint32_t)(cand >> (kCandBits * k)) & ((1u << kCandBits) - 1u);
        o.a[k] = bits ? __ldg(row_first(P, B, key, k)) : 0u;
    }
    return o;
}

// Forces on the particles of a warp from their kept candidates `rem` (0 for a
// lane without any), in index order, one subtotal per cell, the subtotals
// added in cell order (an empty cell adds +0).  Every lane calls it.
template <bool TYPED, bool ATTRACT, bool BATCH>
__device__ __forceinline__ void collide_warp(const KParams& P, const BandArgs& B, const DynSet& in,
                                             Deal<ATTRACT>& S, bool wantPr,
                                             unsigned long long rem,
                                             const RowBase& base, uint32_t key, uint32_t spec,
                                             float2 p, float2 v, float w, float r, uint32_t mat, Pull& o) {
    constexpr unsigned kAll = 0xffffffffu;
    const uint32_t lane = threadIdx.x & 31u;
    Sums sum;
    sum.o = o;  // of a lane that met its neighbours without kept candidates
    while (__any_sync(kAll, rem != 0ull)) {
        uint32_t at[kDeal], row[kDeal];
        float2 qp[kDeal];
        float qr[kDeal];
        unsigned have = 0u;
#pragma unroll
        for (int k = 0; k < kDeal; ++k) {
            at[k] = row[k] = 0u;
            if (rem != 0ull) {
                const uint32_t bit = (uint32_t)__ffsll((long long)rem) - 1u;
                rem &= rem - 1ull;
                row[k] = bit >= 2u * kCandBits ? 2u : (bit >= kCandBits ? 1u : 0u);
                at[k] = (row[k] == 2u ? base.a[2] : (row[k] == 1u ? base.a[1] : base.a[0])) +
                        (bit - row[k] * kCandBits);
                have |= 1u << k;
            }
            qp[k] = __ldg(in.pos + at[k]);
            qr[k] = __ldg(B.stat.radius + at[k]);
        }
        uint32_t total = 0u, cells = 0u, mine = 0u;
#pragma unroll
        for (int k = 0; k < kDeal; ++k) {
            const float dx = qp[k].x - p.x, dy = qp[k].y - p.y;
            const float d2 = dx * dx + dy * dy;
            const float cd = r + qr[k];
            // beyond: sqrtf(d2) >= cd after rounding (or both attraction
            // ranges), no force
            const bool hit = ((have >> k) & 1u) && (ATTRACT ? !attract_out_of_reach(r, qr[k], d2)
                                                            : d2 <= cd * cd * 1.000002f);
            const unsigned hits = __ballot_sync(kAll, hit);
            if (hit) {
                const uint32_t* __restrict__ f = row_first(P, B, key, row[k]);
                S.j[k * 32 + lane] = at[k];
                S.code[total + __popc(hits & ((1u << lane) - 1u))] = (uint8_t)(k * 32 + lane);
                cells |= (3u * row[k] + (at[k] >= __ldg(f + 1) ? 1u : 0u) +
                          (at[k] >= __ldg(f + 2) ? 1u : 0u)) << (4 * k);
                mine |= 1u << k;
            }
            total += (uint32_t)__popc(hits);
        }
        if (total == 0u) continue;
        deal_law<TYPED, ATTRACT>(P, BATCH ? B.table : nullptr, spec, S, wantPr, total, mine, cells,
                                 p, v, w, r, mat, in.pos, in.vel, in.omega, B.stat.radius,
                                 B.stat.type, nullptr, sum);
    }
    o = sum.close();
}

// BATCH: the parameters are those of the slot's specimen (P0's only choose the
// kernel).
template <bool TYPED, bool ATTRACT, bool CULL, bool BATCH, bool CONTROL, int THREADS, int MINB>
__global__ void __launch_bounds__(THREADS, MINB)
band_step_kernel(const __grid_constant__ KParams P0, const __grid_constant__ BandArgs B,
                 const __grid_constant__ DynSet in, const __grid_constant__ DynSet out, uint32_t q,
                 uint32_t everyStep, ControlArgs ctl) {
    __shared__ Deal<ATTRACT> deal[CULL ? THREADS / 32 : 1];
    const uint32_t act = B.ctrl[kBandAct + q], now = B.ctrl[kBandNow + q];
    const uint32_t slot = blockIdx.x * THREADS + threadIdx.x;
    // the lanes past the last slot stand by as copies of it
    const uint32_t i = min(slot, B.slots - 1u);
    const uint32_t key = B.key[i];
    const uint32_t spec = BATCH ? B.slotSpec[i] : 0u;
    const KParams& P = BATCH ? B.table[spec] : P0;
    Dyn s;
    s.p = in.pos[i];
    const float r = B.stat.radius[i];
    s.v = in.vel[i];
    s.w = in.omega[i];
    s.th = in.theta[i];
    const float m = B.stat.mass[i];
    const uint32_t mat = TYPED ? B.stat.type[i] : 0u;
    unsigned long long cand = CULL ? B.cand[i] : kCandNone;
    if (act == 0u) return;
    if (slot == 0u) {
        B.ctrl[kBandCur] = q ^ 1u;
        B.ctrl[kBandLeft] -= 1u;
        B.ctrl[kBandDone] += 1u;
        B.ctrl[kBandStep] = now + 1u;
        B.ctrl[kBandDirty + q] = 0u;  // taken by the fix before this kernel
        // a sort whose wait gave up left no order to build on
        if (*B.errFlag & kSortTimeoutBit) B.ctrl[kBandFull] = 1u;
    }
    const bool mine = slot < B.slots && key != kBandEmpty;
    // the next step overwrites the pressure and the accelerations: only the
    // call's last step makes and stores them
    const bool store = act == 2u || everyStep;
    if (!__any_sync(0xffffffffu, mine)) return;
    Pull o{make_float2(0.0f, 0.0f), 0.0f, 0.0f};
    RowBase base{};
    uint32_t b0 = 0u;  // the slot's band
    if (!mine) {
        cand = 0ull;
    } else {
        b0 = band_of(B, key);
        // one round of loads: whether to search, and the rows of the candidates
        // kept so far.  A cell stamped in the step before (`now`) may have been
        // stamped again by a block of this step (`now` + 1).
        if (CULL) base = row_bases(P, B, key, cand & kCandNone ? 0ull : cand);
        if (CULL && ((cand & kCandNone) || B.stamp[key] - now <= 1u || B.search[b0])) {
            cand = search_candidates<ATTRACT>(P, i, key, s.p, r, B.skin, in.pos, B.stat.radius,
                                              B.first);
            B.cand[i] = cand;
            base = row_bases(P, B, key, cand & kCandNone ? 0ull : cand);
        }
        if (cand & kCandNone) {
            o = collide_slot<TYPED, ATTRACT, CULL>(P, B, in, i, key, s.p, s.v, s.w, r, mat);
            cand = 0ull;
        }
    }
    if (CULL)
        collide_warp<TYPED, ATTRACT, BATCH>(P, B, in, deal[threadIdx.x >> 5], store && B.pressure,
                                            cand, base, key, spec, s.p, s.v, s.w, r, mat, o);
    if (!mine) return;
    if (CONTROL)
        // (within n, also after a sort whose wait gave up)
        meet_control<TYPED, ATTRACT>(P, ctl, min(i - B.gap[b0], B.n - 1u), s.p, s.v, s.w, r, mat,
                                     o.f, o.moment, o.pr);
    // F/m and M/I as the reference divides them; without contacts both are
    // exactly +0 (see finish_particle)
    const bool quiet =
        o.f.x == 0.0f && o.f.y == 0.0f && o.moment == 0.0f && m > 0.0f && m < INFINITY;
    const float two_mrr = 2.0f * m * r * r;
    float2 a = make_float2(0.0f, 0.0f);
    float al = 0.0f;
    if (!(quiet && two_mrr >= 1e-30f && two_mrr <= 1e30f)) {
        a = make_float2(o.f.x / m, o.f.y / m);
        al = o.moment / inertia_of(m, r);
    }
    const float2 was = s.p;
    integrate_one(P, s, a, al, r, m, mat, o.pr);
    out.pos[i] = s.p;
    out.vel[i] = s.v;
    out.theta[i] = s.th;
    out.omega[i] = s.w;
    if (store) {
        if (B.pressure) B.pressure[i] = o.pr;
        if (B.acc) {
            B.acc[i] = a;
            B.alpha[i] = al;
        }
    }
    if (!(isfinite(s.p.x) && isfinite(s.p.y))) atomicOr(B.errFlag, 1u);
    if (CULL) {
        // the band's largest displacement, one atomic a warp while it grows
        uint32_t far = __float_as_uint(fabsf(s.p.x - was.x) + fabsf(s.p.y - was.y)) & 0x7fffffffu;
        const unsigned lanes = __activemask();
        if (__all_sync(lanes, b0 == __shfl_sync(lanes, b0, __ffs(lanes) - 1))) {
            far = __reduce_max_sync(lanes, far);
            if ((threadIdx.x & 31u) != (uint32_t)(__ffs(lanes) - 1)) far = 0u;
        }
        if (far) atomicMax(B.moved[q ^ 1u] + b0, far);
    }
    const int2 gn = grid_pos_fast(P, s.p);
    const uint32_t nk = grid_hash(P, gn.x, gn.y);
    if (nk != key) {
        B.key[i] = nk;
        const uint32_t b1 = band_of(B, nk);
        const uint32_t id = B.stat.id[i];
        BandEvent* e = push_event(B, b1, q ^ 1u);
        if (e) {
            e->a = make_uint4(i, nk, key, id);
            e->b = make_float4(s.p.x, s.p.y, s.v.x, s.v.y);
            e->c = make_float4(s.th, s.w, r, m);
            e->d = make_uint4(mat, 0u, 0u, 0u);
        }
        if (b0 != b1) {
            e = push_event(B, b0, q ^ 1u);
            if (e) e->a = make_uint4(i, nk, key, id);
        }
        // row intervals around both cells change: the slots there search anew
        if (CULL) {
#pragma unroll 1
            for (int k = 0; k < 18; ++k) {
                const uint32_t c = (k < 9 ? key : nk) - P.cellOff;
                const int x = (int)(c & (P.gx - 1u)) + k % 3 - 1;
                const int y = (int)(c >> P.log2gx) + k / 3 % 3 - 1;
                B.stamp[cell_index(P, x, y)] = now + 1u;
            }
        }
    }
}

// --------------------------------------------------------- pack, layout
constexpr int kPackThreads = 256;

// One block: base less the running count of every band.
constexpr int kGapThreads = 1024;
__global__ void __launch_bounds__(kGapThreads) band_gap_kernel(BandArgs B) {
    __shared__ uint32_t warpTot[kGapThreads / 32];
    const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    uint32_t carry = 0u;
    for (uint32_t b0 = 0; b0 < B.bands; b0 += kGapThreads) {
        const uint32_t b = b0 + threadIdx.x;
        const uint32_t v = b < B.bands ? B.count[b] : 0u;
        uint32_t x = v;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t y = __shfl_up_sync(0xffffffffu, x, o);
            if (lane >= (uint32_t)o) x += y;
        }
        if (lane == 31u) warpTot[warp] = x;
        __syncthreads();
        uint32_t below = carry, all = 0u;
        for (uint32_t k = 0; k < (uint32_t)kGapThreads / 32u; ++k) {
            if (k < warp) below += warpTot[k];
            all += warpTot[k];
        }
        if (b < B.bands) B.gap[b] = B.base[b] - (below + x - v);
        carry += all;
        __syncthreads();
    }
}

// Packed slot of band b's first particle: those of its scene's or specimen's
// bands below it are counted (every thread gets the sum).
__device__ __forceinline__ uint32_t packed_base(const BandArgs& B, uint32_t b, const BandGeo& geo) {
    __shared__ uint32_t warpSum[kPackThreads / 32];
    uint32_t v = threadIdx.x == 0 ? geo.scenePart : 0u;
    for (uint32_t k = geo.sceneBand + threadIdx.x; k < b; k += kPackThreads) v += B.count[k];
    v = __reduce_add_sync(0xffffffffu, v);
    if ((threadIdx.x & 31u) == 0) warpSum[threadIdx.x >> 5] = v;
    __syncthreads();
    uint32_t t = 0;
#pragma unroll
    for (int w = 0; w < kPackThreads / 32; ++w) t += warpSum[w];
    return t;
}

// Blocks (band, share): share y of the band's particles.  Bound by DRAM: 40 B
// in and 44 B out per particle.
template <bool TYPED>
__global__ void __launch_bounds__(kPackThreads)
band_pack_kernel(BandArgs B, PackedState o, uint32_t stateOnly) {
    if (B.ctrl[kBandLaid] == 0u) return;
    const uint32_t b = blockIdx.x;
    if (!stateOnly && b == 0u && blockIdx.y == 0u && threadIdx.x == 0u) {
        // a write to host memory costs the call 4 us: only the news is written
        const uint32_t steps = B.ctrl[kBandDone], layouts = B.ctrl[kBandLayouts];
        if (steps && B.load &&
            (band_overload(B.bands, B.ctrl[kBandDirtySum] / steps) ||
             (layouts > 1u && 4u * layouts >= steps)))
            *reinterpret_cast<volatile uint32_t*>(&B.load->busy) = 1u;
        B.ctrl[kBandDirtySum] = B.ctrl[kBandLayouts] = 0u;
    }
    const uint32_t base = B.base[b], cnt = B.count[b];
    const uint32_t to = packed_base(B, b, B.geo[b]);
    const bool one = B.ctrl[kBandCur] != 0u;
    const float2* __restrict__ pos = one ? B.dyn[1].pos : B.dyn[0].pos;
    const float2* __restrict__ vel = one ? B.dyn[1].vel : B.dyn[0].vel;
    const float* __restrict__ theta = one ? B.dyn[1].theta : B.dyn[0].theta;
    const float* __restrict__ omega = one ? B.dyn[1].omega : B.dyn[0].omega;
    // two particles a thread in flight
    const uint32_t step = gridDim.y * kPackThreads;
    for (uint32_t k = blockIdx.y * kPackThreads + threadIdx.x; k < cnt; k += 2u * step) {
        float2 p[2], v[2], ac[2];
        float th[2], om[2], r[2], m[2], pr[2], al[2];
        uint32_t id[2], type[2];
#pragma unroll
        for (int u = 0; u < 2; ++u) {
            // out of range only after a sort whose wait gave up
            const uint32_t s = min(base + min(k + (uint32_t)u * step, cnt - 1u), B.slots - 1u);
            p[u] = pos[s];
            v[u] = vel[s];
            th[u] = theta[s];
            om[u] = omega[s];
            r[u] = B.stat.radius[s];
            m[u] = B.stat.mass[s];
            id[u] = B.stat.id[s];
            if (TYPED) type[u] = B.stat.type[s];
            if (!stateOnly) {
                pr[u] = B.pressure ? B.pressure[s] : 0.0f;
                if (B.acc) {
                    ac[u] = B.acc[s];
                    al[u] = B.alpha[s];
                }
            }
        }
#pragma unroll
        for (int u = 0; u < 2; ++u) {
            const uint32_t i = to + k + (uint32_t)u * step;
            if (k + (uint32_t)u * step >= cnt || i >= B.n) break;
            o.dyn.pos[i] = p[u];
            o.dyn.vel[i] = v[u];
            o.dyn.theta[i] = th[u];
            o.dyn.omega[i] = om[u];
            o.stat.radius[i] = r[u];
            o.stat.mass[i] = m[u];
            o.stat.id[i] = id[u];
            if (TYPED) o.stat.type[i] = type[u];
            if (stateOnly) continue;
            o.loc[id[u]] = i;
            if (B.pressure) o.pressure[i] = pr[u];
            if (B.acc) {
                o.acc[i] = ac[u];
                o.alpha[i] = al[u];
            }
        }
    }
}

// Packed range of the band's cell c, the slots of the band `down` above their
// packed places (within n, also after a sort whose wait gave up).
__device__ __forceinline__ uint2 packed_cell(const BandArgs& B, const BandGeo& geo, uint32_t c,
                                             uint32_t down) {
    const uint32_t* f = B.first + geo.first + (c >> geo.log2gx) * ((1u << geo.log2gx) + 1u) +
                        (c & ((1u << geo.log2gx) - 1u));
    return make_uint2(min(f[0] - down, B.n), min(f[1] - down, B.n));
}

// Blocks (band, share), as band_pack_kernel: the state the step of set q
// stepped (its set is intact, its slots move only in the next fix) and the
// accelerations it stored.
__global__ void __launch_bounds__(kPackThreads)
band_record_kernel(BandArgs B, DynSet d, uint32_t q, StepRec rec, size_t stride) {
    if (B.ctrl[kBandAct + q] == 0u) return;
    const StepRec r = rec_shifted(rec, B.ctrl[kBandDone] - 1u, stride);
    const uint32_t b = blockIdx.x;
    const uint32_t base = B.base[b], cnt = B.count[b];
    const BandGeo geo = B.geo[b];
    const uint32_t to = packed_base(B, b, geo);
    const uint32_t t0 = blockIdx.y * kPackThreads + threadIdx.x, step = gridDim.y * kPackThreads;
    for (uint32_t k = t0; k < cnt; k += step) {
        const uint32_t s = base + k, i = to + k;
        // out of range only after a sort whose wait gave up
        if (s >= B.slots || i >= B.n) break;
        r.pos[i] = d.pos[s];
        r.vel[i] = d.vel[s];
        r.omega[i] = d.omega[s];
        r.radius[i] = B.stat.radius[s];
        r.mass[i] = B.stat.mass[s];
        r.id[i] = B.stat.id[s];
        r.acc[i] = B.acc[s];
        r.alpha[i] = B.alpha[s];
    }
    for (uint32_t c = t0; c < geo.cells; c += step)
        r.cells[geo.cell0 + c] = packed_cell(B, geo, c, base - to);
}

// First particle of every cell in the sorted keys (lower bounds).
__global__ void band_cell_first_kernel(const uint32_t* __restrict__ keys, uint32_t n,
                                       uint32_t cells, uint32_t* __restrict__ first) {
    for (uint32_t c = blockIdx.x * blockDim.x + threadIdx.x; c <= cells;
         c += gridDim.x * blockDim.x)
        first[c] = lower_count(keys, n, c);
}

// A block per band: its base, count and first slots from the packed
// first-particle array f; its empty slots; its counters.  A sort whose wait
// gave up leaves keys in no order: a band may then count slots that
// band_spread_kernel does not fill.  Those hold an id and a type that exist,
// so that whoever indexes with them stays within the arrays.
__global__ void __launch_bounds__(kPackThreads)
band_layout_kernel(BandArgs B, const uint32_t* __restrict__ f) {
    const uint32_t b = blockIdx.x, tid = threadIdx.x;
    const BandGeo geo = B.geo[b];
    const uint32_t p = f[geo.cell0], e = f[geo.cell0 + geo.cells];
    const uint32_t before = free_before(B, b);
    const uint32_t base = min(p + before, B.slots);
    // e < p only after a sort whose wait gave up
    if (tid == 0) {
        B.base[b] = base;
        if (b == B.bands - 1u) B.base[B.bands] = B.slots;
        B.count[b] = e > p ? e - p : 0u;
        B.evCnt[b] = 0u;
        B.moved[0][b] = B.moved[1][b] = 0u;
        B.grown[b] = 0.0f;  // no slot keeps candidates: every one searches
    }
    for (uint32_t s = b * kPackThreads + tid; s < B.slots; s += B.bands * kPackThreads) {
        B.key[s] = kBandEmpty;
        B.stat.id[s] = 0u;
        if (B.stat.type) B.stat.type[s] = 0u;
        if (B.slotSpec) B.slotSpec[s] = 0u;
    }
    const uint32_t gx = 1u << geo.log2gx, words = (geo.cells >> geo.log2gx) * (gx + 1u);
    for (uint32_t k = tid; k < words; k += kPackThreads) {
        const uint32_t row = k / (gx + 1u), x = k - row * (gx + 1u);
        B.first[geo.first + k] = f[geo.cell0 + row * gx + x] + before;
    }
}

__global__ void __launch_bounds__(kPackThreads) band_cell_table_kernel(BandArgs B) {
    const BandGeo geo = B.geo[blockIdx.x];
    for (uint32_t c = threadIdx.x; c < geo.cells; c += kPackThreads)
        B.cellBand[geo.cell0 + c] = blockIdx.x;
}

// See launch_band_estimate.  Bound by DRAM: position and velocity, 16 B a
// particle (16 M of them 55 us, the sixteenth that is looked at 4).
__global__ void __launch_bounds__(kPackThreads)
band_estimate_kernel(const __grid_constant__ KParams P0, BandArgs B, const float2* __restrict__ pos,
                     const float2* __restrict__ vel, const uint32_t* __restrict__ spec, uint32_t n,
                     uint32_t stride, uint32_t serial, uint32_t* __restrict__ out) {
    const uint32_t i = blockIdx.x * stride * kPackThreads + threadIdx.x;
    bool moves = false;
    if (i < n) {
        const KParams& P = spec ? B.table[spec[i]] : P0;
        const float2 p = pos[i], v = vel[i];
        const int2 g0 = grid_pos_fast(P, p);
        const int2 g1 = grid_pos_fast(P, make_float2(p.x + v.x * P.dt, p.y + v.y * P.dt));
        const uint32_t c[2] = {grid_hash(P, g0.x, g0.y), grid_hash(P, g1.x, g1.y)};
        moves = c[0] != c[1];
        for (int k = 0; k < 2 && moves; ++k) {
            uint32_t* m = B.mark + band_of(B, c[k]);
            if (*reinterpret_cast<volatile uint32_t*>(m) != serial &&
                atomicExch(m, serial) != serial)
                atomicAdd(out, 1u);
        }
    }
    const unsigned all = __ballot_sync(0xffffffffu, moves);
    if ((threadIdx.x & 31u) == 0u && all) atomicAdd(out + 1, (uint32_t)__popc(all));
}

// The packed particles, in sorted order, into the slots of the current set.
template <bool TYPED>
__global__ void __launch_bounds__(kPackThreads)
band_spread_kernel(BandArgs B, PackedState in, const uint32_t* __restrict__ keys,
                   const uint32_t* __restrict__ from) {
    const uint32_t i = blockIdx.x * kPackThreads + threadIdx.x;
    if (i == 0u) {
        if (B.ctrl[kBandLaid]) B.ctrl[kBandLayouts] += 1u;
        B.ctrl[kBandFull] = 0u;
        B.ctrl[kBandLaid] = 1u;
        B.ctrl[kBandDirty] = 0u;
        B.ctrl[kBandDirty + 1u] = 0u;
    }
    if (i >= B.n) return;
    // in range unless a wait of the sort gave up (stale words)
    const uint32_t key = min(keys[i], B.cells - 1u), src = min(from[i], B.n - 1u);
    const uint32_t band = band_of(B, key), s = i + free_before(B, band);
    // a specimen's slots are its own: the fixes keep within a band
    if (B.slotSpec) B.slotSpec[s] = B.geo[band].spec;
    const bool one = B.ctrl[kBandCur] != 0u;
    const DynSet d{one ? B.dyn[1].pos : B.dyn[0].pos, one ? B.dyn[1].vel : B.dyn[0].vel,
                   one ? B.dyn[1].theta : B.dyn[0].theta, one ? B.dyn[1].omega : B.dyn[0].omega};
    put<TYPED>(B, d, s, in.dyn.pos[src], in.dyn.vel[src], in.dyn.theta[src],
               in.dyn.omega[src], in.stat.radius[src], in.stat.mass[src], in.stat.id[src],
               TYPED ? in.stat.type[src] : 0u, key, kCandNone);
}

// Blocks (band): packed (start, end) of every cell and first-particle array.
__global__ void __launch_bounds__(kPackThreads)
band_cells_kernel(BandArgs B, uint2* __restrict__ cells, uint32_t* __restrict__ first) {
    if (B.ctrl[kBandLaid] == 0u) return;
    const uint32_t b = blockIdx.x;
    const BandGeo geo = B.geo[b];
    const uint32_t shiftDown = B.base[b] - packed_base(B, b, geo);
    for (uint32_t k = threadIdx.x; k < geo.cells; k += kPackThreads) {
        const uint32_t c = geo.cell0 + k;
        const uint2 r = packed_cell(B, geo, k, shiftDown);
        first[c] = r.x;
        cells[c] = r.x < r.y ? r : make_uint2(kEmptyCell, kEmptyCell);
        if (c == B.cells - 1u) first[B.cells] = r.y;
    }
}

__global__ void band_followed_kernel(BandArgs B, DynSet d, uint32_t q,
                                     const uint32_t* __restrict__ ids,
                                     const uint32_t* __restrict__ countWord,
                                     float* __restrict__ ring) {
    if (B.ctrl[kBandAct + q] == 0u) return;
    const uint32_t count = *countWord;
    float* base = ring + (size_t)(B.ctrl[kBandDone] - 1u) * count * 12;
    for (uint32_t k = blockIdx.x * blockDim.x + threadIdx.x; k < count;
         k += gridDim.x * blockDim.x)
        // (an id that a sort whose wait gave up has lost keeps an old place, or none)
        followed_row(min(B.loc[ids[k]], B.slots - 1u), base + 12ull * k, d, B.stat, B.acc, B.alpha,
                     B.pressure);
}

// ---------------------------------------------------------- conditions
__global__ void band_head_kernel(uint32_t* __restrict__ ctrl, cudaGraphConditionalHandle full,
                                 cudaGraphConditionalHandle loop, int setLoop) {
    cudaGraphSetConditional(full, ctrl[kBandFull] ? 1u : 0u);
    if (setLoop) cudaGraphSetConditional(loop, ctrl[kBandLeft] ? 1u : 0u);
}
__global__ void band_next_kernel(uint32_t* __restrict__ ctrl, cudaGraphConditionalHandle loop,
                                 int whileFull) {
    const bool go = ctrl[kBandLeft] != 0u && (whileFull || ctrl[kBandFull] == 0u);
    cudaGraphSetConditional(loop, go ? 1u : 0u);
}

bool attracts(const KParams& P) {
    for (uint32_t m = 0; m < P.nmat; ++m)
        if (P.at[m] != 0.0f) return true;
    return false;
}

}  // namespace

bool band_shape(KParams* P, uint32_t grids, const uint32_t* partOff, BandArgs& b,
                std::vector<BandGeo>& geo) {
    const bool batch = partOff != nullptr;
    geo.clear();
    uint64_t cell = 0, first = 0, free = 0;
    for (uint32_t s = 0; s < grids; ++s) {
        const uint32_t part = batch ? partOff[s] : 0u;
        const uint32_t count = batch ? partOff[s + 1] - part : 0u;
        const uint32_t gx = P[s].gx, cells = P[s].gx * P[s].gy;
        if (gx > kBandMaxRow) return false;
        uint32_t per = std::max(batch ? kBandBatchCells : kBandMinCells, gx);
        while (!batch && (uint64_t)per * kBandMaxBands < cells) per <<= 1;
        per = std::min(per, cells);  // both powers of two
        P[s].firstOff = (uint32_t)first;
        const uint32_t sceneBand = (uint32_t)geo.size(), bands = cells / per;
        const uint32_t slack = bands == 1u ? 0u : std::max(kBandMinSlack, count / (16u * bands));
        for (uint32_t c = 0; c < cells; c += per) {
            geo.push_back(BandGeo{(uint32_t)cell + c, per, (uint32_t)(first + (c / gx) * (gx + 1ull)),
                                  P[s].log2gx, sceneBand, part, s,
                                  (uint32_t)free | (bands == 1u ? kBandWhole : 0u)});
            free += slack;
        }
        b.shift = 0;
        while ((1u << b.shift) < per) ++b.shift;
        cell += cells;
        first += (uint64_t)P[s].gy * (gx + 1ull);
        if (first >= (1ull << 32) || free >= kBandWhole) return false;
    }
    b.batchFree = batch ? (uint32_t)free : 0u;
    b.cells = (uint32_t)cell;
    b.firstWords = (uint32_t)first;
    b.bands = (uint32_t)geo.size();
    return b.bands != 0;
}

uint32_t band_slack(const BandArgs& b, uint32_t n) {
    return std::max(kBandMinSlack, n / (16u * b.bands));
}
size_t band_slots(const BandArgs& b, uint32_t n, bool batch) {
    return (size_t)n + (batch ? b.batchFree : (size_t)b.bands * band_slack(b, n));
}

namespace {
// The arrays in order: take(bytes) gives each one's address.
template <typename Take>
void band_arrays(BandArgs& b, uint32_t capacity, bool typed, bool pressure, bool accel, bool batch,
                 Take take) {
    const size_t S = band_slots(b, capacity, batch) + kFilterPad;
    for (int k = 0; k < 2; ++k) {
        b.dyn[k].pos = static_cast<float2*>(take(8 * S));
        b.dyn[k].vel = static_cast<float2*>(take(8 * S));
        b.dyn[k].theta = static_cast<float*>(take(4 * S));
        b.dyn[k].omega = static_cast<float*>(take(4 * S));
    }
    b.stat.radius = static_cast<float*>(take(4 * S));
    b.stat.mass = static_cast<float*>(take(4 * S));
    b.stat.id = static_cast<uint32_t*>(take(4 * S));
    b.stat.type = typed ? static_cast<uint32_t*>(take(4 * S)) : nullptr;
    b.key = static_cast<uint32_t*>(take(4 * S));
    b.loc = static_cast<uint32_t*>(take(4ull * capacity));
    b.first = static_cast<uint32_t*>(take(4 * (b.firstWords + 4ull)));
    b.geo = static_cast<const BandGeo*>(take(sizeof(BandGeo) * (size_t)b.bands));
    if (batch) {
        b.cellBand = static_cast<uint32_t*>(take(4ull * b.cells));
        b.slotSpec = static_cast<uint32_t*>(take(4 * S));
    }
    b.base = static_cast<uint32_t*>(take(4ull * (b.bands + 1)));
    b.count = static_cast<uint32_t*>(take(4ull * b.bands));
    b.gap = static_cast<uint32_t*>(take(4ull * b.bands));
    b.evCnt = static_cast<uint32_t*>(take(4ull * b.bands));
    b.ev = static_cast<BandEvent*>(take(sizeof(BandEvent) * (size_t)b.bands * kBandEvents));
    for (int k = 0; k < 2; ++k) b.dirty[k] = static_cast<uint32_t*>(take(4ull * b.bands));
    b.cand = static_cast<unsigned long long*>(take(8 * S));
    b.stamp = static_cast<uint32_t*>(take(4ull * b.cells));
    for (int k = 0; k < 2; ++k) b.moved[k] = static_cast<uint32_t*>(take(4ull * b.bands));
    b.grown = static_cast<float*>(take(4ull * b.bands));
    b.search = static_cast<uint32_t*>(take(4ull * b.bands));
    b.ctrl = static_cast<uint32_t*>(take(4 * kBandCtrlWords));
    b.mark = static_cast<uint32_t*>(take(4ull * b.bands));
    b.pressure = pressure ? static_cast<float*>(take(4 * S)) : nullptr;
    b.acc = accel ? static_cast<float2*>(take(8 * S)) : nullptr;
    b.alpha = accel ? static_cast<float*>(take(4 * S)) : nullptr;
}
}  // namespace

size_t band_bytes(const BandArgs& b, uint32_t capacity, bool typed, bool pressure, bool accel,
                  bool batch) {
    BandArgs t = b;
    size_t total = 0;
    band_arrays(t, capacity, typed, pressure, accel, batch, [&](size_t bytes) -> void* {
        total += al256(bytes);
        return nullptr;
    });
    return total;
}

void carve_bands(BandArgs& b, void* base, uint32_t capacity, bool typed, bool pressure, bool accel,
                 bool batch) {
    char* p = static_cast<char*>(base);
    band_arrays(b, capacity, typed, pressure, accel, batch, [&](size_t bytes) -> void* {
        char* q = p;
        p += al256(bytes);
        return q;
    });
}

cudaError_t launch_band_cell_table(const BandArgs& b, cudaStream_t st) {
    band_cell_table_kernel<<<b.bands, kPackThreads, 0, st>>>(b);
    return cudaGetLastError();
}

cudaError_t launch_band_estimate(const KParams& P, const BandArgs& b, const float2* pos,
                                 const float2* vel, const uint32_t* spec, uint32_t n,
                                 uint32_t serial, uint32_t* out, cudaStream_t st) {
    if (n == 0) return cudaSuccess;
    const uint32_t stride = band_estimate_stride(n), all = blocks_for(n, kPackThreads);
    band_estimate_kernel<<<(all + stride - 1u) / stride, kPackThreads, 0, st>>>(
        P, b, pos, vel, spec, n, stride, serial, out);
    return cudaGetLastError();
}

cudaError_t launch_band_fix(const BandArgs& b, int q, cudaStream_t st) {
    const unsigned blocks = std::min(b.bands, kFixBlocks);
    if (b.stat.type)
        band_fix_kernel<true><<<blocks, kFixThreads, 0, st>>>(b, b.dyn[q], (uint32_t)q);
    else
        band_fix_kernel<false><<<blocks, kFixThreads, 0, st>>>(b, b.dyn[q], (uint32_t)q);
    return cudaGetLastError();
}

cudaError_t launch_band_gaps(const BandArgs& b, cudaStream_t st) {
    band_gap_kernel<<<1, kGapThreads, 0, st>>>(b);
    return cudaGetLastError();
}

// From about this many slots on (80 B each against 126 MB of L2) a step reads its
// state from DRAM, and ten blocks of 48 registers a multiprocessor hide more of
// that than eight of 64 lose to spills: 154.8 -> 145.9 us a step at 4,194,304
// disks, 65.4 -> 63.6 at 1,500,000, 343 -> 327 for 4,096 specimens, but 47.7 -> 48.5
// at 1,100,001 and 13.7 -> 14.4 at 65,536.  Attraction spills more (450 -> 472 at
// 4,000,003).
constexpr uint32_t kFarSlots = 5u << 18;

cudaError_t launch_band_step(const KParams& P, const BandArgs& b, int q, bool everyStep,
                             int variant, ControlArgs ctl, cudaStream_t st) {
    if (variant < 0 || variant >= kStepVariants) return cudaErrorInvalidValue;
    const bool typed = b.stat.type != nullptr && P.nmat > 1;
    const bool attract = attracts(P), batch = b.table != nullptr;
    const bool cull = batch || P.cull != 0u;  // a specimen without culling searches in full
    const DynSet in = b.dyn[q], out = b.dyn[q ^ 1];
    const uint32_t e = everyStep ? 1u : 0u;
    const bool far = !attract && b.slots >= kFarSlots;
#define DEM_BAND_T(T, A, C, TH, MB)                                                            \
    do {                                                                                       \
        const unsigned g = blocks_for(b.slots, TH);                                            \
        if (batch)                                                                             \
            band_step_kernel<T, A, true, true, false, TH, MB><<<g, TH, 0, st>>>(               \
                P, b, in, out, (uint32_t)q, e, ctl);                                           \
        else if (ctl.c)                                                                        \
            band_step_kernel<T, A, C, false, true, 128, 8>                                     \
                <<<blocks_for(b.slots, 128), 128, 0, st>>>(P, b, in, out, (uint32_t)q, e, ctl); \
        else                                                                                   \
            band_step_kernel<T, A, C, false, false, TH, MB><<<g, TH, 0, st>>>(                 \
                P, b, in, out, (uint32_t)q, e, ctl);                                           \
    } while (0)
#define DEM_BAND(T, A, C)                                    \
    do {                                                     \
        switch (variant) {                                   \
            case 1: DEM_BAND_T(T, A, C, 64, 16); break;      \
            case 2: DEM_BAND_T(T, A, C, 256, 4); break;      \
            case 3: DEM_BAND_T(T, A, C, 128, 6); break;      \
            default:                                         \
                if (far) DEM_BAND_T(T, A, C, 128, ((A) ? 8 : 10)); \
                else DEM_BAND_T(T, A, C, 128, 8);            \
                break;                                       \
        }                                                    \
    } while (0)
#define DEM_BAND_AC(T)                                  \
    do {                                                \
        if (attract && cull) DEM_BAND(T, true, true);   \
        else if (attract) DEM_BAND(T, true, false);     \
        else if (cull) DEM_BAND(T, false, true);        \
        else DEM_BAND(T, false, false);                 \
    } while (0)
    if (typed) DEM_BAND_AC(true);
    else DEM_BAND_AC(false);
#undef DEM_BAND_AC
#undef DEM_BAND
#undef DEM_BAND_T
    return cudaGetLastError();
}

cudaError_t launch_band_followed(const BandArgs& b, int q, const uint32_t* ids,
                                 const uint32_t* countWord, float* ring, cudaStream_t st) {
    band_followed_kernel<<<16, 128, 0, st>>>(b, b.dyn[q ^ 1], (uint32_t)q, ids, countWord, ring);
    return cudaGetLastError();
}

cudaError_t launch_band_pack(const BandArgs& b, const PackedState& out, bool stateOnly,
                             cudaStream_t st) {
    // enough blocks to fill the GPU, a share of a band each
    const dim3 grid(b.bands, std::max(1u, 1184u / b.bands));
    if (b.stat.type)
        band_pack_kernel<true><<<grid, kPackThreads, 0, st>>>(b, out, stateOnly ? 1u : 0u);
    else
        band_pack_kernel<false><<<grid, kPackThreads, 0, st>>>(b, out, stateOnly ? 1u : 0u);
    return cudaGetLastError();
}

cudaError_t launch_band_record(const BandArgs& b, int q, void* recBase, size_t stride,
                               cudaStream_t st) {
    const dim3 grid(b.bands, std::max(1u, 592u / b.bands));
    band_record_kernel<<<grid, kPackThreads, 0, st>>>(b, b.dyn[q], (uint32_t)q,
                                                      carve_step(recBase, b.n, b.cells), stride);
    return cudaGetLastError();
}

cudaError_t launch_band_layout(const BandArgs& b, const PackedState& in, const uint32_t* keys,
                               const uint32_t* from, uint32_t* cellFirst, cudaStream_t st) {
    band_cell_first_kernel<<<std::min(blocks_for((size_t)b.cells + 1, kPackThreads), 1184u),
                             kPackThreads, 0, st>>>(keys, b.n, b.cells, cellFirst);
    band_layout_kernel<<<b.bands, kPackThreads, 0, st>>>(b, cellFirst);
    const unsigned g = blocks_for(b.n, kPackThreads);
    if (b.stat.type)
        band_spread_kernel<true><<<g, kPackThreads, 0, st>>>(b, in, keys, from);
    else
        band_spread_kernel<false><<<g, kPackThreads, 0, st>>>(b, in, keys, from);
    return cudaGetLastError();
}

cudaError_t launch_band_cells(const BandArgs& b, uint2* cells, uint32_t* first, cudaStream_t st) {
    band_cells_kernel<<<b.bands, kPackThreads, 0, st>>>(b, cells, first);
    return cudaGetLastError();
}

cudaError_t launch_band_head(const BandArgs& b, cudaGraphConditionalHandle full,
                             cudaGraphConditionalHandle loop, bool setLoop, cudaStream_t st) {
    band_head_kernel<<<1, 1, 0, st>>>(b.ctrl, full, loop, setLoop ? 1 : 0);
    return cudaGetLastError();
}

cudaError_t launch_band_next(const BandArgs& b, cudaGraphConditionalHandle loop, bool whileFull,
                             cudaStream_t st) {
    band_next_kernel<<<1, 1, 0, st>>>(b.ctrl, loop, whileFull ? 1 : 0);
    return cudaGetLastError();
}

}  // namespace dem
