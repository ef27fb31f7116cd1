// DEM step kernels: hash, reorder + cell ranges, collide, integrate, and the
// fused collide/integrate/hash kernel the context's step uses.
#include "dem_collide.cuh"
#include "dem_kernels.cuh"

namespace dem {
namespace {

constexpr int kThreads = 256;
constexpr int kCollideThreads = 128;

inline unsigned blocks_for(uint32_t n, int t) { return (unsigned)((n + (uint32_t)t - 1u) / (uint32_t)t); }

// particles_kernel.cuh:133-151
__global__ void __launch_bounds__(kThreads)
calc_hash_kernel(KParams P, const float2* __restrict__ pos, uint32_t* __restrict__ hash,
                 uint32_t* __restrict__ index, uint32_t n) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const int2 g = grid_pos(P, pos[i]);
    hash[i] = grid_hash(P, g.x, g.y);
    if (index) index[i] = i;
}

// calcHashD for the batched form: each slot hashes with its specimen's grid.
__global__ void __launch_bounds__(kThreads)
calc_hash_batched_kernel(const KParams* __restrict__ table, const uint32_t* __restrict__ spec,
                         const float2* __restrict__ pos, uint32_t* __restrict__ hash, uint32_t n) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const KParams& P = table[spec[i]];
    const int2 g = grid_pos(P, pos[i]);
    hash[i] = grid_hash(P, g.x, g.y);
}

// particles_kernel.cuh:156-233.  A cell starts where the sorted hash differs
// from its predecessor; the predecessor's cell ends there.  The reference
// stages hashes in shared memory; here the neighbour comes from the next lane
// by shuffle and only lane 0 reads hash[i-1] (an L1 hit).
template <bool TYPED>
__global__ void __launch_bounds__(kThreads)
reorder_kernel(uint32_t* __restrict__ cellStart, uint32_t* __restrict__ cellEnd, DynSet s,
               StatSet sS, uint32_t* __restrict__ sLoc, const uint32_t* __restrict__ hash,
               const uint32_t* __restrict__ index, DynSet o, StatSet oS, uint32_t n,
               uint32_t numCells) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    const bool valid = i < n;
    const uint32_t h = valid ? hash[i] : 0u;
    uint32_t hp = __shfl_up_sync(0xffffffffu, h, 1);
    if ((threadIdx.x & 31) == 0 && valid && i > 0) hp = hash[i - 1];
    if (!valid) return;
    // keys outside the grid or indices outside the arrays can only come from a
    // caller's own buffers; such entries are skipped rather than written
    if (i == 0 || h != hp) {
        if (h < numCells) cellStart[h] = i;
        if (i > 0 && hp < numCells) cellEnd[hp] = i;
    }
    if (i == n - 1 && h < numCells) cellEnd[h] = i + 1;
    const uint32_t src = index[i];
    if (src >= n) return;
    s.pos[i] = o.pos[src];
    s.vel[i] = o.vel[src];
    s.theta[i] = o.theta[src];
    s.omega[i] = o.omega[src];
    sS.radius[i] = oS.radius[src];
    sS.mass[i] = oS.mass[src];
    const uint32_t id = oS.id[src];
    sS.id[i] = id;
    if (id < n) sLoc[id] = i;
    if (TYPED) sS.type[i] = oS.type[src];
}

// collideD on the caller's sorted arrays and cell ranges (any ranges: nothing
// is assumed of positions and cells beyond what the reference reads).  Bound
// by issue: about 36 candidates and 3 contacts a particle in a dense packing.
// The three ranges of a cell row load together; where they follow one another,
// as sorted particles' do, they are one interval, walked eight candidates at a
// time, and the touching ones are dealt over the warp (deal_law).  1,048,576
// disks at area fraction 0.78: 143 -> about 90 us (one step through the five
// stages 193 -> 163 us).
template <bool TYPED, bool ATTRACT>
__global__ void __launch_bounds__(kCollideThreads, 8)
collide_kernel(const __grid_constant__ KParams P, const float2* __restrict__ pos,
               const float2* __restrict__ vel, const float* __restrict__ omega,
               const float* __restrict__ radius, const float* __restrict__ mass,
               const uint32_t* __restrict__ type, const uint32_t* __restrict__ cellStart,
               const uint32_t* __restrict__ cellEnd, float2* __restrict__ acc,
               float* __restrict__ alpha, float* __restrict__ pressure, uint32_t n) {
    constexpr unsigned kAll = 0xffffffffu;
    __shared__ Deal<ATTRACT> deal[kCollideThreads / 32];
    Deal<ATTRACT>& S = deal[threadIdx.x >> 5];
    const uint32_t lane = threadIdx.x & 31u;
    const uint32_t slot = blockIdx.x * blockDim.x + threadIdx.x;
    const bool mine = slot < n;
    const uint32_t i = min(slot, n - 1u);  // lanes past the end stand by
    const float2 p = pos[i];
    const float2 v = vel[i];
    const float w = omega[i];
    const float r = radius[i];
    const uint32_t mat = TYPED ? type[i] : 0u;
    int2 g = grid_pos(P, p);
    g.y -= P.rowOff;
    Sums sum;
    uint32_t held = 0u, cells = 0u, total = 0u;  // candidates of the turn
    auto flush = [&]() {
        deal_law<TYPED, ATTRACT>(P, nullptr, 0u, S, pressure != nullptr, total, (1u << held) - 1u, cells, p, v, w, r, mat, pos, vel,
                                 omega, radius, type, nullptr, sum);
        held = cells = total = 0u;
    };
#pragma unroll 1
    for (int dy = -1; dy <= 1; ++dy) {
        uint32_t s[3], e[3];
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            const uint32_t h = cell_index(P, g.x + k - 1, g.y + dy);
            s[k] = __ldg(cellStart + h);
            e[k] = __ldg(cellEnd + h);
        }
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            // an empty cell's end is unspecified; an empty range holds nothing
            if (!mine || s[k] == kEmptyCell || e[k] <= s[k]) s[k] = e[k] = 0u;
        }
        // one interval when each range that holds something starts where the
        // last one ended
        const bool h0 = e[0] != 0u, h1 = e[1] != 0u, h2 = e[2] != 0u;
        const bool joined = (!h0 || !h1 || s[1] == e[0]) &&
                            (!h2 || !(h0 || h1) || s[2] == (h1 ? e[1] : e[0]));
        const uint32_t last = h2 ? e[2] : (h1 ? e[1] : e[0]);
        const uint32_t b2 = h2 ? s[2] : last, b1 = h1 ? s[1] : b2;
#pragma unroll 1
        for (int pass = 0; pass < 3; ++pass) {
            uint32_t a = 0u, b = 0u;
            if (joined) {
                if (pass == 0) {
                    a = h0 ? s[0] : b1;
                    b = last;
                }
            } else {
                a = pass == 0 ? s[0] : (pass == 1 ? s[1] : s[2]);
                b = pass == 0 ? e[0] : (pass == 1 ? e[1] : e[2]);
            }
            if (!__any_sync(kAll, a < b)) continue;
#pragma unroll 1
            for (; __any_sync(kAll, a < b); a += 8u) {
                uint32_t hits = 0u;
                if (a < b) {
                    if (n - a >= 8u) {
                        hits = filter8<ATTRACT>(pos + a, radius + a, p, r);
                    } else {  // the arrays end within the group
                        for (uint32_t k = 0; k < n - a; ++k) {
                            const float2 q = __ldg(pos + a + k);
                            const float rq = __ldg(radius + a + k);
                            const float dx = q.x - p.x, dq = q.y - p.y;
                            const float d2 = dx * dx + dq * dq, cd = r + rq;
                            if (ATTRACT ? !attract_out_of_reach(r, rq, d2)
                                        : d2 <= cd * cd * 1.000002f)
                                hits |= 1u << k;
                        }
                    }
                    // groups are read whole
                    if (b - a < 8u) hits &= (1u << (b - a)) - 1u;
                    if (i - a < 8u) hits &= ~(1u << (i - a));
                }
                while (__any_sync(kAll, hits != 0u)) {
                    if (__any_sync(kAll, held == (uint32_t)kDeal)) flush();
                    const unsigned take = __ballot_sync(kAll, hits != 0u);
                    if (hits) {
                        const uint32_t j = a + (uint32_t)__ffs(hits) - 1u;
                        hits &= hits - 1u;
                        const uint32_t x = joined ? (j >= b1 ? 1u : 0u) + (j >= b2 ? 1u : 0u)
                                                  : (uint32_t)pass;
                        S.j[held * 32u + lane] = j;
                        S.code[total + __popc(take & ((1u << lane) - 1u))] =
                            (uint8_t)(held * 32u + lane);
                        cells |= (3u * (uint32_t)(dy + 1) + x) << (4u * held);
                        ++held;
                    }
                    total += (uint32_t)__popc(take);
                }
            }
        }
    }
    if (__any_sync(kAll, held != 0u)) flush();
    if (!mine) return;
    const Pull o = sum.close();
    const float m = mass[i];
    acc[i] = make_float2(o.f.x / m, o.f.y / m);
    alpha[i] = o.moment / inertia_of(m, r);
    if (pressure) pressure[i] = o.pr;
}

template <bool TYPED>
__global__ void __launch_bounds__(kThreads)
integrate_kernel(KParams P, float2* __restrict__ pos, float2* __restrict__ vel,
                 const float2* __restrict__ acc, float* __restrict__ theta,
                 float* __restrict__ omega, const float* __restrict__ alpha,
                 const uint32_t* __restrict__ type, const float* __restrict__ radius,
                 const float* __restrict__ mass, float* __restrict__ pressure, uint32_t n) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    Dyn s;
    s.p = pos[i];
    s.v = vel[i];
    s.th = theta[i];
    s.w = omega[i];
    float pr = pressure ? pressure[i] : 0.0f;
    const uint32_t mat = TYPED ? type[i] : 0u;
    integrate_one(P, s, acc[i], alpha[i], radius[i], mass[i], mat, pr);
    pos[i] = s.p;
    vel[i] = s.v;
    theta[i] = s.th;
    omega[i] = s.w;
    if (pressure) pressure[i] = pr;
}

// collide_one/rows/staged done: acceleration, integration, next hash, mover
// record (shared tail of step_kernel).  `m` and `s.th` were read with the
// particle's other fields before the collide, so no load waits here.
template <bool TYPED>
__device__ __forceinline__ void finish_particle(
    const KParams& P, uint32_t i, Dyn& s, float2 f, float moment, float pr, float r, float m,
    uint32_t mat, uint32_t id, uint32_t key, const uint2* __restrict__ cellRange, DynSet out,
    StatSet outS, uint32_t* __restrict__ loc, uint32_t* __restrict__ nextHash,
    float* __restrict__ pressure, float2* __restrict__ acc, float* __restrict__ alpha,
    uint32_t* __restrict__ errFlag, MoverSinkArgs sink) {
    // F/m and M/I as the reference divides them.  Without contacts F and M
    // are +0 (sums that start at +0 never become -0), and +0 divided by a
    // positive finite mass or inertia is exactly +0, so the divisions are
    // skipped then; 2 m r^2 in [1e-30, 1e30] keeps the inertia positive and
    // finite.
    const bool quiet = f.x == 0.0f && f.y == 0.0f && moment == 0.0f && m > 0.0f && m < INFINITY;
    const float two_mrr = 2.0f * m * r * r;
    float2 a;
    float al;
    if (quiet && two_mrr >= 1e-30f && two_mrr <= 1e30f) {
        a = make_float2(0.0f, 0.0f);
        al = 0.0f;
    } else {
        a = make_float2(f.x / m, f.y / m);
        al = moment / inertia_of(m, r);
    }
    if (acc) acc[i] = a;
    if (alpha) alpha[i] = al;
    integrate_one(P, s, a, al, r, m, mat, pr);
    // the new state in this step's sorted order
    out.pos[i] = s.p;
    out.vel[i] = s.v;
    out.theta[i] = s.th;
    out.omega[i] = s.w;
    outS.mass[i] = m;
    outS.id[i] = id;
    if (TYPED) outS.type[i] = mat;
    loc[id] = i;
    if (pressure) pressure[i] = pr;
    const int2 gn = grid_pos_fast(P, s.p);
    const uint32_t nk = grid_hash(P, gn.x, gn.y);
    nextHash[i] = nk;
    if (!(isfinite(s.p.x) && isfinite(s.p.y))) atomicOr(errFlag, 1u);
    if (sink.ctrl && nk != key) {
        // a mover: count it as a leaver of its cell and an arrival of the new
        // one, and record it for the next step's incremental sort
        const uint32_t slot = atomicAdd(sink.arrCnt + nk, 1u);
        atomicAdd(sink.leavers + key, 1u);
        if (nk > key) atomicAdd(sink.arrLo + nk, 1u);
        const uint32_t m = atomicAdd(sink.ctrl + 1, 1u);
        const uint2 own = cellRange[key];
        if (m < sink.moverCap) sink.movers[m] = make_uint4(i, nk, key, slot);
        if (m >= sink.moverCap || slot >= kMaxGroup || own.y - own.x > kMaxGroup)
            atomicOr(sink.ctrl, 1u);
        // the cell scan rescans the tiles of both cells
        if (sink.dirty) {
            const uint32_t t0 = key >> sink.tileShift, t1 = nk >> sink.tileShift;
            atomicOr(sink.dirty + (t0 >> 5), 1u << (t0 & 31u));
            if (t1 != t0) atomicOr(sink.dirty + (t1 >> 5), 1u << (t1 & 31u));
        }
    }
}

// collideD + integrateSystemD + calcHashD of the next step for one particle.
// The acceleration stays in registers instead of a round trip through HBM;
// the arithmetic is the same expressions in the same order.
template <bool TYPED, bool ATTRACT, bool CULL, bool CONTROL = false>
__device__ __forceinline__ void step_particle(const KParams& P, uint32_t i, DynSet in,
                                              StatSet inS, const uint32_t* __restrict__ src,
                                              const uint32_t* __restrict__ sortedKey,
                                              const uint2* __restrict__ cellRange,
                                              const uint32_t* __restrict__ cellFirst, DynSet out,
                                              StatSet outS, uint32_t* __restrict__ loc,
                                              uint32_t* __restrict__ nextHash,
                                              float* __restrict__ pressure,
                                              float2* __restrict__ acc,
                                              float* __restrict__ alpha,
                                              uint32_t* __restrict__ errFlag, MoverSinkArgs sink,
                                              ControlArgs ctl = ControlArgs{}) {
    // position and radius are in this step's sorted order; the other fields
    // at the particle's slot of the previous order, src[i]
    Dyn s;
    s.p = in.pos[i];
    const float r = inS.radius[i];
    const uint32_t si = src[i];
    s.v = in.vel[si];
    s.w = in.omega[si];
    s.th = in.theta[si];
    const float m = inS.mass[si];
    const uint32_t id = inS.id[si];
    const uint32_t mat = TYPED ? inS.type[si] : 0u;
    // the sort key of particle i is calcGridPos of this very position, wrapped
    const uint32_t key = sortedKey[i];
    const uint32_t local = key - P.cellOff;
    const int2 g = make_int2((int)(local & (P.gx - 1u)), (int)(local >> P.log2gx));
    float2 f;
    float moment, pr;
    if (!CULL || !P.cull ||
        !collide_rows<TYPED, ATTRACT>(P, i, g, s.p, s.v, s.w, r, mat, in.pos, in.vel, in.omega,
                             inS.radius, inS.type, src, cellFirst, P.gx, f, moment, pr)) {
        if (CULL && !ATTRACT && P.cull)
            collide_one<TYPED, ATTRACT, true>(P, i, g, s.p, s.v, s.w, r, mat, in.pos, in.vel,
                                              in.omega, inS.radius, inS.type, src,
                                              PackedCells{cellRange}, f, moment, pr);
        else
            collide_one<TYPED, ATTRACT, false>(P, i, g, s.p, s.v, s.w, r, mat, in.pos, in.vel,
                                               in.omega, inS.radius, inS.type, src,
                                               PackedCells{cellRange}, f, moment, pr);
    }
    if (CONTROL)
        meet_control<TYPED, ATTRACT>(P, ctl, i, s.p, s.v, s.w, r, mat, f, moment, pr);
    finish_particle<TYPED>(P, i, s, f, moment, pr, r, m, mat, id, key, cellRange, out, outS, loc,
                           nextHash, pressure, acc, alpha, errFlag, sink);
}

// THREADS x MINB: the block size and the blocks per SM the registers are
// capped for (the step variants, chosen by the context's autotuner).
template <bool TYPED, bool ATTRACT, bool CULL, bool CONTROL, int THREADS = kCollideThreads,
          int MINB = 1024 / kCollideThreads>
__global__ void __launch_bounds__(THREADS, MINB)
step_kernel(KParams P, DynSet in, StatSet inS, const uint32_t* __restrict__ src,
            const uint32_t* __restrict__ sortedKey, const uint2* __restrict__ cellRange,
            const uint32_t* __restrict__ cellFirst, DynSet out, StatSet outS,
            uint32_t* __restrict__ loc, uint32_t* __restrict__ nextHash,
            float* __restrict__ pressure, float2* __restrict__ acc, float* __restrict__ alpha,
            uint32_t* __restrict__ errFlag, uint32_t n, MoverSinkArgs sink, ControlArgs ctl) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    step_particle<TYPED, ATTRACT, CULL, CONTROL>(P, i, in, inS, src, sortedKey, cellRange,
                                                 cellFirst, out, outS, loc, nextHash, pressure,
                                                 acc, alpha, errFlag, sink, ctl);
}

// reduceVecD (particles_kernel.cuh:551-578) for the three reaction vectors,
// launched as collide launches it (functions.cu:486-488): blocks of
// min(512, n) threads, a shared-memory tree that halves the block size.
constexpr int kControlThreads = 512;
__global__ void __launch_bounds__(kControlThreads)
control_reduce_kernel(ControlArgs ctl, uint32_t n, float* __restrict__ partials,
                      const uint32_t* __restrict__ active) {
    if (active && *active == 0u) return;
    __shared__ float cache[3][kControlThreads];
    const uint32_t index = blockIdx.x * blockDim.x + threadIdx.x;
    const int t = threadIdx.x;
    const bool in = index < n;
    cache[0][t] = in ? ctl.fx[index] : 0.0f;
    cache[1][t] = in ? ctl.fy[index] : 0.0f;
    cache[2][t] = in ? ctl.fm[index] : 0.0f;
    __syncthreads();
    for (int i = blockDim.x / 2; i != 0; i /= 2) {
        if (t < i) {
            cache[0][t] += cache[0][t + i];
            cache[1][t] += cache[1][t + i];
            cache[2][t] += cache[2][t + i];
        }
        __syncthreads();
    }
    if (t == 0) {
        partials[blockIdx.x] = cache[0][0];
        partials[gridDim.x + blockIdx.x] = cache[1][0];
        partials[2 * gridDim.x + blockIdx.x] = cache[2][0];
    }
}

// the host's sum of the block results in block order (functions.cu:511-519),
// then the host's move of the control particle (main.cu:511-514): float +=
// double, and the wraps.  The sums are three serial chains of adds; the block
// results reach them through shared memory, a tile of kSumTile at a time, so
// that a chain waits for an add (4 cycles) and not for a load from L2 (391
// block results of 200,000 disks: a step 60 -> 45 us).
constexpr int kSumThreads = 256;
constexpr uint32_t kSumTile = 1024;
__global__ void __launch_bounds__(kSumThreads)
control_sum_move_kernel(ControlDev* __restrict__ c, const float* __restrict__ partials,
                        uint32_t blocks, float* __restrict__ out,
                        const uint32_t* __restrict__ active) {
    if (active && *active == 0u) return;
    __shared__ float tile[3][kSumTile];
    const uint32_t t = threadIdx.x, k = t >> 5;  // lane 0 of warp k < 3 adds component k
    float sum = 0.0f;
    for (uint32_t base = 0; base < blocks; base += kSumTile) {
        const uint32_t m = min(blocks - base, kSumTile);
        for (uint32_t b = t; b < m; b += kSumThreads) {
            tile[0][b] = partials[base + b];
            tile[1][b] = partials[blocks + base + b];
            tile[2][b] = partials[2 * blocks + base + b];
        }
        __syncthreads();
        if (k < 3 && (t & 31u) == 0u) {
#pragma unroll 8
            for (uint32_t b = 0; b < m; ++b) sum += tile[k][b];
        }
        __syncthreads();
    }
    if (k < 3 && (t & 31u) == 0u) out[k] = sum;
    if (t != 0) return;
    float2 p = c->pos;
    p.x = (float)((double)p.x + c->drift[0]);
    p.y = (float)((double)p.y + c->drift[1]);
    if ((double)p.y < c->wrapYBelow) p.y = (float)c->wrapYTo;
    if ((double)p.x > c->wrapXAbove) p.x = (float)c->wrapXTo;
    c->pos = p;
}

// Batched form: particle slot i belongs to specimen spec[i] (slots of a
// specimen are contiguous and never change specimen), whose parameters --
// box, grid, cell offset, contact coefficients -- come from a device table.
template <bool TYPED, bool ATTRACT, bool CULL, int THREADS = kCollideThreads,
          int MINB = 1024 / kCollideThreads>
__global__ void __launch_bounds__(THREADS, MINB)
step_kernel_batched(const KParams* __restrict__ table, const uint32_t* __restrict__ spec,
                    DynSet in, StatSet inS, const uint32_t* __restrict__ src,
                    const uint32_t* __restrict__ sortedKey, const uint2* __restrict__ cellRange,
                    const uint32_t* __restrict__ cellFirst, DynSet out, StatSet outS,
                    uint32_t* __restrict__ loc, uint32_t* __restrict__ nextHash,
                    float* __restrict__ pressure, float2* __restrict__ acc,
                    float* __restrict__ alpha, uint32_t* __restrict__ errFlag, uint32_t n,
                    MoverSinkArgs sink) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    step_particle<TYPED, ATTRACT, CULL>(table[spec[i]], i, in, inS, src, sortedKey, cellRange,
                                        cellFirst, out, outS, loc, nextHash, pressure, acc,
                                        alpha, errFlag, sink);
}

// Reorder for the context step: as reorder_kernel, but the cell ranges are
// written as interleaved (start, end) pairs (empty cells hold 0xFFFFFFFF).
template <bool TYPED>
__global__ void __launch_bounds__(kThreads)
reorder_packed_kernel(uint2* __restrict__ cellRange, DynSet s, StatSet sS,
                      uint32_t* __restrict__ sLoc, const uint32_t* __restrict__ hash,
                      const uint32_t* __restrict__ index, DynSet o, StatSet oS, uint32_t n) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    const bool valid = i < n;
    const uint32_t h = valid ? hash[i] : 0u;
    uint32_t hp = __shfl_up_sync(0xffffffffu, h, 1);
    if ((threadIdx.x & 31) == 0 && valid && i > 0) hp = hash[i - 1];
    if (!valid) return;
    if (i == 0 || h != hp) {
        cellRange[h].x = i;
        if (i > 0) cellRange[hp].y = i;
    }
    if (i == n - 1) cellRange[h].y = i + 1;
    const uint32_t src = index[i];
    s.pos[i] = o.pos[src];
    s.vel[i] = o.vel[src];
    s.theta[i] = o.theta[src];
    s.omega[i] = o.omega[src];
    sS.radius[i] = oS.radius[src];
    sS.mass[i] = oS.mass[src];
    const uint32_t id = oS.id[src];
    sS.id[i] = id;
    sLoc[id] = i;
    if (TYPED) sS.type[i] = oS.type[src];
}

__global__ void unpack_cells_kernel(const uint2* __restrict__ range, uint32_t numCells,
                                    uint32_t* __restrict__ cellStart,
                                    uint32_t* __restrict__ cellEnd) {
    const uint32_t c = blockIdx.x * blockDim.x + threadIdx.x;
    if (c >= numCells) return;
    const uint2 v = range[c];
    if (cellStart) cellStart[c] = v.x;
    if (cellEnd) cellEnd[c] = v.y;
}

__global__ void followed_kernel(FollowIds f, const uint32_t* __restrict__ loc, DynSet d, StatSet s,
                                const float2* __restrict__ acc, const float* __restrict__ alpha,
                                const float* __restrict__ pressure, float* __restrict__ rows) {
    const uint32_t k = threadIdx.x;
    if (k >= f.count) return;
    followed_row(loc[f.id[k]], rows + 12 * k, d, s, acc, alpha, pressure);
}

// The rows of ids[0, *count) into row block (slot ? *slot : 0) + add of
// `ring` (*count rows of 12 words per block).
__global__ void followed_ring_kernel(const uint32_t* __restrict__ ids,
                                     const uint32_t* __restrict__ countWord,
                                     const uint32_t* __restrict__ slot, uint32_t add,
                                     const uint32_t* __restrict__ loc, DynSet d, StatSet s,
                                     const float2* __restrict__ acc,
                                     const float* __restrict__ alpha,
                                     const float* __restrict__ pressure, float* __restrict__ ring) {
    const uint32_t count = *countWord;
    float* base = ring + (size_t)((slot ? *slot : 0u) + add) * count * 12;
    for (uint32_t k = blockIdx.x * blockDim.x + threadIdx.x; k < count; k += gridDim.x * blockDim.x)
        followed_row(loc[ids[k]], base + 12ull * k, d, s, acc, alpha, pressure);
}

// Largest radius (positive floats order like their bit patterns).
__global__ void max_radius_kernel(const float* __restrict__ radius, uint32_t n,
                                  uint32_t* __restrict__ out) {
    float m = 0.0f;
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
        m = fmaxf(m, radius[i]);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
    if ((threadIdx.x & 31) == 0) atomicMax(out, __float_as_uint(m));
}

bool has_attraction(const KParams& P) {
    for (uint32_t m = 0; m < P.nmat; ++m)
        if (P.at[m] != 0.0f) return true;
    return false;
}

}  // namespace

cudaError_t launch_followed(const FollowIds& f, const uint32_t* loc, DynSet d, StatSet s,
                            const float2* acc, const float* alpha, const float* pressure,
                            float* rows, cudaStream_t st) {
    followed_kernel<<<1, kFollowBatch, 0, st>>>(f, loc, d, s, acc, alpha, pressure, rows);
    return cudaGetLastError();
}

cudaError_t launch_followed_ring(const uint32_t* ids, const uint32_t* countWord,
                                 const uint32_t* slot, uint32_t add, const uint32_t* loc, DynSet d,
                                 StatSet s, const float2* acc, const float* alpha,
                                 const float* pressure, float* ring, cudaStream_t st) {
    followed_ring_kernel<<<16, 128, 0, st>>>(ids, countWord, slot, add, loc, d, s, acc, alpha,
                                             pressure, ring);
    return cudaGetLastError();
}

cudaError_t launch_max_radius(const float* radius, uint32_t n, uint32_t* out, cudaStream_t st) {
    if (n == 0) return cudaSuccess;
    const unsigned b = blocks_for(n, kThreads) < 1184 ? blocks_for(n, kThreads) : 1184;
    max_radius_kernel<<<b, kThreads, 0, st>>>(radius, n, out);
    return cudaGetLastError();
}

cudaError_t launch_calc_hash_batched(const KParams* table, const uint32_t* spec, const float2* pos,
                                     uint32_t* hash, uint32_t n, cudaStream_t st) {
    if (n == 0) return cudaSuccess;
    calc_hash_batched_kernel<<<blocks_for(n, kThreads), kThreads, 0, st>>>(table, spec, pos, hash,
                                                                           n);
    return cudaGetLastError();
}

cudaError_t launch_calc_hash(const KParams& P, const float2* pos, uint32_t* hash, uint32_t* index,
                             uint32_t n, cudaStream_t st) {
    if (n == 0) return cudaSuccess;
    calc_hash_kernel<<<blocks_for(n, kThreads), kThreads, 0, st>>>(P, pos, hash, index, n);
    return cudaGetLastError();
}

cudaError_t launch_reorder(const KParams& P, uint32_t* cellStart, uint32_t* cellEnd,
                           DynSet sorted, StatSet sortedS, uint32_t* sortedLoc,
                           const uint32_t* hash, const uint32_t* index, DynSet old, StatSet oldS,
                           uint32_t n, uint32_t numCells, bool clearCells, cudaStream_t st,
                           int* launches) {
    (void)P;
    if (clearCells) {
        cudaError_t e = cudaMemsetAsync(cellStart, 0xff, sizeof(uint32_t) * (size_t)numCells, st);
        if (e != cudaSuccess) return e;
    }
    if (n == 0) return cudaSuccess;
    if (sortedS.type && oldS.type)
        reorder_kernel<true><<<blocks_for(n, kThreads), kThreads, 0, st>>>(
            cellStart, cellEnd, sorted, sortedS, sortedLoc, hash, index, old, oldS, n, numCells);
    else
        reorder_kernel<false><<<blocks_for(n, kThreads), kThreads, 0, st>>>(
            cellStart, cellEnd, sorted, sortedS, sortedLoc, hash, index, old, oldS, n, numCells);
    if (launches) ++*launches;
    return cudaGetLastError();
}

cudaError_t launch_collide(const KParams& P, const float2* pos, const float2* vel,
                           const float* omega, const float* radius, const float* mass,
                           const uint32_t* type, const uint32_t* cellStart,
                           const uint32_t* cellEnd, float2* acc, float* alpha, float* pressure,
                           uint32_t n, cudaStream_t st) {
    if (n == 0) return cudaSuccess;
    const bool typed = type != nullptr && P.nmat > 1;
    const bool attract = has_attraction(P);
    const unsigned b = blocks_for(n, kCollideThreads);
#define DEM_COLLIDE(T, A)                                                                     \
    collide_kernel<T, A><<<b, kCollideThreads, 0, st>>>(P, pos, vel, omega, radius, mass, type, \
                                                        cellStart, cellEnd, acc, alpha,        \
                                                        pressure, n)
    if (typed) {
        if (attract) DEM_COLLIDE(true, true); else DEM_COLLIDE(true, false);
    } else {
        if (attract) DEM_COLLIDE(false, true); else DEM_COLLIDE(false, false);
    }
#undef DEM_COLLIDE
    return cudaGetLastError();
}

cudaError_t launch_integrate(const KParams& P, float2* pos, float2* vel, const float2* acc,
                             float* theta, float* omega, const float* alpha, const uint32_t* type,
                             const float* radius, const float* mass, float* pressure, uint32_t n,
                             cudaStream_t st) {
    if (n == 0) return cudaSuccess;
    const unsigned b = blocks_for(n, kThreads);
    if (type != nullptr && P.nmat > 1)
        integrate_kernel<true><<<b, kThreads, 0, st>>>(P, pos, vel, acc, theta, omega, alpha, type,
                                                       radius, mass, pressure, n);
    else
        integrate_kernel<false><<<b, kThreads, 0, st>>>(P, pos, vel, acc, theta, omega, alpha,
                                                        type, radius, mass, pressure, n);
    return cudaGetLastError();
}

cudaError_t launch_step(const KParams& P, DynSet in, StatSet inS, const uint32_t* src,
                        const uint32_t* sortedKey, const uint2* cellRange,
                        const uint32_t* cellFirst, DynSet out, StatSet outS, uint32_t* loc,
                        uint32_t* nextHash, float* pressure, float2* acc, float* alpha,
                        uint32_t* errFlag, uint32_t n, MoverSinkArgs sink, cudaStream_t st,
                        const KParams* table, const uint32_t* spec, ControlArgs ctl,
                        int variant) {
    if (n == 0) return cudaSuccess;
    if (variant < 0 || variant >= kStepVariants) return cudaErrorInvalidValue;
    const bool typed = inS.type != nullptr && P.nmat > 1;
    const bool attract = has_attraction(P);
    const bool cull = table ? true : P.cull != 0u;
#define DEM_STEP_T(T, A, C, TH, MB)                                                            \
    do {                                                                                       \
        const unsigned b = blocks_for(n, TH);                                                  \
        if (table)                                                                             \
            step_kernel_batched<T, A, C, TH, MB><<<b, TH, 0, st>>>(                            \
                table, spec, in, inS, src, sortedKey, cellRange, cellFirst, out, outS, loc,     \
                nextHash, pressure, acc, alpha, \
                errFlag, n, sink);                                                             \
        else if (ctl.c)                                                                        \
            step_kernel<T, A, C, true><<<blocks_for(n, kCollideThreads), kCollideThreads, 0,  \
                                         st>>>(P, in, inS, src, sortedKey, cellRange, cellFirst, \
                                               out, outS, loc, nextHash, \
                                               pressure, acc, alpha, errFlag, n, sink, ctl);  \
        else                                                                                   \
            step_kernel<T, A, C, false, TH, MB><<<b, TH, 0, st>>>(                             \
                P, in, inS, src, sortedKey, cellRange, cellFirst, out, outS, loc, nextHash,    \
                pressure, acc, alpha, errFlag, \
                n, sink, ctl);                                                                 \
    } while (0)
#define DEM_STEP(T, A, C)                                                                      \
    do {                                                                                       \
        switch (variant) {                                                                     \
            case 1: DEM_STEP_T(T, A, C, 64, 16); break;                                        \
            case 2: DEM_STEP_T(T, A, C, 256, 4); break;                                        \
            case 3: DEM_STEP_T(T, A, C, 128, 6); break;                                        \
            default: DEM_STEP_T(T, A, C, 128, 8); break;                                       \
        }                                                                                      \
    } while (0)
    if (typed) {
        if (attract && cull) DEM_STEP(true, true, true);
        else if (attract) DEM_STEP(true, true, false);
        else if (cull) DEM_STEP(true, false, true);
        else DEM_STEP(true, false, false);
    } else {
        if (attract && cull) DEM_STEP(false, true, true);
        else if (attract) DEM_STEP(false, true, false);
        else if (cull) DEM_STEP(false, false, true);
        else DEM_STEP(false, false, false);
    }
#undef DEM_STEP
#undef DEM_STEP_T
    return cudaGetLastError();
}

StepShape step_variant_shape(int variant) {
    switch (variant) {
        case 1: return StepShape{64, 16};
        case 2: return StepShape{256, 4};
        case 3: return StepShape{128, 6};
        default: return StepShape{128, 8};
    }
}

namespace {
__global__ void loop_init_kernel(const uint32_t* __restrict__ req, uint32_t* __restrict__ left,
                                 cudaGraphConditionalHandle h) {
    const uint32_t n = *req;
    *left = n;
    cudaGraphSetConditional(h, n ? 1u : 0u);
}
__global__ void loop_next_kernel(uint32_t* __restrict__ left, uint32_t* __restrict__ idx,
                                 int32_t idxStep, cudaGraphConditionalHandle h) {
    const uint32_t n = *left - 1u;
    *left = n;
    if (idx) *idx += (uint32_t)idxStep;
    cudaGraphSetConditional(h, n ? 1u : 0u);
}
}  // namespace

namespace {
__global__ void set_words_kernel(uint32_t* __restrict__ dst, Words w) {
    for (uint32_t i = 0; i < w.count; ++i) dst[i] = w.v[i];
}
}  // namespace

namespace {
// A row of blocks per array, 16 bytes a thread.  One launch for the dozen arrays
// of a state, which as copies cost a dozen launches: 34 -> 8 us at 65,536 disks.
__global__ void __launch_bounds__(kThreads) copy_arrays_kernel(CopyList c) {
    const int a = blockIdx.y;
    const size_t words = c.words[a], quads = words / 4;
    const uint4* __restrict__ s = reinterpret_cast<const uint4*>(c.src[a]);
    uint4* __restrict__ d = reinterpret_cast<uint4*>(c.dst[a]);
    const size_t t0 = (size_t)blockIdx.x * kThreads + threadIdx.x;
    const size_t stride = (size_t)gridDim.x * kThreads;
    size_t k = t0;
    for (; k + 3 * stride < quads; k += 4 * stride) {
        const uint4 x0 = s[k], x1 = s[k + stride], x2 = s[k + 2 * stride], x3 = s[k + 3 * stride];
        d[k] = x0;
        d[k + stride] = x1;
        d[k + 2 * stride] = x2;
        d[k + 3 * stride] = x3;
    }
    for (; k < quads; k += stride) d[k] = s[k];
    if (t0 < (words & 3u)) c.dst[a][4 * quads + t0] = c.src[a][4 * quads + t0];
}
}  // namespace

cudaError_t launch_copy_arrays(const CopyList& c, cudaStream_t st) {
    if (c.count < 0 || c.count > kCopyMax) return cudaErrorInvalidValue;
    size_t most = 0;
    for (int a = 0; a < c.count; ++a) most = c.words[a] > most ? c.words[a] : most;
    if (most == 0) return cudaSuccess;
    const unsigned b = blocks_for((uint32_t)((most + 3) / 4 < 1u << 30 ? (most + 3) / 4 : 1u << 30),
                                  kThreads);
    copy_arrays_kernel<<<dim3(b < 296u ? b : 296u, (unsigned)c.count), kThreads, 0, st>>>(c);
    return cudaGetLastError();
}

cudaError_t launch_set_words(uint32_t* dst, Words w, cudaStream_t st) {
    if (w.count > 8) return cudaErrorInvalidValue;
    set_words_kernel<<<1, 1, 0, st>>>(dst, w);
    return cudaGetLastError();
}

cudaError_t launch_loop_init(const uint32_t* req, uint32_t* left, cudaGraphConditionalHandle h,
                             cudaStream_t st) {
    loop_init_kernel<<<1, 1, 0, st>>>(req, left, h);
    return cudaGetLastError();
}

cudaError_t launch_loop_next(uint32_t* left, uint32_t* idx, int32_t idxStep,
                             cudaGraphConditionalHandle h, cudaStream_t st) {
    loop_next_kernel<<<1, 1, 0, st>>>(left, idx, idxStep, h);
    return cudaGetLastError();
}

cudaError_t launch_control_post(ControlArgs ctl, ControlDev* c, uint32_t n, float* partials,
                                float* out, cudaStream_t st, int* launches,
                                const uint32_t* active) {
    const uint32_t threads = n < (uint32_t)kControlThreads ? (n ? n : 1u) : (uint32_t)kControlThreads;
    const uint32_t blocks = n ? (n + threads - 1) / threads : 0u;
    if (blocks) control_reduce_kernel<<<blocks, threads, 0, st>>>(ctl, n, partials, active);
    control_sum_move_kernel<<<1, kSumThreads, 0, st>>>(c, partials, blocks, out, active);
    if (launches) *launches += blocks ? 2 : 1;
    return cudaGetLastError();
}

cudaError_t launch_reorder_packed(uint2* cellRange, DynSet sorted, StatSet sortedS,
                                  uint32_t* sortedLoc, const uint32_t* hash, const uint32_t* index,
                                  DynSet old, StatSet oldS, uint32_t n, uint32_t numCells,
                                  cudaStream_t st, int* launches) {
    cudaError_t e = cudaMemsetAsync(cellRange, 0xff, sizeof(uint2) * (size_t)numCells, st);
    if (e != cudaSuccess || n == 0) return e;
    if (sortedS.type && oldS.type)
        reorder_packed_kernel<true><<<blocks_for(n, kThreads), kThreads, 0, st>>>(
            cellRange, sorted, sortedS, sortedLoc, hash, index, old, oldS, n);
    else
        reorder_packed_kernel<false><<<blocks_for(n, kThreads), kThreads, 0, st>>>(
            cellRange, sorted, sortedS, sortedLoc, hash, index, old, oldS, n);
    if (launches) ++*launches;
    return cudaGetLastError();
}

cudaError_t launch_unpack_cells(const uint2* cellRange, uint32_t numCells, uint32_t* cellStart,
                                uint32_t* cellEnd, cudaStream_t st) {
    if (numCells == 0) return cudaSuccess;
    unpack_cells_kernel<<<blocks_for(numCells, kThreads), kThreads, 0, st>>>(cellRange, numCells,
                                                                             cellStart, cellEnd);
    return cudaGetLastError();
}

}  // namespace dem
