// The neighbour search of the step: candidates of the 3 x 3 cells, in the
// reference's order, cell by cell (collide_one) or by row intervals
// (collide_rows).
#pragma once

#include "dem_common.cuh"
#include "dem_kernels.cuh"

namespace dem {

// Cell ranges, read either from the reference's two arrays (cellStart with
// 0xFFFFFFFF for empty cells, cellEnd) or from the context's interleaved
// (start, end) pairs.  An empty cell yields start >= end, so its particle
// loop runs zero times, as the reference's `startIndex != -1` test does.
struct SplitCells {
    const uint32_t* __restrict__ start;
    const uint32_t* __restrict__ end;
    __device__ __forceinline__ uint2 get(uint32_t h) const {
        const uint32_t a = __ldg(start + h);
        return make_uint2(a, a == kEmptyCell ? 0u : __ldg(end + h));
    }
};
struct PackedCells {
    const uint2* __restrict__ range;
    __device__ __forceinline__ uint2 get(uint32_t h) const { return __ldg(range + h); }
};
// First-particle array of gx + 1 words a row, the last one the row's end, of
// the grid whose cells are numbered from cellOff.
struct RowCells {
    const uint32_t* __restrict__ first;
    uint32_t gx, log2gx, cellOff;
    __device__ __forceinline__ uint2 get(uint32_t h) const {
        h -= cellOff;
        const uint32_t* __restrict__ f = first + (size_t)(h >> log2gx) * (gx + 1u) + (h & (gx - 1u));
        return make_uint2(__ldg(f), __ldg(f + 1));
    }
};

// Packed pairs of IEEE single-precision operations (PTX f32x2, round to
// nearest even, sm_100): each lane of the result is the same correctly
// rounded value as the scalar operation.
__device__ __forceinline__ float2 f32x2_add(float2 a, float2 b) {
    float2 d;
    asm("{.reg .b64 ra, rb, rd;\n\t"
        "mov.b64 ra, {%2, %3};\n\tmov.b64 rb, {%4, %5};\n\t"
        "add.rn.f32x2 rd, ra, rb;\n\tmov.b64 {%0, %1}, rd;}"
        : "=f"(d.x), "=f"(d.y)
        : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y));
    return d;
}
__device__ __forceinline__ float2 f32x2_sub(float2 a, float2 b) {
    float2 d;
    asm("{.reg .b64 ra, rb, rd;\n\t"
        "mov.b64 ra, {%2, %3};\n\tmov.b64 rb, {%4, %5};\n\t"
        "sub.rn.f32x2 rd, ra, rb;\n\tmov.b64 {%0, %1}, rd;}"
        : "=f"(d.x), "=f"(d.y)
        : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y));
    return d;
}
__device__ __forceinline__ float2 f32x2_mul(float2 a, float2 b) {
    float2 d;
    asm("{.reg .b64 ra, rb, rd;\n\t"
        "mov.b64 ra, {%2, %3};\n\tmov.b64 rb, {%4, %5};\n\t"
        "mul.rn.f32x2 rd, ra, rb;\n\tmov.b64 {%0, %1}, rd;}"
        : "=f"(d.x), "=f"(d.y)
        : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y));
    return d;
}
__device__ __forceinline__ float2 f32x2_fma(float2 a, float2 b, float2 c) {
    float2 d;
    asm("{.reg .b64 ra, rb, rc, rd;\n\t"
        "mov.b64 ra, {%2, %3};\n\tmov.b64 rb, {%4, %5};\n\tmov.b64 rc, {%6, %7};\n\t"
        "fma.rn.f32x2 rd, ra, rb, rc;\n\tmov.b64 {%0, %1}, rd;}"
        : "=f"(d.x), "=f"(d.y)
        : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y), "f"(c.x), "f"(c.y));
    return d;
}

// A bit for each of the 8 candidates at pq (radii pr) that may touch a particle
// at p of radius r (ATTRACT: that is within attraction reach).  Two candidates
// share each packed f32x2 operation.  d2 is the law's own
// rn(rn(dx^2) + rn(dy^2)); the bound cd^2 (1 + 2e-6) is a fused multiply-add,
// within 2e-7 relative of the exact value, so a rejected candidate still has
// sqrtf(d2) >= rA + rB in the law's arithmetic (the law itself is unchanged).
template <bool ATTRACT>
__device__ __forceinline__ uint32_t filter8(const float2* __restrict__ pq,
                                            const float* __restrict__ pr, float2 p, float r) {
    float2 q[8];
    float rq[8];
#pragma unroll
    for (int k = 0; k < 8; ++k) {
        q[k] = __ldg(pq + k);
        rq[k] = __ldg(pr + k);
    }
    uint32_t m8 = 0u;
#pragma unroll
    for (int k = 0; k < 8; k += 2) {
        const float2 da = f32x2_sub(q[k], p), db = f32x2_sub(q[k + 1], p);
        const float2 sa = f32x2_mul(da, da), sb = f32x2_mul(db, db);
        const float d2a = sa.x + sa.y, d2b = sb.x + sb.y;
        float2 bound;
        if (ATTRACT) {
            bound = make_float2(attract_reach2(r, rq[k]), attract_reach2(r, rq[k + 1]));
        } else {
            const float2 cd = f32x2_add(make_float2(r, r), make_float2(rq[k], rq[k + 1]));
            const float2 c2 = f32x2_mul(cd, cd);
            bound = f32x2_fma(c2, make_float2(2e-6f, 2e-6f), c2);
        }
        // (with attraction a distance that is not a number stays: it adds 0 / (4 pi
        // r^2) to the pressure, which is one to a disk without a radius)
        if (ATTRACT ? !(d2a > bound.x) : d2a <= bound.x) m8 |= 1u << k;
        if (ATTRACT ? !(d2b > bound.y) : d2b <= bound.y) m8 |= 2u << k;
    }
    return m8;
}

// Force, moment and pressure of one particle.
struct Pull {
    float2 f;
    float moment, pr;
};

// The running sums of one particle: a subtotal per cell, added to the force
// when the next cell begins (an empty cell adds +0).
struct Sums {
    Pull o{make_float2(0.0f, 0.0f), 0.0f, 0.0f};
    float2 sub = make_float2(0.0f, 0.0f);
    uint32_t cell = 15u;
    __device__ __forceinline__ void begin(uint32_t c) {
        if (c == cell) return;
        o.f.x += sub.x;
        o.f.y += sub.y;
        sub = make_float2(0.0f, 0.0f);
        cell = c;
    }
    __device__ __forceinline__ Pull close() {
        begin(15u);
        return o;
    }
};

// A warp's contacts, dealt to its lanes.  The contact law is some two hundred
// instructions (five IEEE divisions, four square roots; a double division for the
// pressure where that is wanted) and the particles of a warp touch 0 to 6 others,
// so lane by lane it ran at a third of the lanes.  Instead a turn takes up to kDeal kept candidates of
// every lane, whose loads are in flight together, and writes the touching ones
// into a list in shared memory; the warp evaluates the list 32 at a time, and
// each lane adds up its own results in its own order.  In the band step, with
// its kept candidates, a call of 20 steps: 1,000,003 dense disks 54.1 M warp instructions a
// step at 11 active lanes -> 30 M at 19; 4,194,304 disks 3,911 -> 3,327 us,
// 250,007 cohesive disks 1,339 -> 1,019 us, 50 steps of 65,536 disks
// 1,024 -> 885 us.  What bounds the step now is the latency of its four or five
// rounds of dependent loads (42 % of issue slots used at 4,194,304 disks).
constexpr int kDeal = 4;
template <bool ATTRACT>
struct Deal {
    uint32_t j[kDeal * 32];  // [candidate of the turn][lane]: the neighbour, then the force's x
    float fy[kDeal * 32], moment[kDeal * 32];
    double q[kDeal * 32];
    float ax[ATTRACT ? kDeal * 32 : 1], ay[ATTRACT ? kDeal * 32 : 1];
    double aq[ATTRACT ? kDeal * 32 : 1];
    uint8_t code[kDeal * 32];  // the list: index into the arrays above
};

// The turn's `total` listed contacts through the law, then each lane's own (bit
// k of `mine`: its candidate k; four bits of `cells` each: the cell) into its
// sums.  The neighbours' velocity, spin and type are read through `src` where
// the arrays are in the previous order.  The pressure, which nothing but a
// caller reads, is summed only with `wantPr`.  The parameters are P, or with
// `table` those of the particle's specimen `spec` (a warp may hold particles of
// several).  Every lane calls it.
template <bool TYPED, bool ATTRACT>
__device__ __forceinline__ void deal_law(const KParams& P0, const KParams* __restrict__ table,
                                         uint32_t spec, Deal<ATTRACT>& S, bool wantPr,
                                         uint32_t total, uint32_t mine, uint32_t cells, float2 p, float2 v,
                                         float w, float r, uint32_t mat,
                                         const float2* __restrict__ pos,
                                         const float2* __restrict__ vel,
                                         const float* __restrict__ omega,
                                         const float* __restrict__ radius,
                                         const uint32_t* __restrict__ type,
                                         const uint32_t* __restrict__ src, Sums& sum) {
    constexpr unsigned kAll = 0xffffffffu;
    const uint32_t lane = threadIdx.x & 31u;
    __syncwarp();
    for (uint32_t e0 = 0; e0 < total; e0 += 32u) {
        const uint32_t e = e0 + lane;
        const uint32_t code = e < total ? S.code[e] : lane;
        const int own = (int)(code & 31u);
        const float2 pA = make_float2(__shfl_sync(kAll, p.x, own), __shfl_sync(kAll, p.y, own));
        const float2 vA = make_float2(__shfl_sync(kAll, v.x, own), __shfl_sync(kAll, v.y, own));
        const float wA = __shfl_sync(kAll, w, own), rA = __shfl_sync(kAll, r, own);
        const uint32_t mA = TYPED ? __shfl_sync(kAll, mat, own) : 0u;
        const KParams& P = table ? table[__shfl_sync(kAll, spec, own)] : P0;
        if (e < total) {
            const uint32_t j = S.j[code];
            const uint32_t sj = src ? __ldg(src + j) : j;
            const uint32_t mB = TYPED ? __ldg(type + sj) : 0u;
            const float4 pc = TYPED ? P.pair[mA * P.nmat + mB] : P.pair[0];
            const float2 pB = __ldg(pos + j);
            const float rB = __ldg(radius + j);
            float2 f;
            float m, flen;
            const bool touch = pair_terms(pA, pB, vA, __ldg(vel + sj), wA, __ldg(omega + sj), rA,
                                          rB, pc, P.dt, f, m, flen);
            S.j[code] = __float_as_uint(f.x);
            S.fy[code] = f.y;
            S.moment[code] = m;
            // (a touching disk without a radius: 0 / 0, as the reference has it)
            if (wantPr) S.q[code] = touch ? pressure_term(flen, rA) : 0.0;
            if (ATTRACT) {
                const float2 g = pair_attract_terms(pA, pB, rA, rB, P.at[mA], P.at[mB]);
                S.ax[code] = g.x;
                S.ay[code] = g.y;
                if (wantPr) S.aq[code] = pressure_term(len2(g.x, g.y), rA);
            }
        }
    }
    __syncwarp();
    while (mine) {
        const uint32_t k = (uint32_t)__ffs(mine) - 1u, x = k * 32u + lane;
        mine &= mine - 1u;
        sum.begin((cells >> (4u * k)) & 15u);
        sum.sub.x += __uint_as_float(S.j[x]);
        sum.sub.y += S.fy[x];
        sum.o.moment += S.moment[x];
        if (wantPr) sum.o.pr = (float)((double)sum.o.pr + S.q[x]);
        if (ATTRACT) {
            sum.sub.x += S.ax[x];
            sum.sub.y += S.ay[x];
            if (wantPr) sum.o.pr = (float)((double)sum.o.pr + S.aq[x]);
        }
    }
    __syncwarp();  // the results are read
}

// Contact test and force of one candidate j (the reference's collideSpheres
// and, with ATTRACT, attractSpheres) added to the cell subtotal fc.
template <bool TYPED, bool ATTRACT>
__device__ __forceinline__ void candidate(const KParams& P, uint32_t j, float2 p, float2 v, float w,
                                          float r, uint32_t mat, float2 pj, float d2,
                                          const float2* __restrict__ vel,
                                          const float* __restrict__ omega,
                                          const float* __restrict__ radius,
                                          const uint32_t* __restrict__ type,
                                          const uint32_t* __restrict__ src, float2& fc,
                                          float& moment, float& pr) {
    const float rj = __ldg(radius + j);
    if (ATTRACT && attract_out_of_reach(r, rj, d2)) return;
    // velocity, spin and type of candidate j sit at its slot of the previous
    // order (src), or at j when the arrays are all in one order (src null)
    const uint32_t sj = src ? __ldg(src + j) : j;
    uint32_t mj = 0;
    float4 pc = P.pair[0];
    if (TYPED) {
        mj = __ldg(type + sj);
        pc = P.pair[mat * P.nmat + mj];
    }
    const float cd = r + rj;
    // d2 > cd^2 (1 + 2e-6) implies sqrtf(d2) >= cd after rounding: no contact
    if (d2 <= cd * cd * 1.000002f && sqrtf(d2) < cd) {
        const float2 f = pair_force(p, pj, v, __ldg(vel + sj), w, __ldg(omega + sj), r, rj, pc,
                                    P.dt, moment, pr);
        fc.x += f.x;
        fc.y += f.y;
    }
    if (ATTRACT) {
        const float2 f = pair_attract(p, pj, r, rj, P.at[mat], P.at[mj], pr);
        fc.x += f.x;
        fc.y += f.y;
    }
}

// Sum of the forces on particle i from its 3x3 cell neighbourhood,
// particles_kernel.cuh:459-549 (collideD) with collideCell (:346-385): cells
// y-outer, x-inner, particles in ascending sorted index, each cell's
// subtotal added to the running force.  `g` is the particle's grid position
// (calcGridPos, or the wrapped cell of its sort key: the same neighbour
// cells).  Wrapping makes a 1- or 2-wide grid visit the same cell more than
// once, exactly as the reference does.
//
// Work the reference spends on pairs that are not in contact is skipped
// without changing any result, because such a pair adds nothing (its force
// is +0 -- and a running sum that starts at +0 can never be -0 -- and it
// touches neither moment nor pressure):
//  * a candidate is dropped before the square root when its squared distance
//    exceeds (rA + rB)^2 by a relative 2e-6; then sqrtf(d2) >= rA + rB after
//    rounding, which is the reference's no-contact branch;
//  * with CULL (the context step, which knows an upper bound rmax on all
//    radii), a neighbour column/row is not visited when the particle is
//    farther than rA + rmax (plus a rounding margin) from that side of its
//    own cell, and candidates are first tested against rA + rmax so that
//    the neighbour's radius is loaded only for near pairs.  Culling needs at
//    least 3 cells per axis and cells wider than 2 rmax (then the three
//    columns/rows are distinct cells and a wrapped neighbour is out of
//    reach) and a particle inside the box by more than the margin.
// `g` is the particle's cell in the context's rows (for a row window, the
// scene's row minus rowOff).
template <bool TYPED, bool ATTRACT, bool CULL, typename Cells>
__device__ __forceinline__ void collide_one(const KParams& P, uint32_t i, int2 g, float2 p,
                                            float2 v, float w, float r, uint32_t mat,
                                            const float2* __restrict__ pos,
                                            const float2* __restrict__ vel,
                                            const float* __restrict__ omega,
                                            const float* __restrict__ radius,
                                            const uint32_t* __restrict__ type,
                                            const uint32_t* __restrict__ src, Cells cells,
                                            float2& force, float& moment, float& pr) {
    force = make_float2(0.0f, 0.0f);
    moment = 0.0f;
    pr = 0.0f;
    int y0 = -1, y1 = 1, x0 = -1, x1 = 1;
    float reach2 = INFINITY;
    if (CULL && p.x > P.cullMargin && p.x < P.Lx - P.cullMargin && p.y > P.cullMargin &&
        p.y < P.Ly - P.cullMargin) {
        const float reach = (r + P.rmax) * 1.0001f + P.cullMargin;
        // the cell's lower corner; a row window's rows are the scene's from rowOff
        const float X0 = (float)g.x * P.cellW, Y0 = (float)(g.y + P.rowOff) * P.cellH;
        if (p.x - X0 > reach) x0 = 0;
        if (X0 + P.cellW - p.x > reach) x1 = 0;
        if (p.y - Y0 > reach) y0 = 0;
        if (Y0 + P.cellH - p.y > reach) y1 = 0;
        const float rr = (r + P.rmax) * 1.0001f;
        reach2 = rr * rr;
    }
#pragma unroll 1
    for (int dy = y0; dy <= y1; ++dy) {
#pragma unroll 1
        for (int dx = x0; dx <= x1; ++dx) {
            const uint2 se = cells.get(cell_index(P, g.x + dx, g.y + dy));
            float2 fc = make_float2(0.0f, 0.0f);
            // empty cells have start >= end (start 0xFFFFFFFF): no iterations
            const uint32_t count = se.y > se.x ? se.y - se.x : 0u;
            const uint32_t stop = se.x + (count & ~1u);
            uint32_t j = se.x;
            // two candidates per iteration: two loads in flight
#pragma unroll 1
            for (; j < stop; j += 2) {
                const float2 pa = __ldg(pos + j);
                const float2 pb = __ldg(pos + j + 1);
                const float ax = pa.x - p.x, ay = pa.y - p.y;
                const float bx = pb.x - p.x, by = pb.y - p.y;
                const float da = ax * ax + ay * ay;
                const float db = bx * bx + by * by;
                if (j != i && (ATTRACT || !CULL || da <= reach2))
                    candidate<TYPED, ATTRACT>(P, j, p, v, w, r, mat, pa, da, vel, omega, radius,
                                              type, src, fc, moment, pr);
                if (j + 1 != i && (ATTRACT || !CULL || db <= reach2))
                    candidate<TYPED, ATTRACT>(P, j + 1, p, v, w, r, mat, pb, db, vel, omega,
                                              radius, type, src, fc, moment, pr);
            }
            if ((count & 1u) && j != i) {
                const float2 pa = __ldg(pos + j);
                const float ax = pa.x - p.x, ay = pa.y - p.y;
                const float da = ax * ax + ay * ay;
                if (ATTRACT || !CULL || da <= reach2)
                    candidate<TYPED, ATTRACT>(P, j, p, v, w, r, mat, pa, da, vel, omega, radius,
                                              type, src, fc, moment, pr);
            }
            force.x += fc.x;
            force.y += fc.y;
        }
    }
}

// particles_kernel.cuh:520-541: the contact (and attraction) with the control
// particle after the 3x3 cells; its force is added once, the reaction is stored
// (at `at`, the particle's place in sorted order) for the reduction.
template <bool TYPED, bool ATTRACT>
__device__ __forceinline__ void meet_control(const KParams& P, const ControlArgs& ctl, uint32_t at,
                                             float2 p, float2 v, float w, float r, uint32_t mat,
                                             float2& f, float& moment, float& pr) {
    const ControlDev c = *ctl.c;
    const float4 pc = TYPED ? P.pair[mat * P.nmat + c.mat] : P.pair[0];
    float mc = 0.0f;
    float2 fc = pair_force(p, c.pos, v, c.vel, w, c.omega, r, c.radius, pc, P.dt, mc, pr);
    if (ATTRACT) {
        const float2 fa = pair_attract(p, c.pos, r, c.radius, P.at[mat], P.at[c.mat], pr);
        fc.x += fa.x;
        fc.y += fa.y;
    }
    f.x += fc.x;
    f.y += fc.y;
    moment += mc;
    ctl.fx[at] = -fc.x;
    ctl.fy[at] = -fc.y;
    ctl.fm[at] = -mc / r * c.radius;
}

// Row-interval form of collide_one for the context step (no attraction, no
// x-wrap among the visited columns).  The cells (cx-1, cx, cx+1) of one row
// are consecutive cells, so their particles form one contiguous index
// interval in sorted order, read from the first-particle array (cellFirst,
// `pitch` words a row).
// A lane walks the interval of each row it visits after culling, one row
// after the other, so the lanes of a warp run about as many iterations as
// their own candidates in that row instead of the per-cell maximum.
// Positions and radii are in sorted order; a contact's velocity, spin and
// type are read at the neighbour's slot of the previous order, src[j].
//
// Each interval is walked twice, in chunks of 32 candidates: a lean filter
// sets one bit per candidate whose squared distance is within
// (rA + rB)^2 (1 + 2e-6), up to rounding -- a superset of the contacts -- and the contact
// law then runs on the set bits in increasing index.  The law's own
// `dist < rA + rB` test rejects the few non-contacts among them with a +0
// force, which changes no sum, so every contact is met in the same
// (row, index) order as before.  Keeping the law out of the filter loop
// means a warp runs it once per contact of its busiest lane rather than once
// per candidate slot in which any lane has a contact.
//
// The summation order is the reference's: the cell a contact belongs to is
// found from the cell boundaries, each row keeps one subtotal per cell and
// adds them to the force in cell order at the end of the row (an empty or
// culled cell adds +0, which changes nothing).  Returns false, without
// touching the outputs, when the visited columns wrap; the caller then uses
// collide_one.
//
// With ATTRACT the filter keeps the candidates within attraction reach
// (attract_reach2, a superset of the contacts), and a neighbour column or row
// is skipped beyond the largest such reach (exact where culling is: a cell met
// across the grid's wrap is at least 4 rmax away).
template <bool TYPED, bool ATTRACT>
__device__ __forceinline__ bool collide_rows(const KParams& P, uint32_t i, int2 g, float2 p,
                                             float2 v, float w, float r, uint32_t mat,
                                             const float2* __restrict__ pos,
                                             const float2* __restrict__ vel,
                                             const float* __restrict__ omega,
                                             const float* __restrict__ radius,
                                             const uint32_t* __restrict__ type,
                                             const uint32_t* __restrict__ src,
                                             const uint32_t* __restrict__ cellFirst,
                                             uint32_t pitch, float2& force, float& moment,
                                             float& pr) {
    // a radius that is not positive has no attraction reach (see attract_reach2)
    if (ATTRACT && !(r > 0.0f)) return false;
    int y0 = -1, y1 = 1, x0 = -1, x1 = 1;
    if (p.x > P.cullMargin && p.x < P.Lx - P.cullMargin && p.y > P.cullMargin &&
        p.y < P.Ly - P.cullMargin) {
        const float reach = (ATTRACT ? kAttractReach * P.rmax : r + P.rmax) * 1.0001f + P.cullMargin;
        const float X0 = (float)g.x * P.cellW, Y0 = (float)(g.y + P.rowOff) * P.cellH;
        if (p.x - X0 > reach) x0 = 0;
        if (X0 + P.cellW - p.x > reach) x1 = 0;
        if (p.y - Y0 > reach) y0 = 0;
        if (Y0 + P.cellH - p.y > reach) y1 = 0;
    }
    if (g.x + x0 < 0 || g.x + x1 >= (int)P.gx) return false;
    force = make_float2(0.0f, 0.0f);
    moment = 0.0f;
    pr = 0.0f;
    const float4 pc0 = P.pair[0];
#pragma unroll 1
    for (int dy = y0; dy <= y1; ++dy) {
        const uint32_t row = P.cellOff + (uint32_t)((g.y + dy) & (int)(P.gy - 1u)) * pitch;
        // the visited cells of this row are first = x0 .. x1; visited cell k
        // holds the particles
        // [start[first + k], start[first + k + 1]); a contact at index j
        // belongs to visited cell (j >= b1) + (j >= b2)
        const uint32_t* __restrict__ sc = cellFirst + (row + (uint32_t)(g.x + x0));
        const uint32_t o0 = __ldg(sc), o1 = __ldg(sc + 1), o2 = __ldg(sc + 2), o3 = __ldg(sc + 3);
        const int span = x1 - x0;  // visited cells - 1
        const uint32_t a = o0;
        const uint32_t b = span == 0 ? o1 : (span == 1 ? o2 : o3);
        const uint32_t b1 = span >= 1 ? o1 : 0xffffffffu;
        const uint32_t b2 = span >= 2 ? o2 : 0xffffffffu;
        float2 f0 = make_float2(0.0f, 0.0f), f1 = f0, f2 = f0;
        // filter: a bit per candidate that may touch, then the contact law on
        // the set bits in index order.  Groups of 8 candidates are read whole
        // (the arrays are padded by kFilterPad), the bits past the interval
        // and the particle's own bit are cleared per chunk.
#pragma unroll 1
        for (uint32_t base = a; base < b; base += 32u) {
            const uint32_t cnt = min(b - base, 32u);
            uint32_t mask = 0u;
#pragma unroll 1
            for (uint32_t k0 = 0; k0 < cnt; k0 += 8) {
                const uint32_t m8 =
                    filter8<ATTRACT>(pos + (base + k0), radius + (base + k0), p, r);
                mask |= m8 << k0;
            }
            if (cnt < 32u) mask &= (1u << cnt) - 1u;
            if (i - base < 32u) mask &= ~(1u << (i - base));
            while (mask) {
                const uint32_t j = base + (uint32_t)(__ffs(mask) - 1);
                mask &= mask - 1u;
                float2 fc = j >= b2 ? f2 : (j >= b1 ? f1 : f0);
                if (ATTRACT) {
                    const float2 pj = __ldg(pos + j);
                    const float ax = pj.x - p.x, ay = pj.y - p.y;
                    candidate<TYPED, true>(P, j, p, v, w, r, mat, pj, ax * ax + ay * ay, vel, omega,
                                           radius, type, src, fc, moment, pr);
                } else {
                    const float rj = __ldg(radius + j);
                    float4 pc = pc0;
                    const uint32_t sj = src ? __ldg(src + j) : j;
                    if (TYPED) pc = P.pair[mat * P.nmat + __ldg(type + sj)];
                    const float2 f = pair_force(p, __ldg(pos + j), v, __ldg(vel + sj), w,
                                                __ldg(omega + sj), r, rj, pc, P.dt, moment, pr);
                    fc.x += f.x;
                    fc.y += f.y;
                }
                if (j >= b2) f2 = fc;
                else if (j >= b1) f1 = fc;
                else f0 = fc;
            }
        }
        force.x += f0.x; force.y += f0.y;
        force.x += f1.x; force.y += f1.y;
        force.x += f2.x; force.y += f2.y;
    }
    return true;
}

}  // namespace dem
