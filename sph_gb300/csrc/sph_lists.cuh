// Pair lists for the DFSPH solves.
//
// Between two grid builds the DFSPH step never moves a particle: the
// divergence solve, the next step's warm start and its density solve all run
// at the positions of the last build (DFSPHSolver.cpp:63-97).  So right after
// each build one 27-cell walk computes the densities and alpha factors
// (SPHSolver.cpp:44-91, DFSPHSolver.cpp:114-189) and records, per particle,
// every fluid neighbour with a non-zero kernel gradient together with
// m * gradW_ij, plus the summed Akinci boundary gradient
// sum_b rho0 psi_b gradW_ib.  The solver walks then read those lists instead
// of rescanning ~216 candidates and re-evaluating the kernel per pair.
//
// Layout: slot-major, pairs[k * n + i] = {m gradW_ij, as_float(j)}, so the
// threads of a warp (consecutive particles) read one contiguous 16-byte line
// per slot.  A particle with more than kmax neighbours keeps its count and
// falls back to the cell walk in every list kernel.
//
// Neighbours are listed in the cell walk's order, so each fluid sum adds the
// same non-zero terms in the same order as the reference; the boundary sum is
// pre-added once per build (a re-association of the reference's boundary
// terms, which all share the factor of particle i).
#pragma once

#include <cuda_fp16.h>

#include <cstring>
#include <vector>

#include "sph_kernels.cuh"

namespace sph {

template <typename R> struct Lists {
    P4<R>* pairs;       // kmax * n, slot-major: {m gradW_ij, as-bits j}
    uint32_t* count;    // neighbours with a non-zero gradient (may exceed kmax)
    P4<R>* bgrad;       // xyz: sum_b rho0 psi_b gradW_ib
    R* kbuf;            // k (or kv) of the pass in progress
    uint32_t kmax;
    // A half-precision copy of the cell-relative positions for the build's
    // cull, two particles per 16-byte word ({x, y, z, unused}
    // half2 pairs, z in the cell's modulo-3 frame), or nullptr
    const uint4* posh;
    unsigned* fault;    // status word of the bounds-checked build (SPH_INDEX_OK)
    // Akinci boundary points in the same half-precision form (static between
    // re-layouts) and their cells, for the boundary cull; or nullptr
    const uint4* bposh;
    const uint32_t* bcell;
};

// Where a density pass writes the candidate lists (CandLists, sph_kernels.cuh).
struct CandOut {
    uint32_t* idx;
    uint32_t* cnt;
    uint32_t* bcnt;
    uint32_t kmax;           // slots per lane
    uint32_t lanes;          // lanes per particle of the passes that visit the lists
    const uint4* posh;       // half-precision positions (fluid, boundary or nullptr)
    const uint4* bposh;
    const uint32_t* bcell;
};

// cell offset code of a candidate in cell cj around cell ci (walk_reach's)
__device__ __forceinline__ uint32_t cell_code(uint32_t ci, uint32_t cj)
{
    return (uint32_t)((cell_x(cj) - cell_x(ci) + 1) * 9 + (cell_y(cj) - cell_y(ci) + 1) * 3 + (cell_z(cj) - cell_z(ci) + 1));
}

enum Rank { kNoRank, kCellRank, kColumnRank };

__device__ __forceinline__ __half2 as_half2(uint32_t u) { return *reinterpret_cast<const __half2*>(&u); }

// The scaled quantities of the half-precision test of one particle.
struct HalfTest {
    float x, y, h;  // position in its cell's frame, support radius
    __half2 zq, h3, thr;
};
__device__ __forceinline__ HalfTest half_test(V3<float> xi, int cz, float h, float reach2)
{
    const float sc = half_scale(h);
    return HalfTest{xi.x * sc, xi.y * sc, h * sc, __float2half2_rn(zframe3(xi.z, cz, h) * sc), __float2half2_rn(3.f * h * sc),
                    __float2half2_rn(reach2 * 1.03f * (sc * sc))};
}

// Phase 1 of the list build from the half-precision positions: the
// nine columns of the 27-cell neighbourhood (trimmed as walk() trims them),
// two candidates per half2 operation, accepted indices queued in walk order.
// The caller guarantees that the particle's cell is at least two cells from
// every face of the grid box (all 27 cells exist and hold in-grid particles,
// offsets in [0, h)) and that its own offsets are inside [-h/2, 3h/2].
//
// z needs no per-candidate cell: positions carry z in the frame of their
// cell's z index modulo 3 (in [0, 3h)), so for a candidate in cells
// z-1..z+1 the difference d of the two frame values is the true z distance
// plus a multiple of 3h, and min(|d|, 3h - |d|) is the true |dz| whenever
// |dz| <= 1.5h and above h (so culled) otherwise, up to a sliver of
// |dz| in [1.97h, 2h) that phase 2 drops.
//
// The test uses r^2 <= 1.03 h^2: for a pair within h, half-precision values
// (relative error 2^-11 each; x, y operands within 2.5h, z within 3h)
// move r^2 by less than 1.7 % of h^2, so every pair the exact test accepts
// is kept; pairs beyond h evaluate to W = 0, grad W = 0 in phase 2 and are
// dropped there.  Lengths are scaled by a power of two that brings h into
// [1, 2) (half_scale; exact, so the same bound for any unit of length): the
// values stay within 6 and their squares within 36, and half precision's
// subnormal step of 6e-8 is nothing beside them.  Returns the number of
// accepted candidates (the queue holds the first qcap).
//
// reach2: the square of the distance wanted, up to (1.1 h)^2 (candidate lists;
// the same bounds scale to 1.9 % of h^2 against a slack of 3.6 %, and a true
// |dz| above 1.9 h may read as little as h: such candidates are dropped by
// the exact test on the queued ones).
//
// RANK: each queued candidate with the lane whose part of a cell walk by
// `lanes` lanes it is, above the index's 27 bits: its rank modulo the lanes
// in its cell (kCellRank, the FP32 walk) or in its column (kColumnRank, FP64).
template <Rank RANK = kNoRank>
__device__ __forceinline__ uint32_t cull_half(const GridView& g, const uint32_t* __restrict__ starts, uint32_t pc,
                                              V3<float> xi, float h, float reach2, const uint4* __restrict__ posh,
                                              uint32_t* q, uint32_t qstride, uint32_t qcap, uint32_t lanes = 1u)
{
    const int cx = cell_x(pc), cy = cell_y(pc), cz = cell_z(pc);
    const float ofx = xi.x, ofy = xi.y, ofz = xi.z;
    const float gxm = ofx > 0.f ? ofx * ofx : 0.f, gxp = h - ofx > 0.f ? (h - ofx) * (h - ofx) : 0.f;
    const float gym = ofy > 0.f ? ofy * ofy : 0.f, gyp = h - ofy > 0.f ? (h - ofy) * (h - ofy) : 0.f;
    const float gzm = ofz > 0.f ? ofz * ofz : 0.f, gzp = h - ofz > 0.f ? (h - ofz) * (h - ofz) : 0.f;
    const float lim = fmaxf(reach2, h * h) * (float)(1.0 + 1e-5);
    const HalfTest ht = half_test(xi, cz, h, reach2);
    uint32_t nq = 0;
    // a column's candidate range (empty when trimmed); loaded one column ahead
    auto range = [&](int c, uint32_t* b, uint32_t* e, uint32_t* s1, uint32_t* s2) {
        const int dx = c / 3 - 1, dy = c - (c / 3) * 3 - 1;
        const float gxy = (dx < 0 ? gxm : (dx > 0 ? gxp : 0.f)) + (dy < 0 ? gym : (dy > 0 ? gyp : 0.f));
        if (!(gxy <= lim)) { *b = 0u; *e = 0u; return; }
        const uint32_t base = (__ldg(g.mortx + cx + dx) | __ldg(g.morty + cy + dy)) * (uint32_t)g.nz;
        *b = __ldg(starts + base + (gxy + gzm <= lim ? cz - 1 : cz));
        *e = __ldg(starts + base + (gxy + gzp <= lim ? cz + 2 : cz + 1));
        if constexpr (RANK == kCellRank) {
            *s1 = __ldg(starts + base + cz);
            *s2 = __ldg(starts + base + cz + 1);
        }
        if constexpr (RANK == kColumnRank) *s1 = __ldg(starts + base + cz - 1);
    };
    uint32_t nb, ne, n1 = 0u, n2 = 0u;
    range(0, &nb, &ne, &n1, &n2);
#pragma unroll 1
    for (int c = 0; c < 9; ++c) {
        const int dx = c / 3 - 1, dy = c - (c / 3) * 3 - 1;
        const uint32_t bb = nb, ee = ne, s1 = n1, s2 = n2;
        if (c < 8) range(c + 1, &nb, &ne, &n1, &n2);
        const __half2 sx = __float2half2_rn(ht.x - (float)dx * ht.h), sy = __float2half2_rn(ht.y - (float)dy * ht.h);
        // The column's candidates 32 at a time (16 words): the test's
        // acceptance bits are gathered into one word, candidate j0 + b at
        // bit b, and only the accepted candidates (about one in five) are
        // queued, in walk order.
        for (uint32_t j0 = bb & ~1u; j0 < ee; j0 += 32) {
            const uint32_t nw = min(16u, (ee - j0 + 1) >> 1);
            const uint4* __restrict__ wp = posh + (j0 >> 1);
            // acceptance mask of one word: 0xffff per accepted half
            auto test = [&](const uint4 w) {
                const __half2 ddx = __hsub2(sx, as_half2(w.x));
                const __half2 ddy = __hsub2(sy, as_half2(w.y));
                const __half2 dz = __habs2(__hsub2(ht.zq, as_half2(w.z)));
                const __half2 ddz = __hmin2(dz, __hsub2(ht.h3, dz));
                const __half2 r2 = __hfma2(ddz, ddz, __hfma2(ddy, ddy, __hmul2(ddx, ddx)));
                return __hle2_mask(r2, ht.thr);
            };
            // Two words (four candidates) per iteration: bytes 0 and 2 of
            // each mask (one per half) gathered into one word, then bit 8k+k
            // of that word's byte k moved to bit 24+k by one multiply (the
            // shifted copies land on distinct bits, so nothing carries).  An
            // odd word count reads one word past the range (the buffer holds
            // a spare word); its bits are cleared below.
            uint32_t bits = 0;
#pragma unroll 1
            for (uint32_t k = 0; k < nw; k += 2) {
                const unsigned m0 = test(__ldg(wp + k)), m1 = test(__ldg(wp + k + 1));
                const uint32_t u = __byte_perm(m0, m1, 0x6420u) & 0x08040201u;
                bits |= ((u * 0x01010101u) >> 24) << (2 * k);
            }
            if (nw < 16u) bits &= (1u << (2 * nw)) - 1u;
            // the first word's low particle may precede the column's range
            // (bb odd), the last word's high one follow it (ee odd)
            if (j0 < bb) bits &= ~1u;
            if (j0 + 2 * nw > ee) bits &= ~(1u << (2 * nw - 1));
            while (bits) {
                const uint32_t b = __ffs(bits) - 1;
                bits &= bits - 1;
                uint32_t x = j0 + b;
                if constexpr (RANK == kColumnRank) x |= ((x - s1) & (lanes - 1)) << kCandIdxBits;
                if constexpr (RANK == kCellRank) x |= ((x - (x < s1 ? bb : (x < s2 ? s1 : s2))) & (lanes - 1)) << kCandIdxBits;
                if (nq < qcap) q[nq * qstride + threadIdx.x] = x;
                ++nq;
            }
        }
    }
    return nq;
}

// Whether the half-precision cull serves a particle (see cull_half), and its
// position in its cell's frame.  (h beyond 1e15 either way: h^2 or its FP32
// gaps leave FP32.)
template <typename R>
__device__ __forceinline__ bool half_cull_ok(const GridView& g, uint32_t pc, V3<R> xi, R h, V3<float>* xr)
{
    const int cx = cell_x(pc), cy = cell_y(pc), cz = cell_z(pc);
    if constexpr (sizeof(R) == 4) *xr = xi;
    else *xr = V3<float>{(float)(xi.x - (R)(cx + g.ox) * h), (float)(xi.y - (R)(cy + g.oy) * h),
                         (float)(xi.z - (R)(cz + g.oz) * h)};
    const float hf = (float)h, hh = 0.5f * hf;
    return hf >= 1e-15f && hf <= 1e15f && cx >= 2 && cy >= 2 && cz >= 2 && cx <= g.nx - 3 && cy <= g.ny - 3 && cz <= g.nz - 3 &&
           fabsf(xr->x - hh) <= hf && fabsf(xr->y - hh) <= hf && fabsf(xr->z - hh) <= hf;
}

__device__ __forceinline__ float idx_as(float, uint32_t j) { return __uint_as_float(j); }
__device__ __forceinline__ double idx_as(double, uint32_t j) { return __longlong_as_double((long long)j); }
__device__ __forceinline__ uint32_t as_idx(float w) { return __float_as_uint(w); }
__device__ __forceinline__ uint32_t as_idx(double w) { return (uint32_t)__double_as_longlong(w); }

// Densities + alpha + the lists, one thread per particle, in two phases:
// the cell walk only culls candidates (distance test) and queues the
// accepted indices in shared memory; the kernel values are then evaluated in
// a dense loop over the queue.  (Evaluating inside the walk makes each warp
// execute the expensive branch on nearly every candidate, since some lane
// almost always accepts.)  A particle whose queue overflows is evaluated
// inside the walk instead.
constexpr uint32_t kQueue = 64;

template <typename R>
__device__ __forceinline__ V3<R> pair_vec(V3<R> xi, uint32_t ci, const P4<R>& pj, uint32_t cj, R h)
{
    if constexpr (sizeof(R) == 4) {
        const V3<R> s = {xi.x - (R)(cell_x(cj) - cell_x(ci)) * h, xi.y - (R)(cell_y(cj) - cell_y(ci)) * h,
                         xi.z - (R)(cell_z(cj) - cell_z(ci)) * h};
        return s - xyz(pj);
    } else {
        return xi - xyz(pj);
    }
}

// Per-particle body shared by the single-scene and the pool kernels; q is
// the block's shared queue (kQueue x kBlock).
template <typename R> struct BuildSums {
    R density, sumSq;
    V3<R> sumGrad;
    uint32_t cnt;
};

// A record, stored in 16-byte parts.  Of the one 32-byte store of an FP64
// record the compiler (CUDA 13.0) made nothing in build_walk_all, in all but
// one of its callers' forms: right sums, and lists of whatever the memory held.
// No condition for that is known, so every FP64 record is stored this way.
__device__ __forceinline__ void store_record(P4<float>* d, V3<float> v, uint32_t j) { *d = P4<float>{v.x, v.y, v.z, idx_as(0.f, j)}; }
__device__ __forceinline__ void store_record(P4<double>* d, V3<double> v, uint32_t j)
{
    asm volatile("st.global.v2.f64 [%0], {%1, %2};" ::"l"(d), "d"(v.x), "d"(v.y) : "memory");
    asm volatile("st.global.v2.f64 [%0 + 16], {%1, %2};" ::"l"(d), "d"(v.z), "d"(idx_as(0.0, j)) : "memory");
}

// Particles whose candidates overflow the shared queue: the whole
// evaluation inside the walk.  Out of line, so the common path's register
// allocation does not carry it.
template <typename R, bool FAST>
__device__ __noinline__ BuildSums<R> build_walk_all(uint32_t i, const Fluid<R>& f, const GridView& g,
                                                    const uint32_t* __restrict__ cs, const Consts<R>& c, const Lists<R>& L,
                                                    V3<R> xi, uint32_t pc)
{
    const uint32_t n = f.n;
    BuildSums<R> b{0, 0, {0, 0, 0}, 0};
    walk<R, 1>(g, cs, pc, xi, c.h, 0, [&](uint32_t j, V3<R> s) {
        const V3<R> r = s - xyz(ldg4(f.pos + j));
        const R r2 = dot3(r, r);
        if (!(r2 <= c.cull2)) return;
        R w;
        V3<R> gw;
        cubic_W_gradW<FAST>(c, r, r2, &w, &gw);
        b.density += c.mass * w;
        const V3<R> mg = c.mass * gw;
        const R mg2 = dot3(mg, mg);
        if (mg2 > (R)0) {
            b.sumGrad = b.sumGrad + mg;
            if constexpr (sizeof(R) == 8) {
                const R m = sqrt(mg2);
                b.sumSq += m * m;
            } else {
                b.sumSq += mg2;
            }
            if (b.cnt < L.kmax) store_record(L.pairs + (size_t)b.cnt * n + i, mg, j);
            ++b.cnt;
        }
    });
    return b;
}

// The dot product of the velocity divergence terms with its rounding written
// out (FP32: the contraction the compiler chose for the pass over the lists
// first), so that the sums of the one-scene build and of its passes agree bit
// for bit.  The pool's kernels (kPool) keep the plain expression, whose
// contraction differs from one copy of its unrolled loop to the next.
template <Rounding WHERE = kOneScene, typename R> __device__ __forceinline__ R dot3_div(V3<R> a, V3<R> b)
{
    if constexpr (sizeof(R) == 8 || WHERE == kPool) return dot3(a, b);
    else return __fmaf_rn(a.z, b.z, __fmaf_rn(a.x, b.x, __fmul_rn(a.y, b.y)));
}

// The other contraction of a dot product.
template <Rounding WHERE = kOneScene, typename R> __device__ __forceinline__ R dot3_zyx(V3<R> a, V3<R> b)
{
    if constexpr (sizeof(R) == 8 || WHERE == kPool) return dot3(a, b);
    else return __fmaf_rn(a.z, b.z, __fmaf_rn(a.y, b.y, __fmul_rn(a.x, b.x)));
}

// a * b + c and a + b of the one-scene builds: fused in FP32, two roundings in
// the FP64 parity form (compiled without contraction).
template <Rounding WHERE = kOneScene, typename R> __device__ __forceinline__ R mul_add(R a, R b, R c)
{
    if constexpr (WHERE == kPool) return a * b + c;
    else if constexpr (sizeof(R) == 8) return __dadd_rn(__dmul_rn(a, b), c);
    else return __fmaf_rn(a, b, c);
}
template <Rounding WHERE = kOneScene, typename R> __device__ __forceinline__ R plain_add(R a, R b)
{
    if constexpr (WHERE == kPool) return a + b;
    else if constexpr (sizeof(R) == 8) return __dadd_rn(a, b);
    else return __fadd_rn(a, b);
}

// Forward declarations: the list build's DIV0 form ends with the velocity
// divergence the first divergence-error pass would compute from the lists.
template <typename R> struct DivSum;
template <typename R>
__device__ __noinline__ DivSum<R> velocity_div_cells(const Fluid<R>& f, const P4<R>* __restrict__ bpos, const GridView& g,
                                                     const uint32_t* __restrict__ cs, const uint32_t* __restrict__ bs,
                                                     const Consts<R>& c, int akinci, uint32_t i, V3<R> vi);

template <typename R, Rounding WHERE = kOneScene>
__device__ __noinline__ R reread_div(const Fluid<R>& f, const Lists<R>& L, uint32_t i, V3<R> vi, uint32_t cnt)
{
    const uint32_t n = f.n;
    R dv = 0;
    for (uint32_t k = 0; k < cnt; ++k) {
        const P4<R> pr = L.pairs[(size_t)k * n + i];
        const uint32_t j = as_idx(pr.w);
        if (!SPH_INDEX_OK(j, n, L.fault)) continue;
        dv += dot3_div<WHERE>(vi - xyz(f.vel[j]), xyz(pr));
    }
    return dv;
}

// EB: queued candidates evaluated per round, their loads in flight together.
// The one-scene build has one wave of blocks or less up to ~130k particles and
// waits for its loads (EB = 4); the pool's is bound by issue slots (EB = 1).
//
// DIV0: also sum m (v_i - v_j) . gradW_ij over the pairs as they are listed,
// plus v_i . (boundary gradient): the value velocity_div_one would read from
// the finished lists (same terms, same order), into *div0, with the count of
// neighbours into *nn0 (a particle whose list or queue overflowed takes the
// same list or cell walk as velocity_div_one).
// CAND (scenes with non-pressure forces): also the candidate list those
// forces' passes visit, every candidate within their cull.
template <typename R, bool FAST = false, bool DIV0 = false, int EB = 1, Rounding WHERE = kOneScene, bool CAND = false>
__device__ __forceinline__ void build_lists_one(uint32_t i, const Fluid<R>& f, const P4<R>* __restrict__ bpos,
                                                const GridView& g, const uint32_t* __restrict__ cs,
                                                const uint32_t* __restrict__ bs, const Consts<R>& c, int akinci,
                                                const Lists<R>& L, uint32_t* q, uint32_t qstride = kBlock,
                                                uint32_t qdepth = kQueue, R* div0 = nullptr, uint32_t* nn0 = nullptr,
                                                const CandOut& o = CandOut{})
{
    const uint32_t n = f.n;
    const V3<R> xi = xyz(f.pos[i]);
    const uint32_t pc = f.cell[i];
    const uint32_t qcap = L.kmax < qdepth ? L.kmax : qdepth;
    R density = 0, sumSq = 0;
    V3<R> sumGrad = {0, 0, 0};
    uint32_t cnt = 0;
    V3<R> vi = {0, 0, 0};
    if constexpr (DIV0) vi = xyz(f.vel[i]);
    R dv = 0;
    // vj: the neighbour's velocity (DIV0), loaded beside its position
    auto accept = [&](uint32_t j, V3<R> r, R r2, V3<R> vj) {
        R w;
        V3<R> gw;
        cubic_W_gradW<FAST>(c, r, r2, &w, &gw);
        density = mul_add<WHERE>(c.mass, w, density);
        const V3<R> mg = c.mass * gw;
        const R mg2 = dot3_div<WHERE>(mg, mg);
        if (mg2 > (R)0) {
            sumGrad = V3<R>{plain_add<WHERE>(sumGrad.x, mg.x), plain_add<WHERE>(sumGrad.y, mg.y), plain_add<WHERE>(sumGrad.z, mg.z)};
            if constexpr (sizeof(R) == 8) {
                const R m = sqrt(mg2);
                sumSq += m * m;
            } else {
                sumSq = plain_add<WHERE>(sumSq, mg2);
            }
            if (cnt < L.kmax) store_record(L.pairs + (size_t)cnt * n + i, mg, j);
            ++cnt;
            if constexpr (DIV0) dv += dot3_div<WHERE>(vi - vj, mg);
        }
    };
    // phase 1: cull.  The half-precision cull needs all 27 cells inside the
    // grid box and clear of its border cells (where particles that left the
    // box are kept, with unbounded offsets), and in-cell offsets; elsewhere
    // the cull runs in R.
    uint32_t nq = 0;
    bool half_cull = false;
    V3<float> xr;  // the position in its cell's frame
    half_cull = L.posh && half_cull_ok(g, pc, xi, c.h, &xr);
    constexpr Rank RANK = !CAND ? kNoRank : (sizeof(R) == 4 ? kCellRank : kColumnRank);
    if (half_cull) nq = cull_half<RANK>(g, cs, pc, xr, (float)c.h, (float)c.cull2, L.posh, q, qstride, qcap, o.lanes);
    if (!half_cull)
        walk<R, 1, true, FAST>(g, cs, pc, xi, c.h, 0, [&](uint32_t j, V3<R> s) {
            const V3<R> r = s - xyz(ldg4(f.pos + j));
            if (dot3(r, r) <= c.cull2) {
                if (nq < qcap) q[nq * qstride + threadIdx.x] = j;
                ++nq;
            }
        });
    // CAND: the candidate lists, one per lane of the force passes (CandLists);
    // x: a queued candidate with its lane.  Counts packed in bytes.
    unsigned long long nl = 0, nlf = 0;
    auto list = [&](uint32_t x, uint32_t cj, R r2) {
        if (!(r2 <= c.cull2)) return;
        const uint32_t t = x >> kCandIdxBits, slot = (uint32_t)(nl >> (8 * t)) & 255u;
        if (slot < o.kmax) o.idx[((size_t)slot * n + i) * o.lanes + t] = (x & kCandIdxMask) | (cell_code(pc, cj) << kCandIdxBits);
        nl += 1ull << (8 * t);
    };
    bool fwalk = !half_cull, bwalk = !half_cull;  // its force passes walk
    if (nq <= qcap) {
        // phase 2: evaluate the queued candidates in walk order
        for (uint32_t k = 0; k < nq; k += EB) {
            uint32_t j[EB], cj[EB], x[EB];
            P4<R> pj[EB];
            V3<R> vj[EB];
#pragma unroll
            for (int b = 0; b < EB; ++b) {
                // (past the end: the last candidate once more, not evaluated)
                x[b] = q[(EB == 1 || k + b < nq ? k + b : nq - 1) * qstride + threadIdx.x];
                j[b] = CAND ? x[b] & kCandIdxMask : x[b];
                // (a plain load for the velocity: other threads write its w here)
                vj[b] = V3<R>{0, 0, 0};
                if constexpr (DIV0) vj[b] = xyz(f.vel[j[b]]);
                pj[b] = ldg4(f.pos + j[b]);
                cj[b] = CAND || sizeof(R) == 4 ? __ldg(f.cell + j[b]) : 0u;
            }
#pragma unroll
            for (int b = 0; b < EB; ++b) {
                if (EB > 1 && k + b >= nq) break;
                const V3<R> r = pair_vec(xi, pc, pj[b], cj[b], c.h);
                if constexpr (CAND) list(x[b], cj[b], dot3(r, r));
                accept(j[b], r, dot3(r, r), vj[b]);
            }
        }
    } else {
        const BuildSums<R> b = build_walk_all<R, FAST>(i, f, g, cs, c, L, xi, pc);
        density = b.density;
        sumSq = b.sumSq;
        sumGrad = b.sumGrad;
        cnt = b.cnt;
        fwalk = true;
    }
    nlf = nl;
    V3<R> bg = {0, 0, 0};
    if (akinci) {
        auto bterm = [&](const P4<R>& pb, V3<R> r) {
            const R r2 = dot3(r, r);
            if (!(r2 <= c.cull2)) return;
            R w;
            V3<R> gw;
            cubic_W_gradW<FAST>(c, r, r2, &w, &gw);
            density = mul_add<WHERE>(pb.w, w, density);
            bg = V3<R>{mul_add<WHERE>(pb.w, gw.x, bg.x), mul_add<WHERE>(pb.w, gw.y, bg.y), mul_add<WHERE>(pb.w, gw.z, bg.z)};
        };
        // The boundary candidates as the fluid ones: culled from the static
        // half-precision copy into the (now free) queue, then evaluated in
        // the walk's order (the same cells, trimmed alike: the same terms in
        // the same order as the walk, the gradient sum compiled apart from
        // the walk's, so its last bit may differ); or the walk itself.
        uint32_t nb = qcap + 1u;
        if (half_cull && L.bposh) nb = cull_half<RANK>(g, bs, pc, xr, (float)c.h, (float)c.cull2, L.bposh, q, qstride, qcap, o.lanes);
        if (nb <= qcap) {
            for (uint32_t k = 0; k < nb; k += EB) {
                P4<R> pb[EB];
                uint32_t cb[EB], x[EB];
#pragma unroll
                for (int b = 0; b < EB; ++b) {
                    x[b] = q[(EB == 1 || k + b < nb ? k + b : nb - 1) * qstride + threadIdx.x];
                    const uint32_t j = CAND ? x[b] & kCandIdxMask : x[b];
                    pb[b] = ldg4(bpos + j);
                    cb[b] = CAND || sizeof(R) == 4 ? __ldg(L.bcell + j) : 0u;
                }
#pragma unroll
                for (int b = 0; b < EB; ++b) {
                    if (EB > 1 && k + b >= nb) break;
                    const V3<R> r = pair_vec(xi, pc, pb[b], cb[b], c.h);
                    if constexpr (CAND) list(x[b], cb[b], dot3(r, r));
                    bterm(pb[b], r);
                }
            }
        } else {
            bwalk = true;
            walk<R, 1>(g, bs, pc, xi, c.h, 0, [&](uint32_t j, V3<R> s) {
                const P4<R> pb = ldg4(bpos + j);
                bterm(pb, s - xyz(pb));
            });
        }
    }
    sumGrad = V3<R>{plain_add<WHERE>(sumGrad.x, bg.x), plain_add<WHERE>(sumGrad.y, bg.y), plain_add<WHERE>(sumGrad.z, bg.z)};
    f.rho[i] = density;
    f.vel[i].w = density;
    R den;
    if constexpr (sizeof(R) == 8) {
        const R m = sqrt(dot3(sumGrad, sumGrad));
        den = m * m + sumSq;
    } else {
        den = dot3_zyx<WHERE>(sumGrad, sumGrad) + sumSq;
    }
    f.alpha[i] = (fabs(den) > c.eps) ? density / den : (R)0;
    L.count[i] = cnt;
    L.bgrad[i] = P4<R>{bg.x, bg.y, bg.z, 0};
    if constexpr (CAND) {
        for (uint32_t t = 0; t < o.lanes; ++t) {
            const uint32_t m = (uint32_t)(nlf >> (8 * t)) & 255u, all = (uint32_t)(nl >> (8 * t)) & 255u;
            o.cnt[(size_t)i * o.lanes + t] = fwalk ? o.kmax + 1u : m;
            o.bcnt[(size_t)i * o.lanes + t] = bwalk ? o.kmax + 1u : all - m;
        }
    }
    if constexpr (DIV0) {
        if (cnt > L.kmax) {
            const DivSum<R> d = velocity_div_cells(f, bpos, g, cs, bs, c, akinci, i, vi);
            *div0 = d.dv;
            *nn0 = d.nn;
        } else {
            if (nq > qcap) dv = reread_div<R, WHERE>(f, L, i, vi, cnt);
            if (akinci) dv += dot3_div<WHERE>(vi, bg);
            *div0 = dv;
            *nn0 = cnt;
        }
    }
}

// A particle's first divergence error from its velocity divergence
// (computeDivergenceError's clamps and k; DFSPHSolver.cpp:468-486).
template <typename R>
__device__ __forceinline__ double divergence_error(uint32_t i, const Fluid<R>& f, const Lists<R>& L, const Consts<R>& c, R dt,
                                                   R dv, uint32_t nn)
{
    dv = nn < 20u ? (R)0 : (dv < (R)0 ? (R)0 : dv);
    f.div[i] = dv;
    L.kbuf[i] = dv * f.alpha[i] / (dt * f.rho[i]);
    return rel_error(c, (double)dv);
}

// The divergence solve's loop control after an error pass (INITIAL: before the
// first iteration; DFSPHSolver.cpp:505-585).  One thread.
template <bool INITIAL>
__device__ __forceinline__ void divergence_control(DevScalars* sc, const LoopLimits& lim, double total, uint32_t n,
                                                   cudaGraphConditionalHandle cond)
{
    const double avg = total / (double)n;
    const double lim_v = lim.maxErrorV / sc->dt;
    if (!isfinite(avg)) sc->status |= ST_NONFINITE;
    if (INITIAL) {
        sc->iterationsV = 0;
        sc->avgDivError = avg;
        sc->active = (lim.minItV > 0u) && (lim.maxIt > 0u);
        if (!sc->active) sc->avgDivError = 0.0;
    } else {
        const unsigned it = ++sc->iterationsV;
        sc->avgDivError = avg;
        const unsigned act = ((avg > lim_v) || (it < lim.minItV)) && (it < lim.maxIt);
        sc->active = act;
        if (!act) {
            sc->sumIterationsV += it;
            if (it >= lim.maxIt && avg > lim_v) sc->status |= ST_ITER_CAP_V;
        }
    }
    if (cond) cudaGraphSetConditional(cond, sc->active);
}

// DIV0: the build of a step, which also forms the divergence solve's first
// error pass (its sums, its reduction and the first loop test): one pass over
// the lists and one launch less (13k dam break 164 -> 150 us/step, 125k 275 ->
// 265).  The half-precision cull serves FP64 too, whose distance test alone
// (9 FP64 operations on each of ~150 candidates, at two FP64 lanes per SM)
// was a third of the build: 125k particles 1454 -> 1003 us with the boundary's
// cull and the fused error pass.
template <typename R, bool DIV0, bool CAND, int BLOCK, int MINB, int EB, int QD>
__global__ void __launch_bounds__(BLOCK, MINB) k_build_lists(Fluid<R> f, const P4<R>* __restrict__ bpos, GridView g,
                                                           const uint32_t* __restrict__ cs, const uint32_t* __restrict__ bs,
                                                           Consts<R> c, int akinci, Lists<R> L, DevScalars* sc,
                                                           LoopLimits lim, double* partials, cudaGraphConditionalHandle cond,
                                                           CandOut o)
{
    grid_wait();
    __shared__ uint32_t q[QD * BLOCK];
    const uint32_t i = gtid();
    double err = 0.0;
    if (i < f.count()) {
        R dv = 0;
        uint32_t nn = 0;
        build_lists_one<R, sizeof(R) == 4, DIV0, EB, kOneScene, CAND>(i, f, bpos, g, cs, bs, c, akinci, L, q, BLOCK, QD, &dv,
                                                                  &nn, o);
        if (DIV0) err = divergence_error(i, f, L, c, (R)sc->dt, dv, nn);
    }
    if constexpr (DIV0) {
        __shared__ double sh[33];
        double total;
        if (finish_reduction<false>(err, partials, &sc->block_counter, sh, &total) && threadIdx.x == 0)
            divergence_control<true>(sc, lim, total, f.count(), cond);
    }
}

// ---- the list build with W lanes per particle --------------------------------
//
// A scene of a few thousand particles has fewer warps than the chip has
// schedulers, so one lane's build is one long chain of dependent loads (38 us
// for 2,000 particles as for 24,000; 14 us and 31 us here).  Here W lanes share a particle: each
// looks up its columns' ranges, tests its words of a column's candidates, and
// evaluates its part of the accepted ones; the values go to shared memory and
// are then summed one after another, each of the sums by a lane of its own,
// in the list's order and with the rounding of build_lists_one.  The results
// are bit-identical to it: the sums' rounding is written out in both; the
// distances' and the kernel values' contraction is the compiler's, the same in
// both so far, which test_build_lanes.py checks bit for bit.

constexpr uint32_t kWideBlock = 128, kWideChunk = 32;

// The candidate ranges of cull_half's nine columns, lane gl of W holding
// columns gl, gl + W, ...: in b[], e[] (empty where trimmed, or with !on).
// RANK: also what a candidate's rank is counted from.
template <int W, Rank RANK = kNoRank> struct WideRanges {
    static constexpr int C = (9 + W - 1) / W;
    uint32_t b[C], e[C], m0[RANK ? C : 1], m1[RANK ? C : 1];
};
template <int W, Rank RANK = kNoRank>
__device__ __forceinline__ WideRanges<W, RANK> wide_ranges(bool on, int gl, const GridView& g, const uint32_t* __restrict__ starts,
                                                     uint32_t pc, V3<float> xi, float h, float reach2)
{
    const int cx = cell_x(pc), cy = cell_y(pc), cz = cell_z(pc);
    const float ofx = xi.x, ofy = xi.y, ofz = xi.z;
    const float gxm = ofx > 0.f ? ofx * ofx : 0.f, gxp = h - ofx > 0.f ? (h - ofx) * (h - ofx) : 0.f;
    const float gym = ofy > 0.f ? ofy * ofy : 0.f, gyp = h - ofy > 0.f ? (h - ofy) * (h - ofy) : 0.f;
    const float gzm = ofz > 0.f ? ofz * ofz : 0.f, gzp = h - ofz > 0.f ? (h - ofz) * (h - ofz) : 0.f;
    const float lim = fmaxf(reach2, h * h) * (float)(1.0 + 1e-5);
    WideRanges<W, RANK> r;
#pragma unroll
    for (int t = 0; t < WideRanges<W>::C; ++t) {
        const int c = gl + t * W;
        r.b[t] = r.e[t] = 0u;
        if constexpr (RANK) r.m0[t] = r.m1[t] = 0u;
        if (on && c < 9) {
            const int dx = c / 3 - 1, dy = c % 3 - 1;
            const float gxy = (dx < 0 ? gxm : (dx > 0 ? gxp : 0.f)) + (dy < 0 ? gym : (dy > 0 ? gyp : 0.f));
            if (gxy <= lim) {
                const uint32_t base = (__ldg(g.mortx + cx + dx) | __ldg(g.morty + cy + dy)) * (uint32_t)g.nz;
                r.b[t] = __ldg(starts + base + (gxy + gzm <= lim ? cz - 1 : cz));
                r.e[t] = __ldg(starts + base + (gxy + gzp <= lim ? cz + 2 : cz + 1));
                if constexpr (RANK == kCellRank) {
                    r.m0[t] = __ldg(starts + base + cz);
                    r.m1[t] = __ldg(starts + base + cz + 1);
                }
                if constexpr (RANK == kColumnRank) r.m0[t] = __ldg(starts + base + cz - 1);
            }
        }
    }
    return r;
}

// cull_half by W lanes: accepted candidates in walk order into the group's
// queue; every lane returns their number.  gl = lane in the group; all lanes
// of the warp call it.  RANK: each with the lane whose part of the cell walk
// it is (its rank modulo W) above the index's 27 bits.
template <int W, Rank RANK = kNoRank>
__device__ __forceinline__ uint32_t cull_half_wide(int gl, const WideRanges<W, RANK>& rg, int cz, V3<float> xi, float h, float reach2,
                                                   const uint4* __restrict__ posh, uint32_t* q, uint32_t qcap)
{
    const HalfTest ht = half_test(xi, cz, h, reach2);
    const int g0 = (int)(threadIdx.x & 31) & ~(W - 1);
    // the first round of every column's words, all in flight together
    uint4 w0[9];
#pragma unroll
    for (int c = 0; c < 9; ++c) {
        const uint32_t bb = __shfl_sync(0xffffffffu, rg.b[c / W], c % W, W), ee = __shfl_sync(0xffffffffu, rg.e[c / W], c % W, W);
        const uint32_t word = (bb >> 1) + gl;
        w0[c] = make_uint4(0u, 0u, 0u, 0u);
        if (2 * word < ee) w0[c] = __ldg(posh + word);
    }
    uint32_t nq = 0;
#pragma unroll
    for (int c = 0; c < 9; ++c) {
        const int dx = c / 3 - 1, dy = c % 3 - 1;
        const uint32_t bb = __shfl_sync(0xffffffffu, rg.b[c / W], c % W, W), ee = __shfl_sync(0xffffffffu, rg.e[c / W], c % W, W);
        uint32_t s1 = 0u, s2 = 0u;
        if constexpr (RANK) s1 = __shfl_sync(0xffffffffu, rg.m0[c / W], c % W, W);
        if constexpr (RANK == kCellRank) s2 = __shfl_sync(0xffffffffu, rg.m1[c / W], c % W, W);
        const __half2 sx = __float2half2_rn(ht.x - (float)dx * ht.h), sy = __float2half2_rn(ht.y - (float)dy * ht.h);
        uint32_t word = (bb >> 1) + gl;
        uint4 w = w0[c];
        // rounds of W words; the warp runs the longest of its groups' columns
        while (__any_sync(0xffffffffu, 2 * (word - gl) < ee)) {
            const __half2 ddx = __hsub2(sx, as_half2(w.x)), ddy = __hsub2(sy, as_half2(w.y));
            const __half2 dz = __habs2(__hsub2(ht.zq, as_half2(w.z)));
            const __half2 ddz = __hmin2(dz, __hsub2(ht.h3, dz));
            const __half2 r2 = __hfma2(ddz, ddz, __hfma2(ddy, ddy, __hmul2(ddx, ddx)));
            const unsigned m = __hle2_mask(r2, ht.thr);
            const uint32_t j = 2 * word;
            const bool a0 = (m & 1u) && j >= bb && j < ee;
            const bool a1 = (m & 0x10000u) && j + 1 < ee;
            const uint32_t b0 = (__ballot_sync(0xffffffffu, a0) >> g0) & ((1u << W) - 1u);
            const uint32_t b1 = (__ballot_sync(0xffffffffu, a1) >> g0) & ((1u << W) - 1u);
            const uint32_t below = (1u << gl) - 1u;
            uint32_t at = nq + __popc(b0 & below) + __popc(b1 & below);
            uint32_t t0 = j, t1 = j + 1;
            if constexpr (RANK == kColumnRank) {
                t0 |= ((j - s1) & (W - 1)) << kCandIdxBits;
                t1 |= ((j + 1 - s1) & (W - 1)) << kCandIdxBits;
            }
            if constexpr (RANK == kCellRank) {
                t0 |= ((j - (j < s1 ? bb : (j < s2 ? s1 : s2))) & (W - 1)) << kCandIdxBits;
                t1 |= ((j + 1 - (j + 1 < s1 ? bb : (j + 1 < s2 ? s1 : s2))) & (W - 1)) << kCandIdxBits;
            }
            if (a0) {
                if (at < qcap) q[at] = t0;
                ++at;
            }
            if (a1 && at < qcap) q[at] = t1;
            nq += __popc(b0) + __popc(b1);
            word += W;
            if (2 * word < ee) w = __ldg(posh + word);
        }
    }
    return nq;
}

template <typename R, int W, bool DIV0>
__global__ void __launch_bounds__(kWideBlock, 5) k_build_lists_wide(Fluid<R> f, const P4<R>* __restrict__ bpos, GridView g,
                                                                 const uint32_t* __restrict__ cs, const uint32_t* __restrict__ bs,
                                                                 Consts<R> c, int akinci, Lists<R> L, DevScalars* sc,
                                                                 LoopLimits lim, double* partials, cudaGraphConditionalHandle cond)
{
    grid_wait();
    static_assert(W == 8 || W == 4, "a lane per sum, or two sums a lane");
    constexpr bool FAST = sizeof(R) == 4;
    constexpr uint32_t GROUPS = kWideBlock / W;
    __shared__ uint32_t queue[GROUPS][kQueue], bqueue[GROUPS][kQueue];
    // per entry: W, m grad W, |m grad W|^2 and the divergence term (fluid), or W, grad W and the weight (boundary)
    // of kWideChunk entries at a time (five blocks per SM at W = 4)
    __shared__ R val[GROUPS][kWideChunk][6];
    const int gl = (int)(threadIdx.x % W), grp = (int)(threadIdx.x / W);
    const int lane = threadIdx.x & 31, g0 = lane & ~(W - 1);
    const uint32_t i = (blockIdx.x * kWideBlock + threadIdx.x) / W;
    const uint32_t n = f.n;
    const bool valid = i < f.count();
    uint32_t* q = queue[grp];
    R(*v)[6] = val[grp];
    const uint32_t qcap = L.kmax < kQueue ? L.kmax : kQueue;
    V3<R> xi = {0, 0, 0}, vi = {0, 0, 0};
    uint32_t pc = 0;
    V3<float> xr = {0, 0, 0};
    bool half = false;
    const float hf = (float)c.h;
    if (valid) {
        xi = xyz(f.pos[i]);
        pc = f.cell[i];
        if constexpr (DIV0) vi = xyz(f.vel[i]);
        half = L.posh && half_cull_ok(g, pc, xi, c.h, &xr);
    }
    const bool bhalf = half && akinci && L.bposh;
    const WideRanges<W> rf = wide_ranges<W>(half, gl, g, cs, pc, xr, hf, (float)c.cull2),
                        rb = wide_ranges<W>(bhalf, gl, g, bs, pc, xr, hf, (float)c.cull2);
    uint32_t nq = cull_half_wide<W>(gl, rf, cell_z(pc), xr, hf, (float)c.cull2, L.posh, q, qcap);
    uint32_t nb = __any_sync(0xffffffffu, bhalf)
                      ? cull_half_wide<W>(gl, rb, cell_z(pc), xr, hf, (float)c.cull2, L.bposh, bqueue[grp], qcap) : 0u;
    if (valid && !half) {
        // near the grid box's border: one lane culls in R
        if (gl == 0)
            walk<R, 1, true, true>(g, cs, pc, xi, c.h, 0, [&](uint32_t j, V3<R> s) {
                const V3<R> r = s - xyz(ldg4(f.pos + j));
                if (dot3(r, r) <= c.cull2) {
                    if (nq < qcap) q[nq] = j;
                    ++nq;
                }
            });
    }
    nq = __shfl_sync(0xffffffffu, nq, 0, W);
    __syncwarp();
    const bool over = nq > qcap;
    // the sums in list order: sum s by lane s (W = 8), or s and s + 4 (W = 4)
    R acc[8 / W];
#pragma unroll
    for (int t = 0; t < 8 / W; ++t) acc[t] = 0;
    uint32_t cnt = 0;
    const uint32_t ne = over ? 0u : nq;
    for (uint32_t k0 = 0; __any_sync(0xffffffffu, k0 < ne); k0 += kWideChunk) {
        const uint32_t m = k0 < ne ? (ne - k0 < kWideChunk ? ne - k0 : kWideChunk) : 0u;  // this chunk's entries
        // evaluation, 2 W entries a round (both loads in flight); records in list order
        for (uint32_t k = 0; __any_sync(0xffffffffu, k < m); k += 2 * W) {
            uint32_t j[2], cj[2];
            P4<R> pj[2];
            V3<R> vj[2];
            bool in[2];
#pragma unroll
            for (int t = 0; t < 2; ++t) {
                const uint32_t e = k + t * W + gl;
                in[t] = e < m;
                if (in[t]) {
                    j[t] = q[k0 + e];
                    pj[t] = ldg4(f.pos + j[t]);
                    cj[t] = sizeof(R) == 4 ? __ldg(f.cell + j[t]) : 0u;
                    // (a plain load: other threads write its w here)
                    if constexpr (DIV0) vj[t] = xyz(f.vel[j[t]]);
                }
            }
#pragma unroll
            for (int t = 0; t < 2; ++t) {
                bool listed = false;
                V3<R> mg = {0, 0, 0};
                R r2 = 0;
                if (in[t]) {
                    const V3<R> r = pair_vec(xi, pc, pj[t], cj[t], c.h);
                    r2 = dot3(r, r);
                    R w;
                    V3<R> gw;
                    cubic_W_gradW<FAST>(c, r, r2, &w, &gw);
                    mg = c.mass * gw;
                    const R mg2 = dot3_div(mg, mg);
                    listed = mg2 > (R)0;
                    R sq = mg2;
                    if constexpr (sizeof(R) == 8) {
                        const R m1 = sqrt(mg2);
                        sq = m1 * m1;
                    }
                    R* o = v[k + t * W + gl];
                    o[0] = w;
                    // an unlisted pair adds zeros (it would be left out: the same sums)
                    o[1] = listed ? mg.x : (R)0; o[2] = listed ? mg.y : (R)0; o[3] = listed ? mg.z : (R)0;
                    o[4] = listed ? sq : (R)0;
                    if constexpr (DIV0) o[5] = listed ? dot3_div(vi - vj[t], mg) : (R)0;
                }
                const uint32_t b = (__ballot_sync(0xffffffffu, listed) >> g0) & ((1u << W) - 1u);
                if (listed) {
                    const uint32_t at = cnt + __popc(b & ((1u << gl) - 1u));
                    if (at < L.kmax) store_record(L.pairs + (size_t)at * n + i, mg, j[t]);
                }
                cnt += __popc(b);
            }
        }
        __syncwarp();
#pragma unroll 4
        for (uint32_t k = 0; k < m; ++k) {
#pragma unroll
            for (int t = 0; t < 8 / W; ++t) {
                const int s = gl + t * W;
                if (s < (DIV0 ? 6 : 5)) {
                    const R x = v[k][s];
                    acc[t] = s == 0 ? mul_add(c.mass, x, acc[t]) : acc[t] + x;
                }
            }
        }
        __syncwarp();
    }
    if (over && gl == 0) {
        const BuildSums<R> b = build_walk_all<R, FAST>(i, f, g, cs, c, L, xi, pc);
        v[0][0] = b.density; v[0][1] = b.sumGrad.x; v[0][2] = b.sumGrad.y; v[0][3] = b.sumGrad.z; v[0][4] = b.sumSq;
        cnt = b.cnt;
    }
    __syncwarp();
    cnt = __shfl_sync(0xffffffffu, cnt, 0, W);
    if (over) {
#pragma unroll
        for (int t = 0; t < 8 / W; ++t) acc[t] = gl + t * W < 5 ? v[0][gl + t * W] : (R)0;
    }
    __syncwarp();
    // boundary: W, grad W and weight per entry, then density and gradient sums
    R bacc = 0;  // lanes 1..3: the boundary gradient's components
    const bool bwalk = valid && akinci && (!bhalf || nb > qcap);
    if (bwalk) nb = 0;
    for (uint32_t k0 = 0; __any_sync(0xffffffffu, k0 < nb); k0 += kWideChunk) {
        const uint32_t m = k0 < nb ? (nb - k0 < kWideChunk ? nb - k0 : kWideChunk) : 0u;
        for (uint32_t e = gl; e < m; e += W) {
            const uint32_t j = bqueue[grp][k0 + e];
            const P4<R> pb = ldg4(bpos + j);
            const V3<R> r = pair_vec(xi, pc, pb, sizeof(R) == 4 ? __ldg(L.bcell + j) : 0u, c.h);
            const R r2 = dot3(r, r);
            R w;
            V3<R> gw;
            cubic_W_gradW<FAST>(c, r, r2, &w, &gw);
            const bool in = r2 <= c.cull2;
            v[e][0] = in ? w : (R)0;
            v[e][1] = in ? gw.x : (R)0; v[e][2] = in ? gw.y : (R)0; v[e][3] = in ? gw.z : (R)0;
            v[e][4] = pb.w;
        }
        __syncwarp();
        if (gl == 0)
            for (uint32_t k = 0; k < m; ++k) acc[0] = mul_add(v[k][4], v[k][0], acc[0]);
        else if (gl < 4)
            for (uint32_t k = 0; k < m; ++k) bacc = mul_add(v[k][4], v[k][gl], bacc);
        __syncwarp();
    }
    if (bwalk && gl == 0) {
        V3<R> bg = {0, 0, 0};
        R density = acc[0];
        walk<R, 1, true, true>(g, bs, pc, xi, c.h, 0, [&](uint32_t j, V3<R> s) {
            const P4<R> pb = ldg4(bpos + j);
            const V3<R> r = s - xyz(pb);
            const R r2 = dot3(r, r);
            if (!(r2 <= c.cull2)) return;
            R w;
            V3<R> gw;
            cubic_W_gradW<FAST>(c, r, r2, &w, &gw);
            density = mul_add(pb.w, w, density);
            bg = V3<R>{mul_add(pb.w, gw.x, bg.x), mul_add(pb.w, gw.y, bg.y), mul_add(pb.w, gw.z, bg.z)};
        });
        acc[0] = density;
        v[0][1] = bg.x; v[0][2] = bg.y; v[0][3] = bg.z;
    }
    __syncwarp();
    if (bwalk && gl > 0 && gl < 4) bacc = v[0][gl];
    // everything to the group's first lane
    const R density = acc[0];
    const R sg = acc[0] + bacc;  // lanes 1..3: sum of the gradients
    const V3<R> sumGrad = {__shfl_sync(0xffffffffu, sg, 1, W), __shfl_sync(0xffffffffu, sg, 2, W), __shfl_sync(0xffffffffu, sg, 3, W)};
    const V3<R> bg = {__shfl_sync(0xffffffffu, bacc, 1, W), __shfl_sync(0xffffffffu, bacc, 2, W), __shfl_sync(0xffffffffu, bacc, 3, W)};
    const R sumSq = __shfl_sync(0xffffffffu, acc[W == 8 ? 0 : 4 / W % (8 / W)], W == 8 ? 4 : 0, W);
    R dv = __shfl_sync(0xffffffffu, acc[W == 8 ? 0 : 4 / W % (8 / W)], W == 8 ? 5 : 1, W);
    double err = 0.0;
    if (valid && gl == 0) {
        f.rho[i] = density;
        f.vel[i].w = density;
        R den;
        if constexpr (sizeof(R) == 8) {
            const R m = sqrt(dot3(sumGrad, sumGrad));
            den = m * m + sumSq;
        } else {
            den = dot3_zyx(sumGrad, sumGrad) + sumSq;  // (build_lists_one's rounding)
        }
        f.alpha[i] = (fabs(den) > c.eps) ? density / den : (R)0;
        L.count[i] = cnt;
        L.bgrad[i] = P4<R>{bg.x, bg.y, bg.z, 0};
        if constexpr (DIV0) {
            uint32_t nn = cnt;
            if (cnt > L.kmax) {
                const DivSum<R> d = velocity_div_cells(f, bpos, g, cs, bs, c, akinci, i, vi);
                dv = d.dv;
                nn = d.nn;
            } else {
                if (over) dv = reread_div<R>(f, L, i, vi, cnt);
                if (akinci) dv += dot3_div(vi, bg);
            }
            err = divergence_error(i, f, L, c, (R)sc->dt, dv, nn);
        }
    }
    if constexpr (DIV0) {
        __shared__ double sh[33];
        double total;
        if (finish_reduction<false>(err, partials, &sc->block_counter, sh, &total) && threadIdx.x == 0)
            divergence_control<true>(sc, lim, total, f.count(), cond);
    }
}

// ---- cell-walk fallbacks for particles whose list overflowed -------------

template <typename R, int MODE>
__device__ __noinline__ V3<R> correct_sum_cells(const Fluid<R>& f, const P4<R>* __restrict__ bpos, const GridView& g,
                                   const uint32_t* __restrict__ cs, const uint32_t* __restrict__ bs, const Consts<R>& c,
                                   int akinci, uint32_t i, R ki, const R* __restrict__ kbuf)
{
    V3<R> sum = {0, 0, 0};
    const V3<R> xi = xyz(f.pos[i]);
    const uint32_t pc = f.cell[i];
    walk<R, 1>(g, cs, pc, xi, c.h, 0, [&](uint32_t j, V3<R> s) {
        const R kSum = ki + kbuf[j];
        if (!(fabs(kSum) > c.eps)) return;
        const V3<R> r = s - xyz(ldg4(f.pos + j));
        const R r2 = dot3(r, r);
        if (r2 <= c.cull2) sum = sum + (c.mass * kSum) * cubic_gradW(c, r, r2);
    });
    const R kb = MODE == 0 ? c.bwarm * ki : ki;
    if (akinci && fabs(kb) > c.eps)
        walk<R, 1>(g, bs, pc, xi, c.h, 0, [&](uint32_t j, V3<R> s) {
            const P4<R> pb = ldg4(bpos + j);
            const V3<R> r = s - xyz(pb);
            const R r2 = dot3(r, r);
            if (r2 <= c.cull2) sum = sum + (pb.w * kb) * cubic_gradW(c, r, r2);
        });
    return sum;
}

template <typename R> struct DivSum {
    R dv;
    uint32_t nn;
};

template <typename R>
__device__ __noinline__ DivSum<R> velocity_div_cells(const Fluid<R>& f, const P4<R>* __restrict__ bpos, const GridView& g,
                                                     const uint32_t* __restrict__ cs, const uint32_t* __restrict__ bs,
                                                     const Consts<R>& c, int akinci, uint32_t i, V3<R> vi)
{
    R dv = 0;
    unsigned cnt = 0;
    const V3<R> xi = xyz(f.pos[i]);
    const uint32_t pc = f.cell[i];
    walk<R, 1>(g, cs, pc, xi, c.h, 0, [&](uint32_t j, V3<R> s) {
        const V3<R> r = s - xyz(ldg4(f.pos + j));
        const R r2 = dot3(r, r);
        if (r2 <= c.cull2) {
            const V3<R> gr = cubic_gradW(c, r, r2);
            dv += c.mass * dot3(vi - xyz(ldg4(f.vel + j)), gr);
            if (dot3(gr, gr) > (R)0) cnt++;
        }
    });
    if (akinci)
        walk<R, 1>(g, bs, pc, xi, c.h, 0, [&](uint32_t j, V3<R> s) {
            const P4<R> pb = ldg4(bpos + j);
            const V3<R> r = s - xyz(pb);
            const R r2 = dot3(r, r);
            if (r2 <= c.cull2) dv += pb.w * dot3(vi, cubic_gradW(c, r, r2));
        });
    return DivSum<R>{dv, cnt};
}

// ---- list walks ------------------------------------------------------------

// The FP32 passes stream a particle's records through a ring in shared memory
// filled by asynchronous copies: kRingBatch records are used while the next
// kRingDepth - kRingBatch are on their way, which needs no registers.  Loaded
// into registers, the records in flight and the gathers behind them take turns.
// One scene, us/step: 13,000 particles 132 -> 122, 125,000 259 -> 254,
// 1,000,000 1441 -> 1368 (corrections at 6.6 TB/s of records and fields).
// Each thread copies and reads its own column of the ring, so no block
// synchronisation is needed; a slot is refilled only after the gathers that
// depend on its record have been issued.
constexpr int kRingDepth = 8, kRingBatch = 4;
template <typename R> struct Ring {};
template <> struct Ring<float> {
    float4* slot;    // this thread's first slot; slots are `stride` apart
    uint32_t stride;
};
__device__ __forceinline__ void copy_async16(float4* dst, const P4<float>* src)
{
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src) : "memory");
}

template <typename R> __device__ __forceinline__ Ring<R> make_ring(float4* slots, uint32_t block)
{
    if constexpr (sizeof(R) == 4) return Ring<float>{slots + threadIdx.x, block};
    else return Ring<R>{};
}

// Records p[k * n], k < cnt, a batch at a time: load(j) starts the gather of a
// record's neighbour j, eval(record, loaded) uses it, in list order.
template <typename Load, typename Eval>
__device__ __forceinline__ void stream_pairs(const Ring<float>& ring, const P4<float>* __restrict__ p, size_t n, uint32_t cnt,
                                             uint32_t nj, unsigned* fault, Load&& load, Eval&& eval)
{
    constexpr int D = kRingDepth, B = kRingBatch;
    static_assert(D == 2 * B, "one batch on its way while one is used");
    auto fill = [&](uint32_t k0) {
#pragma unroll
        for (int b = 0; b < B; ++b)
            if (k0 + b < cnt) copy_async16(ring.slot + ((k0 + b) % D) * ring.stride, p + (size_t)(k0 + b) * n);
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    fill(0);
    fill(B);
#pragma unroll 1
    for (uint32_t k = 0; k < cnt; k += B) {
        asm volatile("cp.async.wait_group 1;" ::: "memory");
        float4 r[B];
        decltype(load(0u)) v[B];
        bool ok[B];
#pragma unroll
        for (int b = 0; b < B; ++b) {
            ok[b] = k + b < cnt;
            if (ok[b]) {
                r[b] = ring.slot[((k + b) % D) * ring.stride];
                const uint32_t j = __float_as_uint(r[b].w);
                ok[b] = SPH_INDEX_OK(j, nj, fault);
                if (ok[b]) v[b] = load(j);
            }
        }
        fill(k + D);
#pragma unroll
        for (int b = 0; b < B; ++b)
            if (ok[b]) eval(V3<float>{r[b].x, r[b].y, r[b].z}, v[b]);
    }
    asm volatile("cp.async.wait_all;" ::: "memory");
}

// DFSPH velocity corrections (MODE 0 warm start, 1 density, 2 divergence),
// as k_dfsph_correct but over the pair lists; kbuf holds this pass's k.
// RING: through the ring (FP32), or loaded into registers.
template <typename R, int MODE, bool RING = sizeof(R) == 4>
__device__ __forceinline__ V3<R> correct_sum_one(uint32_t i, const Fluid<R>& f, const P4<R>* __restrict__ bpos,
                                                 const GridView& g, const uint32_t* __restrict__ cs,
                                                 const uint32_t* __restrict__ bs, const Consts<R>& c, int akinci,
                                                 const Lists<R>& L, const Ring<R>& ring)
{
    const uint32_t n = f.n;
    const R* __restrict__ kb_ = L.kbuf;
    const R ki = kb_[i];
    const uint32_t cnt = L.count[i];
    V3<R> sum = {0, 0, 0};
    if (cnt <= L.kmax) {
        const P4<R>* __restrict__ p = L.pairs + i;
        if constexpr (RING) {
            stream_pairs(ring, p, n, cnt, n, L.fault, [&](uint32_t j) { return __ldg(kb_ + j); },
                         [&](V3<R> g, R kj) {
                             const R kSum = ki + kj;
                             if (fabs(kSum) > c.eps) sum = sum + kSum * g;
                         });
        } else {
#pragma unroll 8
            for (uint32_t k = 0; k < cnt; ++k) {
                const P4<R> q = ldcs4(p + (size_t)k * n);
                const uint32_t j = as_idx(q.w);
                if (!SPH_INDEX_OK(j, n, L.fault)) continue;
                const R kSum = ki + __ldg(kb_ + j);
                if (fabs(kSum) > c.eps) sum = sum + kSum * xyz(q);
            }
        }
        const R kb = MODE == 0 ? c.bwarm * ki : ki;
        if (akinci && fabs(kb) > c.eps) sum = sum + kb * xyz(L.bgrad[i]);
    } else {
        sum = correct_sum_cells<R, MODE>(f, bpos, g, cs, bs, c, akinci, i, ki, kb_);
    }
    return sum;
}

// Velocity update after a correction sum (and the k / kv accumulation).
template <typename R, int MODE>
__device__ __forceinline__ void correct_apply(uint32_t i, const Fluid<R>& f, const Consts<R>& c, R dt, V3<R> sum)
{
    if (MODE == 1) f.kappa[i] += (f.pred[i] - c.density0) * f.alpha[i];
    if (MODE == 2) f.kappav[i] += f.div[i] * f.alpha[i];
    P4<R> v = f.vel[i];
    if (MODE == 0) { v.x -= sum.x * dt; v.y -= sum.y * dt; v.z -= sum.z * dt; }
    else { v.x -= dt * sum.x; v.y -= dt * sum.y; v.z -= dt * sum.z; }
    f.vel[i] = v;
}

// DFSPH velocity corrections (MODE 0 warm start, 1 density, 2 divergence),
// as k_dfsph_correct but over the pair lists; kbuf holds this pass's k.
template <typename R, int MODE>
__global__ void __launch_bounds__(kBlock, 8) k_dfsph_correct_list(Fluid<R> f, const P4<R>* __restrict__ bpos, GridView g,
                                                                  const uint32_t* __restrict__ cs, const uint32_t* __restrict__ bs,
                                                                  Consts<R> c, int akinci, const DevScalars* __restrict__ sc,
                                                                  Lists<R> L)
{
    grid_wait();
    __shared__ float4 slots[sizeof(R) == 4 ? kRingDepth * kBlock : 1];
    if (MODE != 0 && !sc->active) return;
    const uint32_t i = gtid_back();
    if (i >= f.count()) return;
    const V3<R> sum = correct_sum_one<R, MODE>(i, f, bpos, g, cs, bs, c, akinci, L, make_ring<R>(slots, kBlock));
    correct_apply<R, MODE>(i, f, c, (R)sc->dt, sum);
}

// Sum over the list of m (v_i - v_j) . gradW_ij plus the boundary term.
template <typename R, Rounding WHERE = kOneScene>
__device__ __forceinline__ R velocity_div_list(const Fluid<R>& f, const Lists<R>& L, uint32_t i, V3<R> vi, int akinci,
                                               const Ring<R>& ring)
{
    const uint32_t n = f.n;
    const uint32_t cnt = L.count[i];
    const P4<R>* __restrict__ p = L.pairs + i;
    R d = 0;
    if constexpr (sizeof(R) == 4 && WHERE == kOneScene) {
        const P4<R>* vel = f.vel;
        stream_pairs(ring, p, n, cnt, n, L.fault, [&](uint32_t j) { return xyz(ldg4(vel + j)); },
                     [&](V3<R> g, V3<R> vj) { d += dot3_div(vi - vj, g); });
    } else {
#pragma unroll 8
        for (uint32_t k = 0; k < cnt; ++k) {
            const P4<R> q = ldcs4(p + (size_t)k * n);
            const uint32_t j = as_idx(q.w);
            if (!SPH_INDEX_OK(j, n, L.fault)) continue;
            d += dot3(vi - xyz(ldg4(f.vel + j)), xyz(q));
        }
    }
    if (akinci) d += dot3_div<WHERE>(vi, xyz(L.bgrad[i]));
    return d;
}

// m (v_i - v_j) . gradW summed over the neighbours (list or fallback walk);
// *nn receives the number of neighbours with a non-zero gradient.
template <typename R, Rounding WHERE = kOneScene>
__device__ __forceinline__ R velocity_div_one(uint32_t i, const Fluid<R>& f, const P4<R>* __restrict__ bpos,
                                              const GridView& g, const uint32_t* __restrict__ cs,
                                              const uint32_t* __restrict__ bs, const Consts<R>& c, int akinci,
                                              const Lists<R>& L, V3<R> vi, uint32_t* nn, const Ring<R>& ring)
{
    const uint32_t cnt = L.count[i];
    if (cnt <= L.kmax) {
        *nn = cnt;
        return velocity_div_list<R, WHERE>(f, L, i, vi, akinci, ring);
    }
    const DivSum<R> d = velocity_div_cells(f, bpos, g, cs, bs, c, akinci, i, vi);
    *nn = d.nn;
    return d.dv;
}

// DFSPHSolver::predictDensities over the lists (+ loop control, as
// k_dfsph_predict_density).
template <typename R, bool INITIAL>
__global__ void __launch_bounds__(kBlock, 8) k_dfsph_predict_density_list(Fluid<R> f, const P4<R>* __restrict__ bpos, GridView g,
                                                                       const uint32_t* __restrict__ cs, const uint32_t* __restrict__ bs,
                                                                       Consts<R> c, int akinci, DevScalars* sc, LoopLimits lim,
                                                                       double* partials, cudaGraphConditionalHandle cond,
                                                                       Lists<R> L)
{
    grid_wait();
    __shared__ float4 slots[sizeof(R) == 4 ? kRingDepth * kBlock : 1];
    __shared__ double sh[33];
    if (!INITIAL && !sc->active) return;
    const uint32_t i = gtid();
    double err = 0.0;
    if (i < f.count()) {
        const V3<R> vi = xyz(f.vel[i]);
        uint32_t nn;
        const R dc = velocity_div_one(i, f, bpos, g, cs, bs, c, akinci, L, vi, &nn, make_ring<R>(slots, kBlock));
        const R dt = (R)sc->dt;
        const R rho = f.rho[i];
        R pred = rho + dc * dt;
        pred = pred < c.density0 ? c.density0 : pred;
        f.pred[i] = pred;
        L.kbuf[i] = (pred - c.density0) * f.alpha[i] / ((dt * dt) * rho);
        err = rel_error(c, (double)pred - (double)c.density0);
    }
    double total;
    if (finish_reduction<false>(err, partials, &sc->block_counter, sh, &total) && threadIdx.x == 0) {
        const double avg = f.count() ? total / (double)f.count() : 0.0;
        if (!isfinite(avg)) sc->status |= ST_NONFINITE;
        if (INITIAL) {
            sc->iterations = 0;
            sc->avgDensError = avg;
            sc->active = (lim.minIt > 0u) && (lim.maxIt > 0u);
            if (!sc->active) sc->avgDensError = 0.0;
        } else {
            const unsigned it = ++sc->iterations;
            sc->avgDensError = avg;
            const unsigned act = ((avg > lim.maxError) || (it < lim.minIt)) && (it < lim.maxIt);
            sc->active = act;
            if (!act) {
                sc->sumIterations += it;
                if (it >= lim.maxIt && avg > lim.maxError) sc->status |= ST_ITER_CAP;
            }
        }
        if (cond) cudaGraphSetConditional(cond, sc->active);
    }
}

// DFSPHSolver::computeDivergenceError over the lists (+ loop control); the
// step's first one (INITIAL) is formed by the list build unless lists are short.
template <typename R, bool INITIAL>
__global__ void __launch_bounds__(kBlock, 8) k_dfsph_divergence_list(Fluid<R> f, const P4<R>* __restrict__ bpos, GridView g,
                                                                  const uint32_t* __restrict__ cs, const uint32_t* __restrict__ bs,
                                                                  Consts<R> c, int akinci, DevScalars* sc, LoopLimits lim,
                                                                  double* partials, cudaGraphConditionalHandle cond,
                                                                  Lists<R> L)
{
    grid_wait();
    __shared__ float4 slots[sizeof(R) == 4 ? kRingDepth * kBlock : 1];
    __shared__ double sh[33];
    if (!INITIAL && !sc->active) return;
    const uint32_t i = gtid();
    double err = 0.0;
    if (i < f.count()) {
        const V3<R> vi = xyz(f.vel[i]);
        uint32_t nn;
        const R dv = velocity_div_one(i, f, bpos, g, cs, bs, c, akinci, L, vi, &nn, make_ring<R>(slots, kBlock));
        err = divergence_error(i, f, L, c, (R)sc->dt, dv, nn);
    }
    double total;
    if (finish_reduction<false>(err, partials, &sc->block_counter, sh, &total) && threadIdx.x == 0)
        divergence_control<INITIAL>(sc, lim, total, f.count(), cond);
}

// The stored lists of the n particles at [base, base + n) of a layout whose
// list slots are `stride` apart (a pooled scene's segment, or a whole scene
// with base 0), keyed by original index: cnt[me] = the particle's neighbour
// count (above kmax when its list overflowed and was not stored) and, with
// off given, the stored neighbours' original indices in list order at
// nbr[off[me]...].
template <typename R>
__global__ void k_pair_lists(uint32_t n, uint32_t base, uint32_t stride, const uint32_t* __restrict__ id, Lists<R> L,
                             const int* __restrict__ off, int* __restrict__ cnt, int* __restrict__ nbr)
{
    grid_wait();
    const uint32_t t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= n) return;
    const uint32_t i = base + t;
    const uint32_t me = id[i];
    const uint32_t c = L.count[i];
    if (cnt) cnt[me] = (int)c;
    if (off && c <= L.kmax) {
        int* o = nbr + off[me];
        for (uint32_t k = 0; k < c; ++k) o[k] = (int)id[as_idx(L.pairs[(size_t)k * stride + i].w)];
    }
}

// Host side of a pair-list dump (one-scene context and pool alike):
// counts, CSR offsets by original index, and the neighbours.  `launch(off,
// cnt, nbr)` enqueues k_pair_lists on `st`; n = particles.
template <typename Launch>
cudaError_t dump_pair_lists(uint32_t n, uint32_t kmax, cudaStream_t st, Launch&& launch, int* count, int* off, int* nbr,
                            long long* total)
{
    int* dc = nullptr;
    int* doff = nullptr;
    int* dn = nullptr;
    std::vector<int> hc(n), ho(n + 1);
    long long a = 0;
    cudaError_t e = cudaMalloc((void**)&dc, sizeof(int) * (n ? n : 1));
    if (e == cudaSuccess && n) {
        launch((const int*)nullptr, dc, (int*)nullptr);
        e = cudaGetLastError();
    }
    if (e == cudaSuccess && n) e = cudaMemcpyAsync(hc.data(), dc, sizeof(int) * n, cudaMemcpyDeviceToHost, st);
    if (e == cudaSuccess) e = cudaStreamSynchronize(st);
    if (e == cudaSuccess) {
        for (uint32_t i = 0; i < n; ++i) {
            ho[i] = (int)a;
            a += (uint32_t)hc[i] <= kmax ? hc[i] : 0;
        }
        ho[n] = (int)a;
        if (total) *total = a;
        if (count && n) std::memcpy(count, hc.data(), sizeof(int) * n);
        if (off) std::memcpy(off, ho.data(), sizeof(int) * (n + 1));
    }
    if (e == cudaSuccess && nbr && a) {
        e = cudaMalloc((void**)&doff, sizeof(int) * (n + 1));
        if (e == cudaSuccess) e = cudaMalloc((void**)&dn, sizeof(int) * (size_t)a);
        if (e == cudaSuccess) e = cudaMemcpyAsync(doff, ho.data(), sizeof(int) * (n + 1), cudaMemcpyHostToDevice, st);
        if (e == cudaSuccess) {
            launch((const int*)doff, (int*)nullptr, dn);
            e = cudaGetLastError();
        }
        if (e == cudaSuccess) e = cudaMemcpyAsync(nbr, dn, sizeof(int) * (size_t)a, cudaMemcpyDeviceToHost, st);
        if (e == cudaSuccess) e = cudaStreamSynchronize(st);
    }
    cudaStreamSynchronize(st);
    cudaFree(dc);
    cudaFree(doff);
    cudaFree(dn);
    return e;
}

// Warm-start scaling (as k_dfsph_predict_v_warm) writing k to the list
// pass's kbuf.
template <typename R>
__global__ void k_dfsph_predict_v_warm_list(Fluid<R> f, Consts<R> c, const DevScalars* __restrict__ sc, R* __restrict__ kbuf)
{
    grid_wait();
    const uint32_t i = gtid();
    if (i >= f.count()) return;
    const R dt = (R)sc->dt;
    P4<R> v = f.vel[i];
    const P4<R> a = f.acc[i];
    v.x = v.x + (a.x + c.gx) * dt; v.y = v.y + (a.y + c.gy) * dt; v.z = v.z + (a.z + c.gz) * dt;
    f.vel[i] = v;
    f.acc[i] = P4<R>{0, 0, 0, 0};
    const R dens = f.rho[i];
    const R ts2 = dt * dt;
    const R t = -f.kappa[i] / dens;
    const R mx = t < (R)-0.000000001 ? (R)-0.000000001 : t;
    kbuf[i] = -mx / ts2;
    f.kappa[i] = 0;
}

}  // namespace sph
