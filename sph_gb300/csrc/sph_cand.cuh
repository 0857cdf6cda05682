// The density passes that build the PCISPH / WCSPH candidate lists (CandLists,
// sph_kernels.cuh), and WCSPH's force pass over them.
//
// Like the DFSPH list build, candidates are culled from the half-precision
// positions into a queue in shared memory and evaluated from it: a walk that
// evaluates as it goes runs the kernel's arithmetic with one lane in five
// active and waits for each candidate's load in turn (90k particles: 78 us,
// 45 us here), and in FP64 fills the two FP64 lanes of an SM with distance
// tests.
#pragma once

#include "sph_divide.h"
#include "sph_lists.cuh"

namespace sph {

template <typename R> struct CandSums {
    R density;
    uint32_t m;
};

// A particle the half-precision cull does not serve, or whose queue
// overflowed: the walk, out of line.  Boundary points (BND) carry their weight.
template <typename R, bool BND>
__device__ __noinline__ CandSums<R> cand_walk(uint32_t i, uint32_t n, const P4<R>* __restrict__ pos, const GridView& g,
                                              const uint32_t* __restrict__ starts, const Consts<R>& c, uint32_t pc, V3<R> xi,
                                              R reach2, uint32_t* idx, uint32_t kmax, uint32_t first, R density)
{
    uint32_t m = 0;
    walk_reach<R>(g, starts, pc, xi, c.h, reach2, [&](uint32_t j, V3<R> s, uint32_t code) {
        const P4<R> p = ldg4(pos + j);
        const V3<R> r = s - xyz(p);
        const R r2 = dot3(r, r);
        if (r2 <= reach2) {
            if (first + m < kmax) idx[(size_t)(first + m) * n + i] = j | (code << kCandIdxBits);
            ++m;
        }
        if (r2 <= c.cull2) density += (BND ? p.w : c.mass) * cubic_W(c, sqrt(r2));
    });
    return CandSums<R>{density, m};
}

// WCSPH's equation of state (WCSPHSolver::computeFluidPressures
// WCSPHSolver.cpp:80-95) and p / rho^2 for the pressure-force pass.
template <typename R> __device__ __forceinline__ void cand_eos(uint32_t i, const Fluid<R>& f, const Consts<R>& c, V3<R> xi, R density)
{
    const R p = fmax((R)0, c.k_eos * (pow(density / c.density0, c.gamma) - (R)1));
    f.press[i] = p;
    f.xk[i] = P4<R>{xi.x, xi.y, xi.z, p / (density * density)};
}

// Densities (SPHSolver::computeFluidDensities SPHSolver.cpp:44-91, as
// k_density<R, 1, false, EOS>, EOS: with WCSPH's equation of state) fused
// with the candidate lists' build, one lane per particle: the terms and their
// order are the cell walk's.
template <typename R, bool EOS>
__global__ void __launch_bounds__(kBlock, 7) k_density_cand(Fluid<R> f, const P4<R>* __restrict__ bpos, GridView g,
                                                            const uint32_t* __restrict__ cs, const uint32_t* __restrict__ bs,
                                                            Consts<R> c, int akinci, R reach2, CandOut o)
{
    grid_wait();
    __shared__ uint32_t q[kQueue * kBlock];
    constexpr int EB = kListBatch<R>;
    const uint32_t i = gtid();
    if (i >= f.count()) return;
    const uint32_t n = f.n;
    const V3<R> xi = xyz(f.pos[i]);
    const uint32_t pc = f.cell[i];
    V3<float> xr;
    const bool half = half_cull_ok(g, pc, xi, c.h, &xr);
    R density = 0;
    uint32_t m = 0;
    uint32_t nq = kQueue + 1u;
    if (half) nq = cull_half(g, cs, pc, xr, (float)c.h, (float)reach2, o.posh, q, kBlock, kQueue);
    if (nq <= kQueue) {
        for (uint32_t k = 0; k < nq; k += EB) {
            uint32_t j[EB], cj[EB];
            P4<R> pj[EB];
#pragma unroll
            for (int b = 0; b < EB; ++b) {
                j[b] = q[(k + b < nq ? k + b : nq - 1) * kBlock + threadIdx.x];
                pj[b] = ldg4(f.pos + j[b]);
                cj[b] = __ldg(f.cell + j[b]);
            }
#pragma unroll
            for (int b = 0; b < EB; ++b) {
                if (k + b >= nq) break;
                const V3<R> r = pair_vec(xi, pc, pj[b], cj[b], c.h);
                const R r2 = dot3(r, r);
                if (r2 <= reach2) {
                    if (m < o.kmax) o.idx[(size_t)m * n + i] = j[b] | (cell_code(pc, cj[b]) << kCandIdxBits);
                    ++m;
                }
                if (r2 <= c.cull2) density += c.mass * cubic_W(c, sqrt(r2));
            }
        }
    } else {
        const CandSums<R> w = cand_walk<R, false>(i, n, f.pos, g, cs, c, pc, xi, reach2, o.idx, o.kmax, 0u, density);
        density = w.density;
        m = w.m;
    }
    uint32_t mb = 0;
    if (akinci) {
        uint32_t nb = kQueue + 1u;
        if (half) nb = cull_half(g, bs, pc, xr, (float)c.h, (float)reach2, o.bposh, q, kBlock, kQueue);
        if (nb <= kQueue) {
            for (uint32_t k = 0; k < nb; k += EB) {
                uint32_t j[EB], cj[EB];
                P4<R> pj[EB];
#pragma unroll
                for (int b = 0; b < EB; ++b) {
                    j[b] = q[(k + b < nb ? k + b : nb - 1) * kBlock + threadIdx.x];
                    pj[b] = ldg4(bpos + j[b]);
                    cj[b] = __ldg(o.bcell + j[b]);
                }
#pragma unroll
                for (int b = 0; b < EB; ++b) {
                    if (k + b >= nb) break;
                    const V3<R> r = pair_vec(xi, pc, pj[b], cj[b], c.h);
                    const R r2 = dot3(r, r);
                    if (r2 <= reach2) {
                        if (m + mb < o.kmax) o.idx[(size_t)(m + mb) * n + i] = j[b] | (cell_code(pc, cj[b]) << kCandIdxBits);
                        ++mb;
                    }
                    if (r2 <= c.cull2) density += pj[b].w * cubic_W(c, sqrt(r2));
                }
            }
        } else {
            const CandSums<R> w = cand_walk<R, true>(i, n, bpos, g, bs, c, pc, xi, reach2, o.idx, o.kmax, m, density);
            density = w.density;
            mb = w.m;
        }
    }
    f.rho[i] = density;
    f.vel[i].w = density;
    o.cnt[i] = m;
    o.bcnt[i] = mb;
    if (EOS) cand_eos(i, f, c, xi, density);
}

// The same with W lanes per particle (small scenes), each lane with a list and
// a partial density of its own.  The lanes share the cull into a common queue.
// EVEN: the listed candidates are dealt to the lanes in turn (a particle's
// lists are then all stored or all walked).  Otherwise each takes the
// candidates of its part of the cell walk (CandLists), so that the solvers'
// sums stay the walk's bit for bit: DFSPH's and PCISPH's solves amplify
// rounding (a change of 1e-7 in the velocities grows to 1e-5 in five steps);
// WCSPH's, and PCISPH's in FP64, do not need it, and the lanes' shares are
// uneven (8,000 WCSPH particles: 36 against 41 us/step, FP64 189 against 279).
// DENS = false: the lists alone (DFSPH's non-pressure forces).
template <typename R, int W, bool EOS, bool EVEN, bool DENS = true>
__global__ void __launch_bounds__(kWideBlock) k_density_cand_wide(Fluid<R> f, const P4<R>* __restrict__ bpos, GridView g,
                                                                  const uint32_t* __restrict__ cs, const uint32_t* __restrict__ bs,
                                                                  Consts<R> c, int akinci, R reach2, CandOut o)
{
    grid_wait();
    constexpr uint32_t GROUPS = kWideBlock / W;
    constexpr uint32_t OWN = kQueue / (W / 2);  // a lane's candidates: twice its even share of the queue
    constexpr int EB = kListBatch<R>;
    __shared__ uint32_t queue[GROUPS][kQueue];
    __shared__ uint32_t own[EVEN ? 1 : OWN][kWideBlock];
    const int gl = (int)(threadIdx.x % W), grp = (int)(threadIdx.x / W);
    const uint32_t i = (blockIdx.x * kWideBlock + threadIdx.x) / W;
    const uint32_t n = f.n;
    const bool valid = i < f.count();
    V3<R> xi = {0, 0, 0};
    uint32_t pc = 0;
    V3<float> xr = {0, 0, 0};
    bool half = false;
    if (valid) {
        xi = xyz(f.pos[i]);
        pc = f.cell[i];
        half = half_cull_ok(g, pc, xi, c.h, &xr);
    }
    const float hf = (float)c.h, rf2 = (float)reach2;
    uint32_t* q = queue[grp];
    constexpr Rank RANK = EVEN ? kNoRank : (sizeof(R) == 4 ? kCellRank : kColumnRank);
    const WideRanges<W, RANK> rf = wide_ranges<W, RANK>(half, gl, g, cs, pc, xr, hf, rf2),
                              rb = wide_ranges<W, RANK>(half && akinci, gl, g, bs, pc, xr, hf, rf2);
    R density = 0;
    // this lane's part of the candidates of one kind; `first` slots are taken
    // (EVEN: the particle's candidates, `first` listed so far)
    auto visit = [&](const WideRanges<W, RANK>& rg, const uint4* posh, const P4<R>* pos, const uint32_t* cell,
                     const uint32_t* __restrict__ starts, bool bnd, uint32_t first) -> uint32_t {
        __syncwarp();  // the queue's last reader
        const uint32_t nq = cull_half_wide<W, RANK>(gl, rg, cell_z(pc), xr, hf, rf2, posh, q, kQueue);
        __syncwarp();
        if constexpr (EVEN) {
            const bool queued = half && nq <= kQueue;
            uint32_t listed = 0;
            for (uint32_t k = 0; __any_sync(0xffffffffu, queued && k < nq); k += W) {
                bool near = false;
                uint32_t entry = 0;
                if (queued && k + gl < nq) {
                    const uint32_t j = q[k + gl];
                    const P4<R> pj = ldg4(pos + j);
                    const uint32_t cj = __ldg(cell + j);
                    const V3<R> r = pair_vec(xi, pc, pj, cj, c.h);
                    const R r2 = dot3(r, r);
                    near = r2 <= reach2;
                    entry = j | (cell_code(pc, cj) << kCandIdxBits);
                    if (r2 <= c.cull2) density += (bnd ? pj.w : c.mass) * cubic_W(c, sqrt(r2));
                }
                const uint32_t b = (__ballot_sync(0xffffffffu, near) >> ((threadIdx.x & 31) & ~(W - 1))) & ((1u << W) - 1u);
                const uint32_t at = first + listed + __popc(b & ((1u << gl) - 1u));
                if (near && at / W < o.kmax) o.idx[((size_t)(at / W) * n + i) * W + at % W] = entry;
                listed += __popc(b);
            }
            if (queued) return listed;
            if (valid)
                walk<R, W, false>(g, starts, pc, xi, c.h, gl, [&](uint32_t j, V3<R> s) {
                    const P4<R> pj = ldg4(pos + j);
                    const V3<R> r = s - xyz(pj);
                    const R r2 = dot3(r, r);
                    if (r2 <= c.cull2) density += (bnd ? pj.w : c.mass) * cubic_W(c, sqrt(r2));
                });
            return W * o.kmax + 1u;  // not stored
        }
        uint32_t listed = 0, mine = 0;
        auto eval = [&](uint32_t j, uint32_t cj, const P4<R>& pj) {
            const V3<R> r = pair_vec(xi, pc, pj, cj, c.h);
            const R r2 = dot3(r, r);
            if (r2 <= reach2) {
                if (first + listed < o.kmax) o.idx[((size_t)(first + listed) * n + i) * W + gl] = j | (cell_code(pc, cj) << kCandIdxBits);
                ++listed;
            }
            if (DENS && r2 <= c.cull2) density += (bnd ? pj.w : c.mass) * cubic_W(c, sqrt(r2));
        };
        if (half && nq <= kQueue) {
#pragma unroll 4
            for (uint32_t e = 0; e < nq; ++e) {
                const uint32_t x = q[e];
                if ((x >> kCandIdxBits) == (uint32_t)gl) {
                    if (mine < OWN) own[mine][threadIdx.x] = x & kCandIdxMask;
                    ++mine;
                }
            }
        }
        if (half && nq <= kQueue && mine <= OWN) {
            for (uint32_t k = 0; k < mine; k += EB) {
                uint32_t j[EB], cj[EB];
                P4<R> pj[EB];
#pragma unroll
                for (int b = 0; b < EB; ++b) {
                    j[b] = own[k + b < mine ? k + b : mine - 1][threadIdx.x];
                    pj[b] = ldg4(pos + j[b]);
                    cj[b] = __ldg(cell + j[b]);
                }
#pragma unroll
                for (int b = 0; b < EB; ++b) {
                    if (k + b >= mine) break;
                    eval(j[b], cj[b], pj[b]);
                }
            }
        } else if (valid) {
            walk<R, W, false>(g, starts, pc, xi, c.h, gl, [&](uint32_t j, V3<R>) { eval(j, __ldg(cell + j), ldg4(pos + j)); });
        }
        return listed;
    };
    uint32_t m = visit(rf, o.posh, f.pos, f.cell, cs, false, 0u);
    uint32_t mb = 0;
    if (akinci) mb = visit(rb, o.bposh, bpos, o.bcell, bs, true, m);
    __syncwarp();
    if constexpr (EVEN) {
        // the particle's counts to this lane's; a particle's lists fit together
        const uint32_t all = m + mb, fits = W * o.kmax, dealt = W - 1u - (uint32_t)gl;
        const uint32_t own_m = m > fits ? o.kmax + 1u : (m + dealt) / W;
        mb = m > fits || all > fits ? o.kmax + 1u : (all + dealt) / W - own_m;
        m = own_m;
    }
    if (valid) {
        o.cnt[(size_t)i * W + gl] = m;
        o.bcnt[(size_t)i * W + gl] = mb;
    }
    if (!DENS) return;
    density = group_sum<W>(density);
    if (!valid || gl != 0) return;
    f.rho[i] = density;
    f.vel[i].w = density;
    if (EOS) cand_eos(i, f, c, xi, density);
}

// u / dt by components, as the divisions round; the rare quotients that
// `quotient` leaves to the division take it out of line.
static __device__ __noinline__ V3<double> divide3(V3<double> u, double b) { return V3<double>{u.x / b, u.y / b, u.z / b}; }
__device__ __forceinline__ V3<double> div3(V3<double> u, const Divisor& d)
{
    V3<double> q;
    const bool x = quotient(u.x, d, &q.x), y = quotient(u.y, d, &q.y), z = quotient(u.z, d, &q.z);
    return x && y && z ? q : divide3(u, d.b);
}
__device__ __forceinline__ V3<float> div3(V3<float> u, float b) { return u / b; }
__device__ __forceinline__ Divisor divisor_of(double b) { return divisor(b); }
__device__ __forceinline__ float divisor_of(float b) { return b; }

// WCSPH with XSPH viscosity (or none of the force plugins' other kinds):
// pressure force (k_wcsph_pressure_force) and viscosity (k_npforce) from one
// visit of the candidates, each sum in its own order; the distance and its
// root are formed once.  us/step: 8,000 particles in FP64 202 -> 148, 90,000
// with Akinci walls 103 -> 91.
template <typename R> struct WcsphFluid { V3<R> p, av; };
template <typename R> struct WcsphBoundary { V3<R> p, avb; };

template <typename R, int G>
__global__ void __launch_bounds__(kBlock) k_wcsph_forces(Fluid<R> f, const P4<R>* __restrict__ bpos, GridView g,
                                                         const uint32_t* __restrict__ cs, const uint32_t* __restrict__ bs,
                                                         Consts<R> c, int akinci, const DevScalars* __restrict__ sc, CandLists L)
{
    grid_wait();
    __shared__ float4 shift[kShiftCodes];
    if (sizeof(R) == 4) fill_shift_table(shift, (float)c.h);
    const uint32_t t = gtid();
    const uint32_t i = t / G;
    const int lane = (int)(t % G);
    const bool valid = i < f.count();
    WcsphFluid<R> sf = {{0, 0, 0}, {0, 0, 0}};
    WcsphBoundary<R> sb = {{0, 0, 0}, {0, 0, 0}};
    if (valid) {
        const P4<R> pi = f.xk[i];
        const V3<R> xi = xyz(pi);
        const R dpi = pi.w;
        const P4<R> vi4 = f.vel[i];
        const V3<R> vi = xyz(vi4);
        const R rho_i = vi4.w;
        const auto dt = divisor_of((R)sc->dt);
        const uint32_t pc = f.cell[i];
        const bool bvisc = (c.force_flags & F_BVISC) != 0;
        const P4<R>*xk = f.xk, *vel = f.vel;
        fluid_visit<R, G, true, kListBatch<R>>(
            L, f.n, i, g, cs, pc, xi, c.h, lane, shift, sf,
            [=](uint32_t j) { return PosVelIdx<R>{ldg4(xk + j), ldg4(vel + j), j}; },
            [=](WcsphFluid<R>& a, const PosVelIdx<R>& q, V3<R> s) {
                const V3<R> r = s - xyz(q.x);
                const R r2 = dot3(r, r);
                if (!(r2 <= c.cull2)) return;
                a.p = a.p - (c.mass * (dpi + q.x.w)) * cubic_gradW(c, r, r2);
                const V3<R> u = ((c.visc * (c.mass / q.v.w)) * (xyz(q.v) - vi)) * cubic_W(c, sqrt(r2));
                a.av = a.av + div3(u, dt);
            });
        sb.p = sf.p;  // one sum: the boundary's terms follow the fluid's
        if (akinci)
            boundary_visit<R, G, true, kListBatch<R>>(
                L, f.n, i, g, bs, pc, xi, c.h, lane, shift, sb, [=](uint32_t j) { return ldg4(bpos + j); },
                [=](WcsphBoundary<R>& a, const P4<R>& pb, V3<R> s) {
                    const V3<R> r = s - xyz(pb);
                    const R r2 = dot3(r, r);
                    if (!(r2 <= c.cull2)) return;
                    a.p = a.p - (pb.w * (dpi * (R)1)) * cubic_gradW(c, r, r2);
                    if (bvisc) {
                        const V3<R> u = ((c.bvisc * (pb.w / rho_i)) * (-vi)) * cubic_W(c, sqrt(r2));
                        a.avb = a.avb + div3(u, dt);
                    }
                });
    }
    V3<R> sum = sb.p;
    if (G > 1) {
        sum = group_sum3<G>(sum);
        sf.av = group_sum3<G>(sf.av);
        sb.avb = group_sum3<G>(sb.avb);
    }
    if (!valid || lane != 0) return;
    P4<R> a = f.acc[i];
    V3<R> tot = {a.x, a.y, a.z};
    tot = tot + sum;
    tot = tot + sf.av;
    tot = tot + sb.avb;
    f.acc[i] = P4<R>{tot.x, tot.y, tot.z, 0};
}

}  // namespace sph
