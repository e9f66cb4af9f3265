// tube_kernel.cuh -- one 1D problem per cluster, one cell per thread, the whole
// time loop in shared memory.
//
// batch_kernel.cuh keeps a problem's rows in global memory: every phase of a
// stage waits for L2 round trips, three cluster barriers a stage, and a thread
// works through two or more cells one after the other (13.9 us a stage for 800
// cells on 8 CTAs).  Here a CTA holds up to 254 cells in shared memory, a cell
// belongs to one thread for the whole run, and a stage has one cluster barrier:
// each CTA reconstructs one cell and solves one face beyond its share instead of
// asking its neighbours, and the cells its neighbours need are pushed into
// their shared memory when they are updated (double-buffered, so nobody reads
// what is being written).  dt: the stage-3 recovery takes the CFL limit of its
// cell, each CTA pushes its minimum with that last barrier.
//
// The reduced 1D state, the expressions and their order are those of
// batch_problem (batch_kernel.cuh), so the bits are the same.  U is not kept: at
// the start of a stage it is what FROMRVETOU makes of the recovered primitives.
#pragma once
#include "batch_kernel.cuh"

namespace cumc {

constexpr int TUBE_MAX_CTAS = 16;
// CTAs of NT threads hold NT - 2 cells (one more is reconstructed on each side);
// a row of one quantity has their 3 + 3 ghosts and two spare
constexpr int tube_row(int nt) { return nt + 8; }

// rows of shared memory, in doubles
enum : int {
    TS_RHO = 0, TS_VX, TS_VY, TS_VZ, TS_P, TS_BX, TS_BY, TS_BZ, TS_FX,  // exchanged: P, cell B, x face; two buffers
    TS_N,
    TS_X = 2 * TS_N,        // left edges of the cells, 7
    TS_Y = TS_X + 7,        // right edges, then the face fluxes and edge EMFs, 7
    TS_O = TS_Y + 7,        // u_old: 5, x face, y face, z face
    TS_E = TS_O + 8, TS_U4, TS_BY1, TS_BZ1, TS_BY0, TS_BZ0, TS_DX,
    TS_ROWS
};
constexpr int tube_smem(int nt) { return TS_ROWS * tube_row(nt) * 8; }

// problems first .. first + gridDim.x / clusterDim.x - 1 of b.order, one each.
// NT = 256: 128 registers, two CTAs an SM (the most cells in flight); 128: twice
// the registers, no spills, and half the warps in each other's way.
template <class T, int REC, int RS, int NT>
__global__ void __launch_bounds__(NT, 2) k_tube(const BatchDev b, int first) {
    constexpr int TUBE_THREADS = NT, TUBE_ROW = tube_row(NT);
    extern __shared__ __align__(16) double sm[];
    __shared__ double part_dt[2][TUBE_MAX_CTAS];
    __shared__ int part_bad[2][TUBE_MAX_CTAS];
    __shared__ double warp_dt[TUBE_THREADS / 32];
    __shared__ int any_bad;
    cg::cluster_group cluster = cg::this_cluster();
    const int size = (int)cluster.num_blocks(), rank = (int)cluster.block_rank();
    const int pid = b.order[first + (int)blockIdx.x / size];
    const long long off = b.prob[pid].off + 2;
    const int n = b.prob[pid].n;
    const double t_end = b.prob[pid].t_end;
    // this CTA's cells lo .. hi-1 (balanced), its thread's cell c; row position q
    const int lo = 1 + (int)((long long)n * rank / size), hi = 1 + (int)((long long)n * (rank + 1) / size);
    const int m = hi - lo, i = threadIdx.x, c = lo - 1 + i, q = i + 2;
    const bool mine = i >= 1 && i <= m;
    const long long g = off + c;
    const double g1 = b.gamma - 1.0;
    auto row = [&](int r) { return sm + r * TUBE_ROW; };
    // exchanged rows of buffer p
    auto S = [&](int p, int v) { return sm + (p * TS_N + v) * TUBE_ROW; };
    auto gbar = [&]() {
        if (size > 1) cluster.sync();
        else __syncthreads();
    };
    // store this cell's exchanged values into buffer p, here, as the ghosts of
    // an end of the problem, and into the neighbour that reads them
    auto publish = [&](int p, const double *v) {
#pragma unroll
        for (int r = 0; r < TS_N; ++r) S(p, r)[q] = v[r];
        if (c == 1) {
            for (int h = 0; h < 3; ++h)
                for (int r = 0; r < TS_FX; ++r) S(p, r)[h] = v[r];
        }
        if (c == n) {
            for (int h = 1; h <= 3; ++h)
                for (int r = 0; r < TS_FX; ++r) S(p, r)[q + h] = v[r];
        }
        if (size > 1 && i <= 3 && rank > 0) {  // right ghosts of the CTA below: its row starts at its lo - 3
            const int below = 1 + (int)((long long)n * (rank - 1) / size);
            for (int r = 0; r < TS_N; ++r) *cluster.map_shared_rank(&S(p, r)[c - (below - 3)], rank - 1) = v[r];
        }
        if (size > 1 && i > m - 3 && rank < size - 1) {  // left ghosts of the CTA above
            for (int r = 0; r < TS_N; ++r) *cluster.map_shared_rank(&S(p, r)[c - (hi - 3)], rank + 1) = v[r];
        }
    };
    // FROMRVETOU + FINDPRESSURE on the values of the cell: fills v, returns c_s
    auto fromrvetou = [&](double bxf, double bxm, double by1, double by0, double bz1, double bz0, double rho, double vx,
                          double vy, double vz, double e, double *v) {
        const double bx = 0.5 * (bxf + bxm);
        const double by = 0.5 * (by1 + by0);
        const double bz = 0.5 * (bz1 + bz0);
        const double vsquare = sum_sq<T>(vx, vy, vz);
        const double bsquare = sum_sq<T>(bx, by, bz);
        row(TS_U4)[i] = energy(rho, e, vsquare, bsquare);
        const double p = rho * e * g1;
        v[TS_RHO] = rho;
        v[TS_VX] = vx;
        v[TS_VY] = vy;
        v[TS_VZ] = vz;
        v[TS_P] = p;
        v[TS_BX] = bx;
        v[TS_BY] = by;
        v[TS_BZ] = bz;
        v[TS_FX] = bxf;
        if (!(rho > 0.0) || !isfinite(e) || !isfinite(p) || !isfinite(vx) || !isfinite(vy) || !isfinite(vz)) any_bad = 1;
        return sqrt(e * g1 + rho * g1 * p / (rho * rho));
    };
    // FINDDT of the cell (rungekutta.f90:221-332), 1D Cartesian
    auto limit = [&](const double *v, double cs) {
        const double rho = v[TS_RHO];
        const double a2 = cs * cs;
        const double a4 = a2 * a2;
        const double bx = v[TS_BX], by = v[TS_BY], bz = v[TS_BZ];
        const double b2x = dv(bx * bx, rho), b2y = dv(by * by, rho), b2z = dv(bz * bz, rho);
        const double b2 = b2x + b2y + b2z;
        const double b4 = b2 * b2;
        const double cfx = sqrt(0.5 * (a2 + b2 + sqrt((a4 + 2.0 * a2 * b2 + b4) - 4.0 * a2 * b2x)));
        const double cfy = sqrt(0.5 * (a2 + b2 + sqrt((a4 + 2.0 * a2 * b2 + b4) - 4.0 * a2 * b2y)));
        const double cfz = sqrt(0.5 * (a2 + b2 + sqrt((a4 + 2.0 * a2 * b2 + b4) - 4.0 * a2 * b2z)));
        const double lambda = dmax3(fabs(v[TS_VX]) + cfx, fabs(v[TS_VY]) + cfy, fabs(v[TS_VZ]) + cfz);
        double tt = row(TS_DX)[i];
        tt = tt * b.cfl / lambda;
        return tt;
    };
    // this CTA's smallest limit (and whether a state is bad) to every CTA; the
    // caller's barrier makes it visible
    auto publish_dt = [&](int slot, double dtl) {
        unsigned long long bits = (unsigned long long)__double_as_longlong(dtl);
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            const unsigned long long x = __shfl_xor_sync(0xffffffffu, bits, o);
            bits = x < bits ? x : bits;
        }
        if ((i & 31) == 0) warp_dt[i >> 5] = __longlong_as_double((long long)bits);
        __syncthreads();
        if (i < size) {
            double d = warp_dt[0];
            for (int w = 1; w < TUBE_THREADS / 32; ++w) d = warp_dt[w] < d ? warp_dt[w] : d;
            *cluster.map_shared_rank(&part_dt[slot][rank], i) = d;
            *cluster.map_shared_rank(&part_bad[slot][rank], i) = any_bad;
        }
    };

    if (i == 0) any_bad = 0;
    // every CTA of the cluster is running before its shared memory is written
    gbar();

    // -------- INITIAL_UPDATE (initial.f90:86-116) --------
    const double bx0 = b.BX[off];  // face 0: never recovered
    double dtl = 1.0e5;
    if (c == 0) {
        S(0, TS_FX)[q] = bx0;
        S(1, TS_FX)[q] = bx0;
    }
    if (mine) {
        double e = b.EPS[g], v[TS_N];
        batch_floor(b, e);
        row(TS_E)[i] = e;
        row(TS_BY1)[i] = b.BY1[g];
        row(TS_BZ1)[i] = b.BZ1[g];
        row(TS_BY0)[i] = b.BY0[g];
        row(TS_BZ0)[i] = b.BZ0[g];
        row(TS_DX)[i] = b.dx[g];
        const double cs = fromrvetou(b.BX[g], b.BX[g - 1], b.BY1[g], b.BY0[g], b.BZ1[g], b.BZ0[g], b.P[0][g], b.P[1][g],
                                     b.P[2][g], b.P[3][g], e, v);
        publish(0, v);
        const double tt = limit(v, cs);
        if (tt < dtl) dtl = tt;
    }
    publish_dt(0, dtl);
    gbar();

    const T *wts = (sizeof(T) == 8) ? reinterpret_cast<const T *>(b.w) : reinterpret_cast<const T *>(b.wf);
    const double rk20 = 3.0 / 4.0, rk21 = 1.0 / 4.0, rk22 = 1.0 / 4.0;
    const double rk30 = 1.0 / 3.0, rk31 = 2.0 / 3.0, rk32 = 2.0 / 3.0;
    double t = 0.0;
    int steps = 0, slot = 0, p = 0;
    bool bad = false;
    while (true) {
        double dt = part_dt[slot][0];
        bad = part_bad[slot][0] != 0;
        for (int r = 1; r < size; ++r) {
            dt = part_dt[slot][r] < dt ? part_dt[slot][r] : dt;
            bad = bad || part_bad[slot][r] != 0;
        }
        if (bad || !(t < t_end) || steps >= b.max_steps) break;
        slot ^= 1;
        if (!(dt < 1.0e5)) dt = 1.0e5;
        if (t + dt > t_end) dt = t_end - t;
        for (int stage = 1; stage <= 3; ++stage) {
            // ---- A: reconstruction of the cells lo-1 .. hi ----
            if (i <= m + 1) {
                const T *wp = wts + (size_t)g * 14;
                T w[14];
                constexpr int NW = (REC == REC_PPM) ? 14 : (REC == REC_WENO) ? 10 : 2;
#pragma unroll
                for (int k = 0; k < NW; ++k) w[k] = __ldg(wp + k);
                // rho, vx, vy, vz, p, By, Bz
                auto at = [&](int v, int k) -> T { return (T)S(p, v < 5 ? v : v + 1)[q + k]; };
                auto put = [&](int v, T vm, T vp) {
                    reinterpret_cast<T *>(row(TS_X + v))[i] = vm;
                    *reinterpret_cast<T *>(&row(TS_Y + v)[i]) = vp;
                };
                recon_all<T, REC, 0>(w, false, b.pos_fallback, nullptr, at, at, put);
            }
            __syncthreads();
            // ---- B: Riemann solve on the faces lo-1 .. hi-1, the edge EMFs there ----
            double F[5], ey = 0.0, ez = 0.0;
            if (i <= m) {
                T pl[9], pr[9], fo[9];
                constexpr int slot_of[7] = {irho, ivx, ivy, ivz, itau, iby, ibz};
#pragma unroll
                for (int v = 0; v < 7; ++v) {
                    pl[slot_of[v]] = *reinterpret_cast<const T *>(&row(TS_Y + v)[i]);
                    pr[slot_of[v]] = reinterpret_cast<const T *>(row(TS_X + v))[i + 1];
                }
                const T bn = (T)S(p, TS_FX)[q];
                pl[ibx] = bn;
                pr[ibx] = bn;
                face_flux<T, 0, RS>(pl, pr, (T)b.gamma, fo);
#pragma unroll
                for (int v = 0; v < 5; ++v) F[v] = (double)fo[1 + v];
                const double fyx = (double)fo[ibz];   // eface(iyx) = flux(ibz)
                const double fzx = -(double)fo[iby];  // eface(izx) = -flux(iby)
                const double ey_a = S(p, TS_VX)[q] * S(p, TS_BZ)[q] - S(p, TS_VZ)[q] * S(p, TS_BX)[q];
                const double ez_a = S(p, TS_VY)[q] * S(p, TS_BX)[q] - S(p, TS_VX)[q] * S(p, TS_BY)[q];
                const double ey_b = S(p, TS_VX)[q + 1] * S(p, TS_BZ)[q + 1] - S(p, TS_VZ)[q + 1] * S(p, TS_BX)[q + 1];
                const double ez_b = S(p, TS_VY)[q + 1] * S(p, TS_BX)[q + 1] - S(p, TS_VX)[q + 1] * S(p, TS_BY)[q + 1];
                ey = 0.50 * (fyx + fyx + ey_a + ey_b) - 0.25 * (ey_a + ey_a + ey_b + ey_b);
                ez = 0.50 * (fzx + fzx + ez_a + ez_b) - 0.25 * (ez_a + ez_a + ez_b + ez_b);
#pragma unroll
                for (int v = 0; v < 5; ++v) row(TS_Y + v)[i] = F[v];
                row(TS_Y + 5)[i] = ey;
                row(TS_Y + 6)[i] = ez;
                if (stage == 1) row(TS_O + 5)[i] = S(p, TS_FX)[q];
            }
            __syncthreads();
            // ---- C: du/dt + the Shu-Osher combination, FROMUTORVE + floor,
            // FROMRVETOU + FINDPRESSURE of the thread's cell ----
            dtl = 1.0e5;
            if (mine) {
                const Den64 rdx = den64(row(TS_DX)[i]);
                // the quotient by dx, through the plain division where over() asks for it
                auto by_dx = [&](double x) {
                    bool ok = true;
                    const double r = over(x, rdx, ok);
                    return ok ? r : x / rdx.b;
                };
                double lr[5];
#pragma unroll
                for (int v = 0; v < 5; ++v) {
                    const double dflux = by_dx(F[v] - row(TS_Y + v)[i - 1]);
                    lr[v] = -dflux;
                    lr[v] = lr[v] + 0.0;  // + sc (no sources)
                }
                const double zero = 0.0;
                const double lbx = -((zero) / 1.0 - (zero) / 1.0);
                const double lby = -((zero) / 1.0 - by_dx(ez - row(TS_Y + 6)[i - 1]));
                const double lbz = -(by_dx(ey - row(TS_Y + 5)[i - 1]) - (zero) / 1.0);
                auto combo = [&](double u, double o, double lrv) {
                    if (stage == 1) return __dadd_rn(u, __dmul_rn(dt, lrv));
                    if (stage == 2)
                        return __dadd_rn(__dadd_rn(__dmul_rn(rk20, o), __dmul_rn(rk21, u)), __dmul_rn(__dmul_rn(rk22, dt), lrv));
                    return __dadd_rn(__dadd_rn(__dmul_rn(rk30, o), __dmul_rn(rk31, u)), __dmul_rn(__dmul_rn(rk32, dt), lrv));
                };
                const double r0 = S(p, TS_RHO)[q];
                // U 0..4, the x, y and z faces
                const double uu[8] = {r0,
                                      __dmul_rn(S(p, TS_VX)[q], r0),
                                      __dmul_rn(S(p, TS_VY)[q], r0),
                                      __dmul_rn(S(p, TS_VZ)[q], r0),
                                      row(TS_U4)[i],
                                      S(p, TS_FX)[q],
                                      row(TS_BY1)[i],
                                      row(TS_BZ1)[i]};
                const double lv[8] = {lr[0], lr[1], lr[2], lr[3], lr[4], lbx, lby, lbz};
                double un[8];
#pragma unroll
                for (int v = 0; v < 8; ++v) {
                    double o = uu[v];
                    if (stage == 1) {
                        if (v != 5) row(TS_O + v)[i] = o;  // the x face: above, its left neighbour's too
                    } else {
                        o = row(TS_O + v)[i];
                    }
                    un[v] = combo(uu[v], o, lv[v]);
                }
                // the updated x face below (face 0 starts every stage from bx0)
                const double um = S(p, TS_FX)[q - 1], om = stage == 1 ? um : row(TS_O + 5)[i - 1];
                const double ubxm = combo(um, om, lbx);
                const double by0 = row(TS_BY0)[i], bz0 = row(TS_BZ0)[i];
                const double uby0 = combo(by0, by0, lby), ubz0 = combo(bz0, bz0, lbz);
                const double ubx = un[5], uby1 = un[6], ubz1 = un[7];
                const double u0 = un[0], u1 = un[1], u2 = un[2], u3 = un[3], u4 = un[4];
                const double bxu = 0.5 * (ubx + ubxm);
                const double byu = 0.5 * (uby1 + uby0);
                const double bzu = 0.5 * (ubz1 + ubz0);
                const double bsquare = sum_sq<T>(bxu, byu, bzu);
                const double ne = u4 - 0.5 * bsquare;
                const Den64 ru = den64(u0);
                bool ok = true;
                double vx = over(u1, ru, ok), vy = over(u2, ru, ok), vz = over(u3, ru, ok), qe = over(ne, ru, ok);
                if (!ok) {
                    vx = u1 / u0;
                    vy = u2 / u0;
                    vz = u3 / u0;
                    qe = ne / u0;
                }
                const double vsquare = sum_sq<T>(vx, vy, vz);
                double e = qe - 0.5 * vsquare;
                batch_floor(b, e);
                if (stage == 3) batch_floor(b, e);
                row(TS_E)[i] = e;
                row(TS_BY1)[i] = uby1;
                row(TS_BZ1)[i] = ubz1;
                double v[TS_N];
                const double cs = fromrvetou(ubx, c == 1 ? bx0 : ubxm, uby1, by0, ubz1, bz0, u0, vx, vy, vz, e, v);
                publish(p ^ 1, v);
                if (stage == 3) {
                    const double tt = limit(v, cs);
                    if (tt < dtl) dtl = tt;
                }
            }
            if (stage == 3) publish_dt(slot, dtl);
            p ^= 1;
            gbar();
        }
        t = t + dt;
        steps += 1;
    }
    // the state, and BOUNDARY once (outflow x; boundary.f90:439-505) so that it
    // carries its ghosts
    if (mine) {
        auto store = [&](long long at, bool ghost) {
#pragma unroll
            for (int v = 0; v < 5; ++v) b.P[v][at] = S(p, v)[q];
            b.EPS[at] = row(TS_E)[i];
            b.BY1[at] = row(TS_BY1)[i];
            b.BZ1[at] = row(TS_BZ1)[i];
            if (!ghost) b.BX[at] = S(p, TS_FX)[q];
        };
        store(g, false);
        if (c == 1)
            for (int h = 0; h < 3; ++h) store(off - h, true);
        if (c == n)
            for (int h = 1; h <= 3; ++h) store(off + n + h, true);
    }
    if (rank == 0 && i == 0) {
        b.prob[pid].t = t;
        b.prob[pid].steps = steps;
        b.prob[pid].status = bad ? CUMC_ESTATE : 0;
    }
    gbar();  // no CTA leaves while another may still write to it
}

template <class T, int REC, int RS, int NT>
static cudaError_t launch_tube_one(const BatchDev &b, int first, int count, int size, cudaStream_t s) {
    cudaError_t e = cudaFuncSetAttribute(k_tube<T, REC, RS, NT>, cudaFuncAttributeMaxDynamicSharedMemorySize, tube_smem(NT));
    if (e == cudaSuccess && size > 8)
        e = cudaFuncSetAttribute(k_tube<T, REC, RS, NT>, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
    if (e != cudaSuccess) return e;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(count * size);
    cfg.blockDim = dim3(NT);
    cfg.dynamicSmemBytes = tube_smem(NT);
    cfg.stream = s;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = size;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, k_tube<T, REC, RS, NT>, b, first);
}

template <class T>
static cudaError_t launch_tube_t(const BatchDev &b, int rec, int rs, int first, int count, int size, int wide, cudaStream_t s) {
#define CUMC_TUBE_RS(R)                                                                    \
    switch (rs) {                                                                          \
        case RS_LF: return wide ? launch_tube_one<T, R, RS_LF, 256>(b, first, count, size, s) : launch_tube_one<T, R, RS_LF, 128>(b, first, count, size, s); \
        case RS_HLL: return wide ? launch_tube_one<T, R, RS_HLL, 256>(b, first, count, size, s) : launch_tube_one<T, R, RS_HLL, 128>(b, first, count, size, s); \
        case RS_HLLC: return wide ? launch_tube_one<T, R, RS_HLLC, 256>(b, first, count, size, s) : launch_tube_one<T, R, RS_HLLC, 128>(b, first, count, size, s); \
        default: return wide ? launch_tube_one<T, R, RS_HLLD, 256>(b, first, count, size, s) : launch_tube_one<T, R, RS_HLLD, 128>(b, first, count, size, s); \
    }
    switch (rec) {
        case REC_TVD_MM: CUMC_TUBE_RS(REC_TVD_MM);
        case REC_TVD_VL: CUMC_TUBE_RS(REC_TVD_VL);
        case REC_TVD_MC: CUMC_TUBE_RS(REC_TVD_MC);
        case REC_PPM: CUMC_TUBE_RS(REC_PPM);
        default: CUMC_TUBE_RS(REC_WENO);
    }
#undef CUMC_TUBE_RS
}

}  // namespace cumc
