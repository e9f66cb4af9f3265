// poisson.cu -- red-black SOR for the self-gravity potential of the collapsar
// model on a spherical grid (layout and state: poisson.cuh).  Compiled with
// --fmad=false: every expression rounds as the Fortran does.
//
// One iteration (model/collapsar/src/custom.f90:489-616) is the red sweep and
// the black sweep, which keep the ghost copies along phi and take the
// convergence check; the first iteration of a solve reads the ghosts as given
// and ends with a pass that fills them.
// The reference copies phi to phi_old before the sweeps and takes
// max |(phi - phi_old) / phi_old| afterwards; each interior cell is updated
// exactly once per iteration, so the sweep that updates a cell has both
// values at hand and takes the maximum itself (no copy).  The maximum of
// non-negative doubles is exact and independent of order, so the iteration
// count and every bit of phi match a sequential run of the same loops.
#include <cmath>

#include "poisson.cuh"

namespace cumc {

// poisson_coef (model/collapsar/src/poisson.f90:34-64) at every interior
// cell; x, y, z point at the centres of index 0 (valid for -1..n+2).
// Natural layouts: ajp1/ajm1 by j, bkp1/bkm1 by j + (nx+2) k, the rest by
// j + (nx+2) (k + (ny+2) l).
void sor_coefficients(int nx, int ny, int nz, const double *x, const double *y, const double *z, double *ajp1,
                      double *ajm1, double *bkp1, double *bkm1, double *clp1, double *clm1, double *epsc) {
    const long long px = nx + 2, py = (long long)(nx + 2) * (ny + 2);
    for (int i = 1; i <= nx; ++i)
        for (int j = 1; j <= ny; ++j)
            for (int k = 1; k <= nz; ++k) {
                const double xm1 = x[i - 1], xc = x[i], xp1 = x[i + 1];
                const double ym1 = y[j - 1], yc = y[j], yp1 = y[j + 1];
                const double zm1 = z[k - 1], zc = z[k], zp1 = z[k + 1];
                const double ty = std::tan(yc), sy = std::sin(yc);
                const long long c = i + px * j + py * k;
                epsc[c] = 2.0 * (xp1 + xm1 - 3.0 * xc) / xc / (xp1 - xc) / (xc - xm1) +
                          (yp1 + ym1 - 2.0 * yc - 2.0 * ty) / (xc * xc) / ty / (yp1 - yc) / (yc - ym1) -
                          2.0 / (xc * xc) / (sy * sy) / (zp1 - zc) / (zc - zm1);
                ajp1[i] = 2.0 * (2.0 * xc - xm1) / (xp1 - xm1) / (xp1 - xc) / xc;
                ajm1[i] = 2.0 * (2.0 * xc - xp1) / (xp1 - xm1) / (xc - xm1) / xc;
                bkp1[i + px * j] = (2.0 * ty + yc - ym1) / (xc * xc) / ty / (yp1 - yc) / (yp1 - ym1);
                bkm1[i + px * j] = (2.0 * ty + yc - yp1) / (xc * xc) / ty / (yp1 - ym1) / (yc - ym1);
                clp1[c] = 2.0 / (xc * xc) / (sy * sy) / (zp1 - zm1) / (zp1 - zc);
                clm1[c] = 2.0 / (xc * xc) / (sy * sy) / (zp1 - zm1) / (zc - zm1);
            }
}

// 4 pi rho_in per interior cell, rho_in = rho where rho exceeds the
// atmosphere density, else 0 (custom.f90:527-529).  rho in the engine's
// padded layout (index (j+2) + NX ((k+2) + NY (l+2))).
__global__ void k_sor_source(const SorDev s, const double *__restrict__ rho, int NX, int NY, double rho_atm,
                             double fourpi) {
    const int j = blockIdx.x * blockDim.x + threadIdx.x + 1;
    const int k = blockIdx.y * blockDim.y + threadIdx.y + 1;
    const int l = blockIdx.z + 1;
    if (j > s.nx || k > s.ny) return;
    const double r = rho[(j + 2) + (long long)NX * ((k + 2) + (long long)NY * (l + 2))];
    const double diff = r - rho_atm;
    const double factor = diff > 0.0 ? 1.0 : 0.0;
    const double rho_in = factor * r;
    s.src[(j + k + l) & 1][sor_index(s, j, k, l)] = fourpi * rho_in;
}

// IF (abserror <= tolerance) EXIT and the iteration limit, on the maximum of a
// finished iteration (slot p of err: iterations alternate, so that the next
// one's maximum can grow while this is read): 0 go on, 1 converged, 2 limit
__device__ __forceinline__ int sor_exit_test(const SorDev &s, int p) {
    const double e = __longlong_as_double((long long)s.err[p]);
    return e <= *s.tol ? 1 : s.state[0] >= s.state[2] ? 2 : 0;
}

// One colour: C = 0 red ((-1)**(j+k+l) > 0), 1 black; a 32 x 8 block covers
// 32 half-row cells (h) of 16 rows (k, every 8th row per thread) of plane
// l = blockIdx.z + 1, so a thread has the loads of two cells in flight.
//
// INNER: every iteration of a solve but its first.  The ghosts are then copies
// of interior cells as they stood when the last iteration ended, so a sweep
// needs no pass that refills them: beside r = 0 and the theta ends a ghost is
// the cell's own old value; along phi the sweep keeps the copies itself.  A
// ghost phi(j,k,0) is read only by the cell (j,k,1), of the other colour.  nz
// even: it has its source's colour; the red sweep writes the old value (the
// black sweep of this iteration must see it), the black sweep the new one.  nz
// odd: it has the other colour; a sweep copies the sources of the colour it does
// not touch.  A red sweep first takes the exit test of the iteration before it,
// every CTA for itself on values nothing changes meanwhile; the black sweep
// counts the iteration.  p: the iteration's slot of err.  At 32 registers (8
// blocks an SM; 42 as the compiler chose) an iteration takes 13.6 against 15.5
// us at 156 x 44 x 128, 172 against 199 at 384 x 192 x 192; the three launches
// with a ghost pass took 17.5 and 173.
template <int C, int INNER>
__global__ void __launch_bounds__(256, 8) k_sor_sweep(const SorDev s, int p) {
    if (s.state[1]) return;
    const bool lead = (blockIdx.x | blockIdx.y | blockIdx.z | threadIdx.x | threadIdx.y) == 0;
    if (INNER && C == 0) {
        const int stop = sor_exit_test(s, p ^ 1);
        if (stop) {
            if (lead) {
                *s.err_last = __longlong_as_double((long long)s.err[p ^ 1]);
                s.state[1] = stop;
            }
            return;
        }
    }
    if (C == 1 && lead) {
        s.state[0] = s.state[0] + 1;
        s.err[p ^ 1] = (unsigned long long)__double_as_longlong(1.0e-50);  // the next iteration's start, as the reference's
    }
    const int ys = s.hx, zs = s.hx * (s.ny + 2);
    const int h = blockIdx.x * 32 + threadIdx.x, l = blockIdx.z + 1;
    const double *o = s.phi[1 - C];
    unsigned long long e = 0ull;
#pragma unroll
    for (int r = 0; r < 2; ++r) {
        const int k = (blockIdx.y * 2 + r) * 8 + threadIdx.y + 1;
        if (h >= s.hx || k > s.ny) continue;
        const int j = 2 * h + ((C + k + l) & 1);
        const int row = s.hx * (k + (s.ny + 2) * l);
        const int c = h + row;
        if (INNER && (s.nz & 1) && (l == 1 || l == s.nz)) {
            // nz odd: the other colour's cell of the pair (2h, 2h + 1)
            const int jo = j ^ 1;
            if (jo >= 1 && jo <= s.nx) {
                const double v = o[c];
                if (l == 1) s.phi[C][c + s.nz * zs] = v;
                if (l == s.nz) s.phi[C][c - s.nz * zs] = v;
            }
        }
        if (j < 1 || j > s.nx) continue;
        const double old = s.phi[C][c];
        const double pE = o[((j + 1) >> 1) + row];
        double pW = o[((j - 1) >> 1) + row], pN = o[c + ys], pS = o[c - ys];
        const double pU = o[c + zs], pD = o[c - zs];
        if (INNER) {
            if (j == 1) pW = old;
            if (k == 1) pS = old;
            if (k == s.ny) pN = old;
        }
        const int b = j + (s.nx + 2) * k;
        double sum = s.ajp1[j] * pE + s.ajm1[j] * pW;
        sum = sum + s.bkp1[b] * pN;
        sum = sum + s.bkm1[b] * pS;
        sum = sum + s.clp1[C][c] * pU;
        sum = sum + s.clm1[C][c] * pD;
        const double eps = s.epsc[C][c], num = s.src[C][c] - sum;
        // (plain divisions: with shared-seed quotients and their tests, as the flux
        // kernels use, this memory-bound sweep was 6% slower)
        const double rhs = num / eps;
        const double nw = (1.0 - s.omega) * old + s.omega * rhs;
        s.phi[C][c] = nw;
        if (INNER && !(s.nz & 1)) {
            if (l == 1) s.phi[C][c + s.nz * zs] = C ? nw : old;
            if (l == s.nz) s.phi[C][c - s.nz * zs] = C ? nw : old;
        }
        const double rel = fabs((nw - old) / old);
        // |x| of a double keeps the bit order of its magnitude (NaN above +inf)
        const unsigned long long v = (unsigned long long)__double_as_longlong(rel);
        e = v > e ? v : e;
    }
#pragma unroll
    for (int m = 16; m > 0; m >>= 1) {
        const unsigned long long v = __shfl_xor_sync(0xffffffffu, e, m);
        e = v > e ? v : e;
    }
    __shared__ unsigned long long wmax[8];
    const int tid = threadIdx.y * 32 + threadIdx.x;
    if ((tid & 31) == 0) wmax[tid >> 5] = e;
    __syncthreads();
    if (tid == 0) {
        unsigned long long m = wmax[0];
        for (int w = 1; w < 8; ++w) m = wmax[w] > m ? wmax[w] : m;
        if (m) atomicMax(s.err + p, m);
    }
}

// ghost layers (custom.f90:578-612): phi(0) = phi(1), phi(nx+1) = -1 along
// r; copies of the first and last row along theta; periodic along phi.  The
// three sets are disjoint and read interior cells only.  Run after the first
// iteration of a solve (whose sweeps read the ghosts as given) and once after
// the last (end 1), where thread 0 takes the exit test if no sweep has.
__global__ void k_sor_ghosts(const SorDev s, int end) {
    const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (end && t == 0 && s.state[1] == 0) {
        *s.err_last = __longlong_as_double((long long)s.err[s.state[0] & 1]);
        s.state[1] = sor_exit_test(s, s.state[0] & 1);
    }
    const long long nyz = (long long)s.ny * s.nz, nxz = (long long)s.nx * s.nz, nxy = (long long)s.nx * s.ny;
    auto at = [&](int j, int k, int l) -> double & { return s.phi[(j + k + l) & 1][sor_index(s, j, k, l)]; };
    if (t < nyz) {
        const int k = (int)(t % s.ny) + 1, l = (int)(t / s.ny) + 1;
        at(0, k, l) = at(1, k, l);
        at(s.nx + 1, k, l) = -1.0;
    } else if (t < nyz + nxz) {
        const long long u = t - nyz;
        const int j = (int)(u % s.nx) + 1, l = (int)(u / s.nx) + 1;
        at(j, 0, l) = at(j, 1, l);
        at(j, s.ny + 1, l) = at(j, s.ny, l);
    } else if (t < nyz + nxz + nxy) {
        const long long u = t - nyz - nxz;
        const int j = (int)(u % s.nx) + 1, k = (int)(u / s.nx) + 1;
        at(j, k, 0) = at(j, k, s.nz);
        at(j, k, s.nz + 1) = at(j, k, 1);
    }
}

// phi between the natural order (j + (nx+2) (k + (ny+2) l), cells 0..n+1) and
// the colour-split arrays
__global__ void k_sor_order(const SorDev s, double *__restrict__ nat, int split) {
    const int j = blockIdx.x * 32 + threadIdx.x, k = blockIdx.y * 8 + threadIdx.y, l = blockIdx.z;
    if (j > s.nx + 1 || k > s.ny + 1) return;
    double &p = s.phi[(j + k + l) & 1][sor_index(s, j, k, l)];
    double &n = nat[j + (long long)(s.nx + 2) * (k + (long long)(s.ny + 2) * l)];
    if (split) p = n;
    else n = p;
}
void launch_sor_order(const SorDev &s, double *nat, int split, cudaStream_t st) {
    k_sor_order<<<dim3((s.nx + 33) / 32, (s.ny + 9) / 8, s.nz + 2), dim3(32, 8), 0, st>>>(s, nat, split);
}

__global__ void k_sor_reset(const SorDev s) {
    s.state[0] = 0;
    s.state[1] = 0;
    s.err[0] = s.err[1] = (unsigned long long)__double_as_longlong(1.0e-50);
}

void launch_sor_source(const SorDev &s, const double *rho, int NX, int NY, double rho_atm, cudaStream_t st) {
    const double fourpi = 4.0 * (4.0 * std::atan(1.0));  // 4.0d0*pi, pi = 4.D0*DATAN(1.D0)
    const dim3 b(32, 8, 1), g((s.nx + 31) / 32, (s.ny + 7) / 8, s.nz);
    k_sor_source<<<g, b, 0, st>>>(s, rho, NX, NY, rho_atm, fourpi);
}

void launch_sor_ghosts(const SorDev &s, int end, cudaStream_t st) {
    const long long ng = (long long)s.ny * s.nz + (long long)s.nx * s.nz + (long long)s.nx * s.ny;
    k_sor_ghosts<<<(unsigned)((ng + 255) / 256), 256, 0, st>>>(s, end);
}

// iteration it = 1, 2, ... of a solve; a captured one may stand for any it of
// its parity but 1
void launch_sor_iteration(const SorDev &s, int it, cudaStream_t st) {
    const dim3 t(32, 8, 1), g((s.hx + 31) / 32, (s.ny + 15) / 16, s.nz);
    if (it == 1) {
        k_sor_sweep<0, 0><<<g, t, 0, st>>>(s, 1);
        k_sor_sweep<1, 0><<<g, t, 0, st>>>(s, 1);
        launch_sor_ghosts(s, 0, st);
    } else {
        k_sor_sweep<0, 1><<<g, t, 0, st>>>(s, it & 1);
        k_sor_sweep<1, 1><<<g, t, 0, st>>>(s, it & 1);
    }
}

void launch_sor_reset(const SorDev &s, cudaStream_t st) { k_sor_reset<<<1, 1, 0, st>>>(s); }

}  // namespace cumc
