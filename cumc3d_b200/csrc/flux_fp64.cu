// flux_fp64.cu -- FP64 instantiations of the face-flux kernels (plain form,
// and the FP64 form with the learned flag).  Built with --fmad=false: each expression keeps the reference's
// rounding sequence, so results match the Fortran semantics bit for bit.
#include "flux_kernel.cuh"

namespace cumc {
void launch_flux_fp64(const Dev &d, int dir, int rec, int rs, dim3 grid, dim3 block, size_t smem, cudaStream_t s) {
    launch_flux_t<double>(d, dir, rec, rs, grid, block, smem, s);
}

// the faces the sweeps of a stage left on the list, with the plain HLLD; the
// list is emptied by the next kernel of the stage (k_edge)
__global__ void __launch_bounds__(128) k_faces_deferred(const Dev d) {
    pdl_wait();
    if (d.S->done) return;
    const unsigned all = *d.fix_n, n = all < d.fix_cap ? all : d.fix_cap;
    if (blockIdx.x == 0 && threadIdx.x == 0 && all > d.fix_n[1]) d.fix_n[1] = all;  // cumc_deferred_faces
    for (unsigned i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        double q[17], f[9];
#pragma unroll
        for (int v = 1; v <= 16; ++v) q[v] = d.fix[(size_t)(v - 1) * d.fix_cap + i];
        const unsigned a = d.fix_at[i];
        const int ci = (int)(a / 3u), dir = (int)(a - 3u * (unsigned)ci);
        if (dir == 0) {
            hlld_out_of_line<0>(q, d.gamma, f);
            store_face<double, 0>(d, ci, f);
        } else if (dir == 1) {
            hlld_out_of_line<1>(q, d.gamma, f);
            store_face<double, 1>(d, ci, f);
        } else {
            hlld_out_of_line<2>(q, d.gamma, f);
            store_face<double, 2>(d, ci, f);
        }
    }
}
void launch_faces_deferred(const Dev &d, cudaStream_t s) {
    const unsigned most = 4u * (unsigned)d.num_sms, want = (d.fix_cap + 127u) / 128u;
    launch(k_faces_deferred, want < most ? want : most, 128, 0, s, d.pdl, d);
}
void launch_split_fp64(const Dev &d, int dir, int rec, int rs, cudaStream_t s, const TmaMaps *tma) {
    launch_split_t<double>(d, dir, rec, rs, s, tma);
}

// FP64 WENO with the learned flag: the network (FP32 unit) sets the flags on
// refresh stages, the staged FP64 reconstruction uses them on every stage
template <int DIR>
static void launch_learned64_dir(const Dev &d, int rs, int stage, cudaStream_t s) {
    launch_learned_flags(d, DIR, stage, s);
    const dim3 tb(32, 8, 1);
    if (d.recon_tile == 2) {
        const dim3 g = recon_tile_grid(d, DIR, 2);
        if (d.wuni[DIR]) launch(k_recon_tile<double, DIR, REC_WENO, 1, 2, 2, 2>, g, tb, 0, s, d.pdl, d, stage);
        else launch(k_recon_tile<double, DIR, REC_WENO, 0, 2, 2, 2>, g, tb, 0, s, d.pdl, d, stage);
    } else {
        const dim3 g = recon_tile_grid(d, DIR, 1);
        if (d.wuni[DIR]) launch(k_recon_tile<double, DIR, REC_WENO, 1, 1, 2, 3>, g, tb, 0, s, d.pdl, d, stage);
        else launch(k_recon_tile<double, DIR, REC_WENO, 0, 1, 2, 3>, g, tb, 0, s, d.pdl, d, stage);
    }
    dim3 g, b;
    split_dims(d, DIR, false, g, b);
    switch (d.riemann_minb) {
        case 4: launch_riemann_m<double, DIR, 4>(d, rs, g, b, s); break;
        case 5: launch_riemann_m<double, DIR, 5>(d, rs, g, b, s); break;
        case 6: launch_riemann_m<double, DIR, 6>(d, rs, g, b, s); break;
        case 14: launch_riemann_pf<double, DIR, 4>(d, rs, s); break;
        case 15: launch_riemann_pf<double, DIR, 5>(d, rs, s); break;
        case 16: launch_riemann_pf<double, DIR, 6>(d, rs, s); break;
        default: launch_riemann_m<double, DIR, 1>(d, rs, g, b, s); break;
    }
}
void launch_split_learned_fp64(const Dev &d, int dir, int rs, int stage, cudaStream_t s) {
    if (dir == 0) launch_learned64_dir<0>(d, rs, stage, s);
    else if (dir == 1) launch_learned64_dir<1>(d, rs, stage, s);
    else launch_learned64_dir<2>(d, rs, stage, s);
}
}  // namespace cumc
