// Adjoint (reverse-mode) pass on register patches, for small and middle-sized
// tiles: the stages and cells of adjoint_kernel.cuh with the regions and
// exchanges of patch.cuh, psi and lambda a patch each.
#pragma once
#include "adjoint_kernel.cuh"
#include "patch.cuh"

namespace tsb {

template <class A, int N>
using AdjShape = PatchShape<Variant<double, 2, A::IMAG, false, 0>, N>;

template <class A, class S, bool EDGE>
__device__ __forceinline__ void adj_region(Patch<S> &ps, Patch<S> &la, const AdjArgs &a, double cin,
                                           double cnext, double m2, double &kacc) {
    constexpr int N = S::N;
    constexpr bool INV = A::MODE == 0;
    if constexpr (EDGE) {
        patch_masks(ps, a.W, a.H);
        la.hm = ps.hm;
        la.vm = ps.vm;
    }
    const PatchTile<S, EDGE, false> tp(ps, a, a.psi_in), tl(ps, a, a.lam_in);
    const PatchTable<S, EDGE> table(ps, a);
#pragma unroll
    for (int j = 0; j < N; ++j) {
        tp.row(ps, a, j, ps.c[j]);
        tl.row(ps, a, j, la.c[j]);
    }
    if constexpr (A::IMAG) {
        // psi_k = c_k phi_k; lambda = c_{k+1} (Lambda - mu c_{k+1} phi_{k+1})
        const PatchTile<S, EDGE, false> tn(ps, a, a.psn_in);
#pragma unroll
        for (int j = 0; j < N; ++j) {
            Cx<double> n[N];
            tn.row(ps, a, j, n);
#pragma unroll
            for (int i = 0; i < N; ++i) {
                ps.c[j][i] = scale_cx(ps.c[j][i], cin);
                la.c[j][i].re = __dmul_rn(cnext, __fma_rn(-m2, n[i].re, la.c[j][i].re));
                la.c[j][i].im = __dmul_rn(cnext, __fma_rn(-m2, n[i].im, la.c[j][i].im));
            }
        }
    }
    patch_vsweep<S, EDGE, 0>(ps);
    patch_vsweep<S, EDGE, 0>(la);
    patch_hsweep<S, EDGE, 0, 0>(ps);
    patch_hsweep<S, EDGE, 0, 0>(la);
    patch_vsweep<S, EDGE, 1>(ps);
    patch_vsweep<S, EDGE, 1>(la);
    patch_hsweep<S, EDGE, 1, 1>(ps);
    patch_hsweep<S, EDGE, 1, 1>(la);
    // the region without its rim
    const bool out = ps.px >= S::MX && ps.px < S::TX - S::MX && ps.py >= S::MY &&
                     ps.py < S::TX - S::MY;
#pragma unroll
    for (int j = 0; j < N; ++j) {
        typename A::TabT tv[N];
        table.row(ps, a, j, tv);
        double *grow = a.gv + (ptrdiff_t)(ps.gy + j) * a.P + ps.gx;
#pragma unroll
        for (int i = 0; i < N; ++i) {
            const bool mine = out && (!EDGE || (ps.gx + i < a.W && ps.gy + j < a.H));
            double g = 0.0, kf = 0.0, sd = 0.0;
            if (mine) g = grow[i];
            adj_cell<A>(a, ps.c[j][i], la.c[j][i], tv[i], g, kf, sd);
            if (mine) {
                grow[i] = g;
                if constexpr (A::IMAG) kacc = __fma_rn(kf, sd, kacc);
            }
        }
    }
    patch_hsweep<S, EDGE, 1, 0>(la);
    if constexpr (INV) patch_hsweep<S, EDGE, 1, 0>(ps);
    patch_vsweep<S, EDGE, 1>(la);
    if constexpr (INV) patch_vsweep<S, EDGE, 1>(ps);
    patch_hsweep<S, EDGE, 0, 1>(la);
    if constexpr (INV) patch_hsweep<S, EDGE, 0, 1>(ps);
    patch_vsweep<S, EDGE, 0>(la);
    if constexpr (INV) patch_vsweep<S, EDGE, 0>(ps);
    if (!out) return;
    Cx<double> *ol = reinterpret_cast<Cx<double> *>(a.lam_out) + (size_t)ps.gy * a.P + ps.gx;
    Cx<double> *op = reinterpret_cast<Cx<double> *>(a.psi_out) + (size_t)ps.gy * a.P + ps.gx;
#pragma unroll
    for (int j = 0; j < N; ++j) {
        if (EDGE && ps.gy + j >= a.H) break;
        if (!EDGE || ps.gx + N <= a.W) {
            patch_store_row<N>(ol + (size_t)j * a.P, la.c[j]);
            if constexpr (INV) patch_store_row<N>(op + (size_t)j * a.P, ps.c[j]);
        } else {
#pragma unroll
            for (int i = 0; i < N; ++i) {
                if (ps.gx + i >= a.W) continue;
                st_cx_global(ol + (size_t)j * a.P + i, la.c[j][i]);
                if constexpr (INV) st_cx_global(op + (size_t)j * a.P + i, ps.c[j][i]);
            }
        }
    }
}

// a.n_strips x a.n_segs regions, taken by the blocks in turn.
template <class A, int N>
__global__ void __launch_bounds__(256, kAdjPatchBlocks) adj_patch_kernel(AdjArgs a) {
    using S = AdjShape<A, N>;
    __shared__ __align__(16) unsigned char exch[4 * S::EXCH];
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    Patch<S> ps, la;
    patch_thread(ps, exch);
    patch_thread(la, exch + 2 * S::EXCH);
    // psi: inverse rotations (INVERSE) or forward ones; lambda: the transposed
    // stages (b -> -b in real time, the same in imaginary time)
    const double sp = A::MODE == 0 ? -1.0 : 1.0, sl = A::IMAG ? 1.0 : -1.0;
    ps.aH = la.aH = a.aH;
    ps.aV = la.aV = a.aV;
    ps.bH = sp * a.bH;
    ps.bV = sp * a.bV;
    la.bH = sl * a.bH;
    la.bV = sl * a.bV;
    asm volatile("griddepcontrol.wait;" ::: "memory");
    double cin = 1.0, cnext = 1.0, m2 = 0.0, kacc = 0.0;
    if constexpr (A::IMAG) {
        cin = *a.c_in;
        cnext = *a.c_next;
        m2 = *a.mu_next * cnext;
    }
    const int n = a.n_strips * a.n_segs;
    for (int t = blockIdx.x; t < n; t += gridDim.x) {
        const int X0 = (t % a.n_strips) * S::OX - S::MX * N, Y0 = (t / a.n_strips) * S::OY - S::MY * N;
        ps.gx = la.gx = X0 + ps.px * N;
        ps.gy = la.gy = Y0 + ps.py * N;
        if (X0 >= 0 && Y0 >= 0 && X0 + S::R <= a.W && Y0 + S::R <= a.H)
            adj_region<A, S, false>(ps, la, a, cin, cnext, m2, kacc);
        else
            adj_region<A, S, true>(ps, la, a, cin, cnext, m2, kacc);
    }
    if constexpr (A::IMAG)
        adj_finish(a, kacc, 8, (int)(threadIdx.x >> 5), (int)(threadIdx.x & 31));
}

}  // namespace tsb
