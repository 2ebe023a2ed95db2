// Fused Trotter-Suzuki step on register patches, for small and middle-sized
// tiles.
//
// A block holds one region of the tile in registers: 16 x 16 threads, each a
// patch of N x N cells (N = 2 or 4; a warp: two patch columns).  The sweeps
// V0 H0 V1 H1 P H1 V1 H0 V0 (src/cpukernel.cpp:22-92) run on the whole region
// at once; every sweep spoils one more row or column at the region's rim, so
// the block writes the region without it.  Pairs inside a patch are register
// operations; vertical pairs across patches take a warp shuffle per value,
// horizontal ones shuffles between the warp's two columns and an exchange
// through shared memory between warps (two buffers in turn, one block barrier
// per horizontal sweep).  The arithmetic of a cell is that of the row walks
// (the same pair forms and potential row): in real time the bits are theirs.  Two
// things depend on how a tile is cut: the order of the norm's sum in imaginary
// time, and the warp's choice of a nonlinear phase's evaluation in imaginary time
// and in a double rotating frame, once phases pass 2^-8 (step_kernel.cuh).
//
// Against the look-ahead walk (walk2.cuh) a step is one load, nine stages of
// a region and one store instead of a chain of nine stages per row: what a
// step of a small tile costs is its latency (128^2 double: 12.2 -> 3.1 us),
// and a walk's short segments recompute more (8-row segments 2.3 cells per
// cell written, a 32 x 32 region 1.8, a 64 x 64 one 1.3).  On large tiles the
// walk's asynchronous row copies and its 4 independent warps per scheduler
// keep the FP64 pipe busier (2048^2 double: 38.6 us against 63).
//
// Regions that reach over the tile's edge (EDGE) mask the pairs across it:
// the identity, as closed boundaries skip them (src/cpucartesian.cpp:4-70);
// with StepArgs::wrap they also read the periodic halo from the cells it
// copies (src/cpukernel.cpp:706-716,738-746), which spares the refresh a
// launch of its own between two steps.
//
// Variants: those of the look-ahead walk: a rotating frame, cylinders, one
// species of a pair, potential rows.
#pragma once
#include "patch_decl.h"
#include "walk2.cuh"

namespace tsb {

// M steps of a region in one launch (patch_steps_kernel).
template <class V_, int N_, int M_ = 1>
struct PatchShape {
    using V = V_;
    using T = typename V::T;
    using TabT = typename V::TabT;
    static constexpr int N = N_;                   // patch side
    static constexpr int M = M_;
    static constexpr int TX = 16, THREADS = TX * TX;
    static constexpr int R = TX * N;               // region side
    static constexpr int WX = 2;                   // patch columns of a warp
    // rim: V::HX columns and V::HY rows per step, in whole patches
    static constexpr int MX = (M * V::HX + N - 1) / N, MY = (M * V::HY + N - 1) / N;
    static constexpr int OX = R - 2 * MX * N, OY = R - 2 * MY * N;  // written cells
    // rows that an exchange carries: half of them in a kinetic sweep, all in
    // a rotation row or radial sweep
    static constexpr int NE = (V::ROT || V::CYL) ? N : N / 2;
    static constexpr int PLANE = THREADS * (int)sizeof(Cx<T>);
    static constexpr int EXCH = NE * PLANE;        // one exchange buffer
    static constexpr int BLOCKS = M > 1 ? patch_steps_blocks(N, sizeof(T) == 4)
                                        : patch_blocks(N, sizeof(T) == 4);
    // table rows loaded before the sweep that precedes the potential
    static constexpr int TAB_AHEAD = N * N * (int)sizeof(Cx<T>) <= 128 ? N : 1;
    static_assert(OX == patch_out(N, M * V::HX) && OY == patch_out(N, M * V::HY), "patch_out");
    static_assert(OX > 0 && OY > 0, "no cell left to write");
    static_assert(EXCH >= kFinishScratch * 8, "the finish's scratch");
};

template <class S>
struct Patch {
    using T = typename S::T;
    Cx<T> c[S::N][S::N];
    T aH, bH, aV, bV, ca, caa;
    int px, py;           // this thread's patch of the region
    int gx, gy;           // its first cell in the tile
    unsigned char *exch;  // this thread's cell of the exchange planes
    int outer;            // byte offset to the neighbour warp's cell (own at the region's rim)
    unsigned hm, vm;      // EDGE: bit i + 1: the pair (i, i + 1) crosses the tile's edge
};

// This thread's place in the region; exch: the block's exchange buffers.
template <class S>
__device__ __forceinline__ void patch_thread(Patch<S> &p, unsigned char *exch) {
    using T = typename S::T;
    const int lane = threadIdx.x & 31;
    p.px = (int)(threadIdx.x >> 5) * S::WX + lane % S::WX;
    p.py = lane / S::WX;
    p.exch = exch + threadIdx.x * (int)sizeof(Cx<T>);
    // the outer edge's neighbour is the other column of the next warp
    p.outer = (p.px == 0 || p.px == S::TX - 1) ? 0
                                               : (p.px & 1 ? 31 : -31) * (int)sizeof(Cx<T>);
    p.hm = p.vm = 0u;
}

// EDGE: the pairs of this patch that cross the edge of a W x H tile.
template <class S>
__device__ __forceinline__ void patch_masks(Patch<S> &p, int W, int H) {
    const int rx = W - p.gx, ry = H - p.gy;  // cells to the tile's end
    p.hm = (p.gx == 0 ? 1u : 0u) | ((rx >= 0 && rx <= S::N) ? 1u << rx : 0u);
    p.vm = (p.gy == 0 ? 1u : 0u) | ((ry >= 0 && ry <= S::N) ? 1u << ry : 0u);
}

template <class T>
__device__ __forceinline__ T patch_one() {
    return DeltaForm<T>::value ? T(0) : T(1);
}

// The patch columns' edges, K rows from row F in steps of D, through buffer
// BUF: send before the work inside the patch, recv after it.
template <class S, int BUF, int F, int D, int K>
__device__ __forceinline__ void patch_send(Patch<S> &p, Cx<typename S::T> (&in)[K]) {
    using T = typename S::T;
    using V2 = typename Vec2T<T>::type;
    const bool odd = p.px & 1;
#pragma unroll
    for (int k = 0; k < K; ++k) {
        const Cx<T> l = p.c[F + D * k][0], r = p.c[F + D * k][S::N - 1];
        const Cx<T> outer = odd ? r : l, inner = odd ? l : r;
        *reinterpret_cast<V2 *>(p.exch + BUF * S::EXCH + k * S::PLANE) = V2{outer.re, outer.im};
        in[k].re = __shfl_xor_sync(0xffffffffu, inner.re, 1);
        in[k].im = __shfl_xor_sync(0xffffffffu, inner.im, 1);
    }
}
// l, r: the cells left and right of the patch
template <class S, int BUF, int K>
__device__ __forceinline__ void patch_recv(const Patch<S> &p, const Cx<typename S::T> (&in)[K],
                                           Cx<typename S::T> (&l)[K], Cx<typename S::T> (&r)[K]) {
    using T = typename S::T;
    __syncthreads();
    const bool odd = p.px & 1;
#pragma unroll
    for (int k = 0; k < K; ++k) {
        const Cx<T> o = ld_cx_shared(
            reinterpret_cast<const Cx<T> *>(p.exch + BUF * S::EXCH + p.outer + k * S::PLANE));
        l[k] = odd ? in[k] : o;
        r[k] = odd ? o : in[k];
    }
}

// Horizontal kinetic sweep SW; BUF: the exchange buffer it uses.
template <class S, bool EDGE, int SW, int BUF>
__device__ __forceinline__ void patch_hsweep(Patch<S> &p) {
    using T = typename S::T;
    constexpr bool IMAG = S::V::IMAG;
    constexpr int N = S::N, E0 = SW ^ 1, K = N / 2;  // rows that pair across patches
    const T one = patch_one<T>();
    Cx<T> in[K], l[K], r[K];
    patch_send<S, BUF, E0, 2, K>(p, in);
#pragma unroll
    for (int i = 0; i + 1 < N; ++i) {
        const bool cut = EDGE && ((p.hm >> (i + 1)) & 1u);
        const T a = cut ? one : p.aH, b = cut ? T(0) : p.bH;
#pragma unroll
        for (int j = (i + SW) & 1; j < N; j += 2) {
            const Cx<T> x = p.c[j][i], y = p.c[j][i + 1];
            p.c[j][i] = kin<IMAG>(x, y, a, b);
            p.c[j][i + 1] = kin<IMAG>(y, x, a, b);
        }
    }
    patch_recv<S, BUF, K>(p, in, l, r);
    const bool cl = EDGE && (p.hm & 1u), cr = EDGE && ((p.hm >> N) & 1u);
    const T al = cl ? one : p.aH, bl = cl ? T(0) : p.bH;
    const T ar = cr ? one : p.aH, br = cr ? T(0) : p.bH;
#pragma unroll
    for (int k = 0; k < K; ++k) {
        Cx<T>(&row)[N] = p.c[E0 + 2 * k];
        row[0] = kin<IMAG>(row[0], l[k], al, bl);
        row[N - 1] = kin<IMAG>(row[N - 1], r[k], ar, br);
    }
}

// Vertical kinetic sweep SW: the patches above and below are WX lanes away.
template <class S, bool EDGE, int SW>
__device__ __forceinline__ void patch_vsweep(Patch<S> &p) {
    using T = typename S::T;
    constexpr bool IMAG = S::V::IMAG;
    constexpr int N = S::N;
    const T one = patch_one<T>();
    Cx<T> u[N / 2], d[N / 2];
#pragma unroll
    for (int k = 0; k < N / 2; ++k) {
        const int i = (SW ^ 1) + 2 * k;
        u[k].re = __shfl_up_sync(0xffffffffu, p.c[N - 1][i].re, S::WX);
        u[k].im = __shfl_up_sync(0xffffffffu, p.c[N - 1][i].im, S::WX);
        d[k].re = __shfl_down_sync(0xffffffffu, p.c[0][i].re, S::WX);
        d[k].im = __shfl_down_sync(0xffffffffu, p.c[0][i].im, S::WX);
    }
#pragma unroll
    for (int j = 0; j + 1 < N; ++j) {
        const bool cut = EDGE && ((p.vm >> (j + 1)) & 1u);
        const T a = cut ? one : p.aV, b = cut ? T(0) : p.bV;
#pragma unroll
        for (int i = (j + SW) & 1; i < N; i += 2) {
            const Cx<T> x = p.c[j][i], y = p.c[j + 1][i];
            p.c[j][i] = kin<IMAG>(x, y, a, b);
            p.c[j + 1][i] = kin<IMAG>(y, x, a, b);
        }
    }
    const bool cu = EDGE && (p.vm & 1u), cd = EDGE && ((p.vm >> N) & 1u);
    const T au = cu ? one : p.aV, bu = cu ? T(0) : p.bV;
    const T ad = cd ? one : p.aV, bd = cd ? T(0) : p.bV;
#pragma unroll
    for (int k = 0; k < N / 2; ++k) {
        const int i = (SW ^ 1) + 2 * k;
        p.c[0][i] = kin<IMAG>(p.c[0][i], u[k], au, bu);
        p.c[N - 1][i] = kin<IMAG>(p.c[N - 1][i], d[k], ad, bd);
    }
}

// Cylinder: radial sweep of parity PAR, pairs (x, x + 1) with x = PAR mod 2 in
// every row; rad holds (a, b), (c, 0) per column x, the pair's cells take
// (a, b) and (a, c) (src/cpucylindrical.cpp:4-81).
template <class S, bool EDGE, int PAR, int BUF>
__device__ __forceinline__ void patch_radial(Patch<S> &p, const StepArgs<typename S::T> &a) {
    using T = typename S::T;
    constexpr bool IMAG = S::V::IMAG;
    constexpr int N = S::N;
    const Cx<T> *rad = reinterpret_cast<const Cx<T> *>(a.rad);
    auto coef = [&](int x, T &ca, T &cb, T &cc) {
        const bool ok = !EDGE || (x >= 0 && x + 1 < a.W);
        const Cx<T> ab = ok ? rad[2 * x] : Cx<T>{patch_one<T>(), T(0)};
        ca = ab.re;
        cb = ab.im;
        cc = ok ? rad[2 * x + 1].re : T(0);
    };
    Cx<T> in[N], l[N], r[N];
    if constexpr (PAR == 1) patch_send<S, BUF, 0, 1, N>(p, in);
#pragma unroll
    for (int i = PAR; i + 1 < N; i += 2) {
        T ca, cb, cc;
        coef(p.gx + i, ca, cb, cc);
#pragma unroll
        for (int j = 0; j < N; ++j) {
            const Cx<T> x = p.c[j][i], y = p.c[j][i + 1];
            p.c[j][i] = kin<IMAG>(x, y, ca, cb);
            p.c[j][i + 1] = kin<IMAG>(y, x, ca, cc);
        }
    }
    if constexpr (PAR == 1) {
        patch_recv<S, BUF, N>(p, in, l, r);
        T la, lb, lc, ra, rb, rc;
        coef(p.gx - 1, la, lb, lc);
        coef(p.gx + N - 1, ra, rb, rc);
#pragma unroll
        for (int j = 0; j < N; ++j) {
            p.c[j][0] = kin<IMAG>(p.c[j][0], l[j], la, lc);
            p.c[j][N - 1] = kin<IMAG>(p.c[j][N - 1], r[j], ra, rb);
        }
    }
}

// Rotating frame: the row rotation sweeps of parity 0 and 1 (pairs (x, x + 1)
// of every row, coefficients per row, src/cpucartesian.cpp:141-176).
template <class S, bool EDGE, int BUF>
__device__ __forceinline__ void patch_rrow(Patch<S> &p, const StepArgs<typename S::T> &a) {
    using T = typename S::T;
    constexpr bool IMAG = S::V::IMAG;
    constexpr int N = S::N;
    const Cx<T> *tab = reinterpret_cast<const Cx<T> *>(a.row_ab);
    const Cx<T> id{patch_one<T>(), T(0)};
    Cx<T> ab[N], in[N], l[N], r[N];
#pragma unroll
    for (int j = 0; j < N; ++j) {
        const int y = EDGE ? min(max(p.gy + j, 0), a.H - 1) : p.gy + j;
        ab[j] = tab[y];
    }
    auto pick = [&](int bit, int j) {
        return (EDGE && ((p.hm >> bit) & 1u)) ? id : ab[j];
    };
#pragma unroll
    for (int j = 0; j < N; ++j)
#pragma unroll
        for (int i = 0; i + 1 < N; i += 2) {
            const Cx<T> f = p.c[j][i], s = p.c[j][i + 1], k = pick(i + 1, j);
            p.c[j][i] = rot_first<IMAG>(f, s, k.re, k.im);
            p.c[j][i + 1] = rot_second<IMAG>(s, f, k.re, k.im);
        }
    patch_send<S, BUF, 0, 1, N>(p, in);
#pragma unroll
    for (int j = 0; j < N; ++j)
#pragma unroll
        for (int i = 1; i + 1 < N; i += 2) {
            const Cx<T> f = p.c[j][i], s = p.c[j][i + 1], k = pick(i + 1, j);
            p.c[j][i] = rot_first<IMAG>(f, s, k.re, k.im);
            p.c[j][i + 1] = rot_second<IMAG>(s, f, k.re, k.im);
        }
    patch_recv<S, BUF, N>(p, in, l, r);
#pragma unroll
    for (int j = 0; j < N; ++j) {
        const Cx<T> kl = pick(0, j), kr = pick(N, j);
        p.c[j][0] = rot_second<IMAG>(p.c[j][0], l[j], kl.re, kl.im);
        p.c[j][N - 1] = rot_first<IMAG>(p.c[j][N - 1], r[j], kr.re, kr.im);
    }
}

// and the column rotation sweeps on the pairs starting at even, then odd rows
// (coefficients per column, src/cpucartesian.cpp:179-204).
template <class S, bool EDGE>
__device__ __forceinline__ void patch_rcol(Patch<S> &p, const StepArgs<typename S::T> &a) {
    using T = typename S::T;
    constexpr bool IMAG = S::V::IMAG;
    constexpr int N = S::N;
    const Cx<T> *tab = reinterpret_cast<const Cx<T> *>(a.col_ab);
    const Cx<T> id{patch_one<T>(), T(0)};
    Cx<T> ab[N];
#pragma unroll
    for (int i = 0; i < N; ++i) {
        const int x = EDGE ? min(max(p.gx + i, 0), a.W - 1) : p.gx + i;
        ab[i] = tab[x];
    }
    auto pick = [&](int bit, int i) {
        return (EDGE && ((p.vm >> bit) & 1u)) ? id : ab[i];
    };
#pragma unroll
    for (int par = 0; par < 2; ++par) {
        Cx<T> u[N], d[N];
        if (par == 1) {
#pragma unroll
            for (int i = 0; i < N; ++i) {
                u[i].re = __shfl_up_sync(0xffffffffu, p.c[N - 1][i].re, S::WX);
                u[i].im = __shfl_up_sync(0xffffffffu, p.c[N - 1][i].im, S::WX);
                d[i].re = __shfl_down_sync(0xffffffffu, p.c[0][i].re, S::WX);
                d[i].im = __shfl_down_sync(0xffffffffu, p.c[0][i].im, S::WX);
            }
        }
#pragma unroll
        for (int j = par; j + 1 < N; j += 2)
#pragma unroll
            for (int i = 0; i < N; ++i) {
                const Cx<T> f = p.c[j][i], s = p.c[j + 1][i], k = pick(j + 1, i);
                p.c[j][i] = rot_first<IMAG>(f, s, k.re, k.im);
                p.c[j + 1][i] = rot_second<IMAG>(s, f, k.re, k.im);
            }
        if (par == 1) {
#pragma unroll
            for (int i = 0; i < N; ++i) {
                const Cx<T> ku = pick(0, i), kd = pick(N, i);
                p.c[0][i] = rot_second<IMAG>(p.c[0][i], u[i], ku.re, ku.im);
                p.c[N - 1][i] = rot_first<IMAG>(p.c[N - 1][i], d[i], kd.re, kd.im);
            }
        }
    }
}

// B bytes (a multiple of 8, aligned to min(B, 32)) of a patch row, past L1
// (no other thread of the block reads them): up to 32 bytes per load.
template <int B>
__device__ __forceinline__ void patch_ld(const void *src, void *dst) {
    const unsigned char *p = reinterpret_cast<const unsigned char *>(src);
    uint32_t *d = reinterpret_cast<uint32_t *>(dst);
    if constexpr (B >= 32) {
#pragma unroll
        for (int i = 0; i < B; i += 32)
            asm volatile(
                "ld.global.L1::no_allocate.v8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
                : "=r"(d[i / 4]), "=r"(d[i / 4 + 1]), "=r"(d[i / 4 + 2]), "=r"(d[i / 4 + 3]),
                  "=r"(d[i / 4 + 4]), "=r"(d[i / 4 + 5]), "=r"(d[i / 4 + 6]), "=r"(d[i / 4 + 7])
                : "l"(p + i)
                : "memory");
    } else if constexpr (B == 16) {
        asm volatile("ld.global.L1::no_allocate.v4.b32 {%0, %1, %2, %3}, [%4];"
                     : "=r"(d[0]), "=r"(d[1]), "=r"(d[2]), "=r"(d[3])
                     : "l"(p)
                     : "memory");
    } else {
        static_assert(B == 8, "patch rows of 8, 16 or a multiple of 32 bytes");
        asm volatile("ld.global.L1::no_allocate.v2.b32 {%0, %1}, [%2];"
                     : "=r"(d[0]), "=r"(d[1])
                     : "l"(p)
                     : "memory");
    }
}

// This thread's patch of a tile of psi cells: in EDGE, cells outside the tile
// are 0 and, with WRAP, halo cells come from the cells the periodic refresh
// would copy into them.  Rows are loaded whole where their cells lie side by
// side in the tile.
template <class S, bool EDGE, bool WRAP>
struct PatchTile {
    using T = typename S::T;
    static constexpr int N = S::N;
    const Cx<T> *at;  // the patch's first cell
    int P;
    bool whole;       // EDGE: no cell of a row outside the tile or wrapped in x

    template <class Args>
    __device__ __forceinline__ PatchTile(const Patch<S> &p, const Args &a, const void *tile)
        : at(reinterpret_cast<const Cx<T> *>(tile) + (ptrdiff_t)p.gy * a.P + p.gx), P(a.P) {
        int wx = 0;
        if constexpr (WRAP) wx = (a.wrap & 1) ? a.wrap_hx : 0;
        whole = !EDGE || (p.gx >= wx && p.gx + N <= a.W - wx);
    }
    template <class Args>
    __device__ __forceinline__ void row(const Patch<S> &p, const Args &a, int j,
                                        Cx<T> (&v)[N]) const {
        alignas(16) Cx<T> w[N];
        if constexpr (!EDGE) {
            patch_ld<N * (int)sizeof(Cx<T>)>(at + (ptrdiff_t)j * P, w);
        } else {
#pragma unroll
            for (int i = 0; i < N; ++i) w[i] = Cx<T>{T(0), T(0)};
            const int y = p.gy + j;
            if (y >= 0 && y < a.H) {
                int dy = j;
                if constexpr (WRAP) {
                    if (a.wrap & 2) {
                        if (y < a.wrap_hy) dy += a.H - 2 * a.wrap_hy;
                        else if (y >= a.H - a.wrap_hy) dy -= a.H - 2 * a.wrap_hy;
                    }
                }
                const Cx<T> *r = at + (ptrdiff_t)dy * P;
                if (whole) {
                    patch_ld<N * (int)sizeof(Cx<T>)>(r, w);
                } else {
                    const int ys = p.gy + dy;
#pragma unroll
                    for (int i = 0; i < N; ++i) {
                        const int x = p.gx + i;
                        int dx = i;
                        if constexpr (WRAP) {
                            if ((a.wrap & 1) && ys >= a.wrap_y0 && ys < a.wrap_y1) {
                                if (x < a.wrap_hx) dx += a.W - 2 * a.wrap_hx;
                                else if (x >= a.W - a.wrap_hx) dx -= a.W - 2 * a.wrap_hx;
                            }
                        }
                        if (x >= 0 && x < a.W) w[i] = ld_cx_shared(r + dx);
                    }
                }
            }
        }
#pragma unroll
        for (int i = 0; i < N; ++i) v[i] = w[i];
    }
};

// This thread's patch of the table (of the potential with V::VPOT, whose rows
// are aligned to 16 bytes only); 0 outside the tile.
template <class S, bool EDGE>
struct PatchTable {
    using T = typename S::T;
    using TabT = typename S::TabT;
    static constexpr int N = S::N;
    const TabT *at;
    ptrdiff_t pitch;
    bool whole;

    template <class Args>
    __device__ __forceinline__ PatchTable(const Patch<S> &p, const Args &a) {
        pitch = a.P;
        if constexpr (S::V::VPOT) pitch = (ptrdiff_t)(a.pot_pitch / sizeof(TabT));
        at = reinterpret_cast<const TabT *>(a.pot) + p.gy * pitch + p.gx;
        whole = !EDGE || (p.gx >= 0 && p.gx + N <= a.W);
    }
    template <class Args>
    __device__ __forceinline__ void row(const Patch<S> &p, const Args &a, int j,
                                        TabT (&v)[N]) const {
        alignas(16) TabT w[N];
#pragma unroll
        for (int i = 0; i < N; ++i) w[i] = TabT{};
        const TabT *r = at + j * pitch;
        if (!EDGE || (p.gy + j >= 0 && p.gy + j < a.H)) {
            if (whole) {
                if constexpr (S::V::VPOT) {
#pragma unroll
                    for (int i = 0; i < N; i += 2) patch_ld<2 * (int)sizeof(TabT)>(r + i, w + i);
                } else {
                    patch_ld<N * (int)sizeof(TabT)>(r, w);
                }
            } else {
#pragma unroll
                for (int i = 0; i < N; ++i)
                    if (p.gx + i >= 0 && p.gx + i < a.W) w[i] = r[i];
            }
        }
#pragma unroll
        for (int i = 0; i < N; ++i) v[i] = w[i];
    }
};

// Full rows of a patch in stores of 32 bytes (16 where the row is shorter).
template <int N>
__device__ __forceinline__ void patch_store_row(Cx<double> *o, const Cx<double> (&v)[N]) {
#pragma unroll
    for (int i = 0; i < N; i += 2)
        asm volatile("st.global.v4.f64 [%0], {%1, %2, %3, %4};" ::"l"(o + i), "d"(v[i].re),
                     "d"(v[i].im), "d"(v[i + 1].re), "d"(v[i + 1].im)
                     : "memory");
}
template <int N>
__device__ __forceinline__ void patch_store_row(Cx<float> *o, const Cx<float> (&v)[N]) {
    if constexpr (N % 4 == 0) {
#pragma unroll
        for (int i = 0; i < N; i += 4)
            asm volatile("st.global.v8.f32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"l"(o + i),
                         "f"(v[i].re), "f"(v[i].im), "f"(v[i + 1].re), "f"(v[i + 1].im),
                         "f"(v[i + 2].re), "f"(v[i + 2].im), "f"(v[i + 3].re), "f"(v[i + 3].im)
                         : "memory");
    } else {
#pragma unroll
        for (int i = 0; i < N; i += 2)
            *reinterpret_cast<float4 *>(o + i) =
                make_float4(v[i].re, v[i].im, v[i + 1].re, v[i + 1].im);
    }
}

// Factors of the other species and of the deferred renormalisation.
template <typename T>
struct PatchScale {
    T inv, pbs, cab, rcc, rsr, rsi, ror, roi, vdt;
};

// The region without its rim; its squared norm within the norm's bounds to nacc.
template <class S, bool EDGE>
__device__ __forceinline__ void patch_write(const Patch<S> &p, const StepArgs<typename S::T> &a,
                                            double &nacc) {
    using V = typename S::V;
    using T = typename S::T;
    constexpr int N = S::N;
    if (p.px < S::MX || p.px >= S::TX - S::MX || p.py < S::MY || p.py >= S::TX - S::MY) return;
    Cx<T> *o = reinterpret_cast<Cx<T> *>(a.psi_out) + (size_t)p.gy * a.P + p.gx;
#pragma unroll
    for (int j = 0; j < N; ++j) {
        if (EDGE && p.gy + j >= a.H) break;
        if (!EDGE || p.gx + N <= a.W) {
            patch_store_row<N>(o + (size_t)j * a.P, p.c[j]);
        } else {
#pragma unroll
            for (int i = 0; i < N; ++i)
                if (p.gx + i < a.W) st_cx_global(o + (size_t)j * a.P + i, p.c[j][i]);
        }
        if constexpr (V::IMAG) {
#pragma unroll
            for (int i = 0; i < N; ++i) {
                const Cx<T> v = p.c[j][i];
                if (!EDGE || (p.gx + i >= a.ix0 && p.gx + i < a.ix1 && p.gy + j >= a.iy0 &&
                              p.gy + j < a.iy1))
                    nacc += (double)v.re * (double)v.re + (double)v.im * (double)v.im;
            }
        }
    }
}

// One region: origin (X0, Y0) in tile cells.
template <class S, bool EDGE>
__device__ __forceinline__ void patch_region(Patch<S> &p, const StepArgs<typename S::T> &a, int X0,
                                             int Y0, const PatchScale<typename S::T> &f,
                                             double &nacc) {
    using V = typename S::V;
    using T = typename S::T;
    using TabT = typename S::TabT;
    constexpr int N = S::N;
    constexpr bool WRAP = !V::PB;
    p.gx = X0 + p.px * N;
    p.gy = Y0 + p.py * N;
    if constexpr (EDGE) patch_masks(p, a.W, a.H);
    const PatchTile<S, EDGE, WRAP> tile(p, a, a.psi_in);
    const PatchTable<S, EDGE> table(p, a);
#pragma unroll
    for (int j = 0; j < N; ++j) tile.row(p, a, j, p.c[j]);
    if constexpr (V::RABI) {
        // the Rabi rotation of the previous step
        const PatchTile<S, EDGE, false> other(p, a, a.pb);
#pragma unroll
        for (int j = 0; j < N; ++j) {
            Cx<T> u[N];
            other.row(p, a, j, u);
#pragma unroll
            for (int i = 0; i < N; ++i)
                p.c[j][i] = rabi_cell(p.c[j][i], scale_cx(u[i], f.pbs), f.rcc, f.rsr, f.rsi);
        }
    }
    if constexpr (V::IMAG) {
#pragma unroll
        for (int j = 0; j < N; ++j)
#pragma unroll
            for (int i = 0; i < N; ++i) p.c[j][i] = scale_cx(p.c[j][i], f.inv);
    }
    patch_vsweep<S, EDGE, 0>(p);
    patch_hsweep<S, EDGE, 0, 0>(p);
    patch_vsweep<S, EDGE, 1>(p);
    // the table of the first rows on its way during the next sweep
    constexpr int AHEAD = S::TAB_AHEAD;
    TabT tv[N][N];
#pragma unroll
    for (int j = 0; j < AHEAD; ++j) table.row(p, a, j, tv[j]);
    patch_hsweep<S, EDGE, 1, 1>(p);
    if constexpr (V::CYL) {
        patch_radial<S, EDGE, 0, 0>(p, a);
        patch_radial<S, EDGE, 1, 0>(p, a);
    }
#pragma unroll
    for (int j = 0; j < N; ++j) {
        if (j + AHEAD < N) table.row(p, a, j + AHEAD, tv[j + AHEAD]);
        if constexpr (V::PB) {
            Cx<T> ub[N], own[N];
            PatchTile<S, EDGE, false>(p, a, a.pb).row(p, a, j, ub);
            if constexpr (V::RABI) tile.row(p, a, j, own);
#pragma unroll
            for (int i = 0; i < N; ++i) {
                ub[i] = scale_cx(ub[i], f.pbs);
                if constexpr (V::RABI) ub[i] = rabi_cell(ub[i], own[i], f.rcc, f.ror, f.roi);
            }
            potential_row<V::IMAG, V::PHASE, false, true, N, false>(p.c[j], tv[j], p.ca, p.caa, &ub,
                                                                    f.cab);
        } else if constexpr (V::VPOT) {
            Cx<T> te[N];
#pragma unroll
            for (int i = 0; i < N; ++i) te[i] = vpot_table_entry(f.vdt * tv[j][i]);
            potential_row<V::IMAG, V::PHASE, V::LHY, false, N>(p.c[j], te, p.ca, p.caa);
        } else {
            potential_row<V::IMAG, V::PHASE, V::LHY, false, N, true, V::ROT>(p.c[j], tv[j], p.ca,
                                                                            p.caa);
        }
    }
    if constexpr (V::ROT) {
        patch_rrow<S, EDGE, 0>(p, a);
        patch_rcol<S, EDGE>(p, a);
        patch_rrow<S, EDGE, 1>(p, a);
    }
    if constexpr (V::CYL) {
        patch_radial<S, EDGE, 1, 1>(p, a);
        patch_radial<S, EDGE, 0, 1>(p, a);
    }
    patch_hsweep<S, EDGE, 1, 0>(p);
    patch_vsweep<S, EDGE, 1>(p);
    patch_hsweep<S, EDGE, 0, 1>(p);
    patch_vsweep<S, EDGE, 0>(p);
    if constexpr (V::CYL && V::IMAG) {
        // column 0 mirrors column 1 (src/cpukernel.cpp:669-689)
        if (p.gx == 0) {
#pragma unroll
            for (int j = 0; j < N; ++j) p.c[j][0] = Cx<T>{a.mirror_sign * p.c[j][1].re,
                                                          a.mirror_sign * p.c[j][1].im};
        }
    }
    patch_write<S, EDGE>(p, a, nacc);
}

// a.n_strips x a.n_segs regions, taken by the blocks in turn.
template <class S>
__global__ void __launch_bounds__(S::THREADS, S::BLOCKS) patch_kernel(StepArgs<typename S::T> a) {
    using V = typename S::V;
    using T = typename S::T;
    __shared__ __align__(16) unsigned char exch[2 * S::EXCH];
    // as the walks: the next step's blocks may be scheduled as this step's retire
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    const int warp = __shfl_sync(0xffffffffu, (int)(threadIdx.x >> 5), 0), lane = threadIdx.x & 31;
    Patch<S> p;
    patch_thread(p, exch);
    asm volatile("griddepcontrol.wait;" ::: "memory");
    p.aH = a.aH;
    p.bH = a.bH;
    p.aV = a.aV;
    p.bV = a.bV;
    if constexpr (DeltaForm<T>::value && !V::IMAG) {
        if (a.kin_sched) {
            const unsigned int step = __ldcg(&a.scal->step);
            const float4 c = __ldg(&a.kin_sched[step % (unsigned int)a.sched_len]);
            p.aH = c.x;
            p.bH = c.y;
            p.aV = c.z;
            p.bV = c.w;
        }
    }
    p.ca = a.ca;
    p.caa = a.caa;
    PatchScale<T> f{};
    if constexpr (V::IMAG) f.inv = (T)a.scal->pending_inv;
    if constexpr (V::PB) {
        f.pbs = (T)__ldcg(a.pb_scale);
        f.cab = a.cab;
    }
    if constexpr (V::RABI) {
        f.rcc = a.rabi_cc;
        f.rsr = a.rabi_sr;
        f.rsi = a.rabi_si;
        f.ror = a.rabi_or;
        f.roi = a.rabi_oi;
    }
    if constexpr (V::VPOT) f.vdt = (T)a.pot_dt;
    // inside a region: no pair across the tile's edge, no wrapped cell, every
    // written cell in the norm's region
    const int wx = (a.wrap & 1) ? a.wrap_hx : 0, wy = (a.wrap & 2) ? a.wrap_hy : 0;
    double nacc = 0.0;
    const int n = a.n_strips * a.n_segs;
    for (int t = blockIdx.x; t < n; t += gridDim.x) {
        const int X0 = (t % a.n_strips) * S::OX - S::MX * S::N;
        const int Y0 = (t / a.n_strips) * S::OY - S::MY * S::N;
        const bool inside = X0 >= wx && Y0 >= wy && X0 + S::R <= a.W - wx && Y0 + S::R <= a.H - wy &&
                            X0 + S::MX * S::N >= a.ix0 && X0 + S::MX * S::N + S::OX <= a.ix1 &&
                            Y0 + S::MY * S::N >= a.iy0 && Y0 + S::MY * S::N + S::OY <= a.iy1;
        if (inside)
            patch_region<S, false>(p, a, X0, Y0, f, nacc);
        else
            patch_region<S, true>(p, a, X0, Y0, f, nacc);
    }
    // the first exchange buffer is free: every thread is past its last read of
    // it when the last sweep's barrier opens
    w2_finish<V>(a, nacc, S::THREADS / 32, warp, lane, reinterpret_cast<double *>(exch));
}

// M steps of a closed tile in real time: each spoils V::HX more columns and
// V::HY more rows at the region's rim, so that M steps recompute more cells
// than M launches, but load, store and launch once.  Of a small tile's step of
// 3.1 us, 2.4 are those and 0.7 the nine stages (64^2 double, two steps 3.8).
// Nothing leaves the region between steps: a periodic halo, a squared norm or
// another species would have to.
template <class S, bool EDGE>
__device__ __forceinline__ void patch_region_steps(Patch<S> &p, const StepArgs<typename S::T> &a,
                                                   int X0, int Y0) {
    using V = typename S::V;
    using T = typename S::T;
    using TabT = typename S::TabT;
    constexpr int N = S::N;
    // the table stays in registers where it takes 4 cells
    constexpr bool HOLD = N == 2;
    p.gx = X0 + p.px * N;
    p.gy = Y0 + p.py * N;
    if constexpr (EDGE) patch_masks(p, a.W, a.H);
    const PatchTile<S, EDGE, false> tile(p, a, a.psi_in);
    const PatchTable<S, EDGE> table(p, a);
#pragma unroll
    for (int j = 0; j < N; ++j) tile.row(p, a, j, p.c[j]);
    TabT tv[HOLD ? N : 1][N];
    if constexpr (HOLD) {
#pragma unroll
        for (int j = 0; j < N; ++j) table.row(p, a, j, tv[j]);
    }
    unsigned int step = 0;
    if constexpr (DeltaForm<T>::value) step = __ldcg(&a.scal->step);
#pragma unroll 1
    for (int m = 0; m < S::M; ++m) {
        if constexpr (DeltaForm<T>::value) {
            const float4 c = __ldg(&a.kin_sched[(step + m) % (unsigned int)a.sched_len]);
            p.aH = c.x;
            p.bH = c.y;
            p.aV = c.z;
            p.bV = c.w;
        }
        patch_vsweep<S, EDGE, 0>(p);
        patch_hsweep<S, EDGE, 0, 0>(p);
        patch_vsweep<S, EDGE, 1>(p);
        if constexpr (!HOLD) table.row(p, a, 0, tv[0]);
        patch_hsweep<S, EDGE, 1, 1>(p);
#pragma unroll
        for (int j = 0; j < N; ++j) {
            if (!HOLD && j > 0) table.row(p, a, j, tv[0]);
            potential_row<false, V::PHASE, V::LHY, false, N, true, false>(p.c[j], tv[HOLD ? j : 0],
                                                                          p.ca, p.caa);
        }
        patch_hsweep<S, EDGE, 1, 0>(p);
        patch_vsweep<S, EDGE, 1>(p);
        patch_hsweep<S, EDGE, 0, 1>(p);
        patch_vsweep<S, EDGE, 0>(p);
    }
    double none = 0.0;
    patch_write<S, EDGE>(p, a, none);
}

template <class S>
__global__ void __launch_bounds__(S::THREADS, S::BLOCKS)
    patch_steps_kernel(StepArgs<typename S::T> a) {
    using V = typename S::V;
    static_assert(!V::IMAG && !V::ROT && !V::CYL && !V::PB && !V::VPOT, "plain real time only");
    __shared__ __align__(16) unsigned char exch[2 * S::EXCH];
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    const int warp = __shfl_sync(0xffffffffu, (int)(threadIdx.x >> 5), 0), lane = threadIdx.x & 31;
    Patch<S> p;
    patch_thread(p, exch);
    asm volatile("griddepcontrol.wait;" ::: "memory");
    p.aH = a.aH;
    p.bH = a.bH;
    p.aV = a.aV;
    p.bV = a.bV;
    p.ca = a.ca;
    p.caa = a.caa;
    const int n = a.n_strips * a.n_segs;
    for (int t = blockIdx.x; t < n; t += gridDim.x) {
        const int X0 = (t % a.n_strips) * S::OX - S::MX * S::N;
        const int Y0 = (t / a.n_strips) * S::OY - S::MY * S::N;
        if (X0 >= 0 && Y0 >= 0 && X0 + S::R <= a.W && Y0 + S::R <= a.H)
            patch_region_steps<S, false>(p, a, X0, Y0);
        else
            patch_region_steps<S, true>(p, a, X0, Y0);
    }
    w2_finish<V>(a, 0.0, S::THREADS / 32, warp, lane, nullptr, S::M);
}

}  // namespace tsb
