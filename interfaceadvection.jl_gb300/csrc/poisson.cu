// Variable-coefficient pressure Poisson solve of the projection step
// (InterfaceAdvection.jl src/flow.jl:328-347, where WaterLily's
// MultiLevelPoisson `solver!` runs V-cycles inside a PCG wrapper).
//
// Operator (WaterLily `mult`): (A x)_I = Σ_i L[I,i] x[I-δi] + L[I+δi,i] x[I+δi]
// + D_I x_I with D_I = -Σ_i (L[I,i] + L[I+δi,i]); L = μ₀ = 1/ρ on faces, zero
// on wall faces, periodic dimensions wrap.  The solver is this library's own:
//
//  * geometric multigrid on cell-centred levels of any size (a dimension halves,
//    an odd one with a single cell left at its end); coarse face coefficient =
//    Σ of the fine faces it covers times the ratio of the cell distances (½ away
//    from single cells); restriction sums the children, prolongation injects;
//    red-black Gauss-Seidel, ν₁ sweeps red→black
//    before and ν₂ black→red after, so the V-cycle is a symmetric
//    preconditioner; the coarsest level is solved by one block with a fixed
//    number of symmetric sweeps on the mean-free right-hand side;
//  * flexible CG around it (β from the residual change, so an inexact
//    V-cycle stays admissible).
//
// IA_POISSON_FP64 runs all of it in FP64 and stops on the L∞ norm of the CG's
// residual, which starts as the true one of the dt-scaled system and follows
// its recurrence (apart by rounding alone).  IA_POISSON_MIXED corrects in FP64
// with inner CG solves in FP32 (FP32 copies of every level's operator) and
// stops on the FP64 true residual, formed anew after every correction.
// IA_POISSON_LEARNED keeps the MIXED structure and preconditions the inner FCG
// with the conv net (nn.cu), composed with the V-cycle (hybrid) or alone; an
// outer correction that fails to halve the FP64 true residual switches the
// rest of the solve to the plain V-cycle.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstring>
#include <type_traits>
#include <vector>

#include "capi_internal.cuh"
#include "ia_bc.cuh"
#include "ff.cuh"
#include "poisson.cuh"

namespace ia {

namespace {

inline dim3 blk() { return dim3(32, 8, 1); }
inline dim3 grd(const Grid& g) { return dim3((g.n[0] + 31) / 32, (g.n[1] + 7) / 8, g.n[2]); }

// face coefficient as the arithmetic type of the sweep (the finest mixed level may store them as FP16)
__device__ __forceinline__ float cf(float v) { return v; }
__device__ __forceinline__ double cf(double v) { return v; }
__device__ __forceinline__ float cf(__half v) { return __half2float(v); }

// ---- dimension-specialised stencil with 32-bit cell offsets (a grid holds < 2^31 cells)
struct Nb {
    int xl, xh, yl, yh, zl, zh;   // offsets of the six neighbours; periodic ends wrap
};
template <int D>
__device__ __forceinline__ Nb nb_of(const Grid& g, int x, int y, int z) {
    Nb o;
    const int s1 = int(g.s[1]), s2 = int(g.s[2]);
    o.xl = (g.isper(0) && x == 1) ? g.n[0] - 3 : -1;
    o.xh = (g.isper(0) && x == g.n[0] - 2) ? 3 - g.n[0] : 1;
    o.yl = (g.isper(1) && y == 1) ? (g.n[1] - 3) * s1 : -s1;
    o.yh = (g.isper(1) && y == g.n[1] - 2) ? (3 - g.n[1]) * s1 : s1;
    o.zl = o.zh = 0;
    if (D == 3) {
        o.zl = (g.isper(2) && z == 1) ? (g.n[2] - 3) * s2 : -s2;
        o.zh = (g.isper(2) && z == g.n[2] - 2) ? (3 - g.n[2]) * s2 : s2;
    }
    return o;
}
// Σ_i L[I,i] v[I-δi] + L[I+δi,i] v[I+δi]
template <int D, class T, class TL>
__device__ __forceinline__ T off7(const Grid& g, const TL* __restrict__ L, const T* v, int I, const Nb& o) {
    const int s1 = int(g.s[1]), s2 = int(g.s[2]);
    const TL* L1 = L + g.N;
    T a = cf(L[I]) * v[I + o.xl] + cf(L[I + 1]) * v[I + o.xh];
    a += cf(L1[I]) * v[I + o.yl] + cf(L1[I + s1]) * v[I + o.yh];
    if (D == 3) {
        const TL* L2 = L1 + g.N;
        a += cf(L2[I]) * v[I + o.zl] + cf(L2[I + s2]) * v[I + o.zh];
    }
    return a;
}
// b - Σ_i L[I,i] v[I-δi] + L[I+δi,i] v[I+δi] as one chain of multiply-adds
template <int D, class T>
__device__ __forceinline__ T resid7(const Grid& g, const T* __restrict__ L, T b, const T* v, int I, const Nb& o) {
    const int s1 = int(g.s[1]), s2 = int(g.s[2]);
    const T* L1 = L + g.N;
    T a = fma(-L[I], v[I + o.xl], b);
    a = fma(-L[I + 1], v[I + o.xh], a);
    a = fma(-L1[I], v[I + o.yl], a);
    a = fma(-L1[I + s1], v[I + o.yh], a);
    if (D == 3) {
        const T* L2 = L1 + g.N;
        a = fma(-L2[I], v[I + o.zl], a);
        a = fma(-L2[I + s2], v[I + o.zh], a);
    }
    return a;
}
// b + Σ_i L[I,i] v[I-δi] + L[I+δi,i] v[I+δi] likewise (a result's sign is an FP64 operation too)
template <int D, class T>
__device__ __forceinline__ T product7(const Grid& g, const T* __restrict__ L, T b, const T* v, int I, const Nb& o) {
    const int s1 = int(g.s[1]), s2 = int(g.s[2]);
    const T* L1 = L + g.N;
    T a = fma(L[I], v[I + o.xl], b);
    a = fma(L[I + 1], v[I + o.xh], a);
    a = fma(L1[I], v[I + o.yl], a);
    a = fma(L1[I + s1], v[I + o.yh], a);
    if (D == 3) {
        const T* L2 = L1 + g.N;
        a = fma(L2[I], v[I + o.zl], a);
        a = fma(L2[I + s2], v[I + o.zh], a);
    }
    return a;
}
// D_I = -Σ_i (L[I,i] + L[I+δi,i])
template <int D, class TL>
__device__ __forceinline__ auto diag7(const Grid& g, const TL* __restrict__ L, int I) -> decltype(cf(L[0])) {
    using T = decltype(cf(L[0]));
    const int s1 = int(g.s[1]), s2 = int(g.s[2]);
    const TL* L1 = L + g.N;
    T dd = T(0);
    dd -= cf(L[I]) + cf(L[I + 1]);
    dd -= cf(L1[I]) + cf(L1[I + s1]);
    if (D == 3) {
        const TL* L2 = L1 + g.N;
        dd -= cf(L2[I]) + cf(L2[I + s2]);
    }
    return dd;
}
// interior-cell launch: x, y from the 2D block, z from blockIdx.z (3D) or 0 (2D)
#define CELL_INTERIOR(g)                                                  \
    const int x = 1 + blockIdx.x * blockDim.x + threadIdx.x;              \
    const int y = 1 + blockIdx.y * blockDim.y + threadIdx.y;              \
    const int z = D == 3 ? 1 + int(blockIdx.z) : 0;                       \
    if (x > (g).n[0] - 2 || y > (g).n[1] - 2) return;                     \
    const int I = x + y * int((g).s[1]) + z * int((g).s[2]);
// v == 1; in FP64 on the bit pattern, as a comparison takes the FP64 pipe as long as a sum
__device__ __forceinline__ bool is_one(float v) { return v == 1.f; }
__device__ __forceinline__ bool is_one(double v) { return __double_as_longlong(v) == 0x3FF0000000000000ll; }
// The column and row of a thread of a smoother or restriction launch on a level of nx columns.  FP32: a warp takes 32
// columns of a row.  FP64: rows follow one another through the lanes, as a warp's instruction takes as long with half of
// its lanes idle (100x200x100, whose 50 pairs a row fill 78 % of two warps: a half-sweep, mean over the levels, 8.1 us with
// rows of their own and 6.3 so).
template <class T>
__device__ __forceinline__ void plane_cell(int nx, int& col, int& row) {
    if (sizeof(T) == 8) {
        const int t = int(blockIdx.x) * 256 + int(threadIdx.y) * 32 + int(threadIdx.x);
        row = t / nx;
        col = t - row * nx;
    } else {
        col = int(blockIdx.x) * 32 + int(threadIdx.x);
        row = int(blockIdx.y) * 8 + int(threadIdx.y);
    }
}
template <class T>
inline dim3 plane_grid(int nx, int rows, int planes) {
    if (sizeof(T) == 8) return dim3(unsigned(((long long)nx * rows + 255) / 256), 1, planes);
    return dim3((nx + 31) / 32, (rows + 7) / 8, planes);
}
inline dim3 cell_grid(const Grid& g) {
    return dim3((g.n[0] - 2 + 31) / 32, (g.n[1] - 2 + 7) / 8, g.D == 3 ? g.n[2] - 2 : 1);
}
// launch K<D> for the grid's dimension
#define LAUNCH_D(gg, K, grid, block, ...)                                             \
    do {                                                                              \
        if ((gg).D == 3) { K<3><<<grid, block, 0, st>>>(__VA_ARGS__); ia::note_launch(); } \
        else { K<2><<<grid, block, 0, st>>>(__VA_ARGS__); ia::note_launch(); }             \
    } while (0)

#define INTERIOR_XYZ                                                                                     \
    const int x = blockIdx.x * blockDim.x + threadIdx.x, y = blockIdx.y * blockDim.y + threadIdx.y;     \
    const int z = blockIdx.z;                                                                            \
    if (x < 1 || y < 1 || x > g.n[0] - 2 || y > g.n[1] - 2) return;                                      \
    if (g.D == 3 && (z < 1 || z > g.n[2] - 2)) return;                                                   \
    [[maybe_unused]] const int c[3] = {x, y, z};                                                         \
    const long long I = lin(g, x, y, z);

template <class T>
__global__ void set_diag_k(Grid g, const T* __restrict__ L, T* __restrict__ iD, T* __restrict__ diag) {
    INTERIOR_XYZ
    T dd = T(0);
    for (int i = 0; i < g.D; ++i) dd -= L[I + i * g.N] + L[I + g.s[i] + i * g.N];
    const T eps = sizeof(T) == 8 ? T(2.220446049250313e-16) : T(1.1920929e-7);
    iD[I] = (dd * dd < T(2) * eps) ? T(0) : T(1) / dd;
    if (diag) diag[I] = dd;
}

// Coarsening along a dimension e of n cells: the first pr[e] coarse cells cover two fine cells each, the
// others one.  A dimension between walls takes (n+1)/2 coarse cells (one single when n is odd); a periodic
// one the next even number of them, so that the red-black colouring closes across the wrap on every coarse
// level (2 singles when n/2 is odd), and one cell after two (its faces then join the cell to itself and
// carry no coefficient).
// Fine cell c lies in coarse cell mg_parent; coarse cell c covers mg_children fine cells from mg_child on.
__device__ __forceinline__ int mg_parent(const Grid& gc, int e, int c) { return max((c + 1) >> 1, c - gc.pr[e]); }
__device__ __forceinline__ int mg_child(const Grid& gc, int e, int c) { return c <= gc.pr[e] ? 2 * c - 1 : c + gc.pr[e]; }
__device__ __forceinline__ int mg_children(const Grid& gc, int e, int c) { return c <= gc.pr[e] ? 2 : 1; }
// REG: every coarse cell covers two fine ones along each dimension, so that the parent is (c+1)/2; on the finest
// levels of a large grid the general form's extra index arithmetic costs 8 to 16 % of a kernel's time.
template <bool REG>
__device__ __forceinline__ int mg_up(const Grid& gc, int e, int c) { return REG ? (c + 1) >> 1 : mg_parent(gc, e, c); }
template <bool REG>
__device__ __forceinline__ long long mg_parent_cell(const Grid& gc, int x, int y, int z) {
    return lin(gc, mg_up<REG>(gc, 0, x), mg_up<REG>(gc, 1, y), gc.D == 3 ? mg_up<REG>(gc, 2, z) : 0);
}
inline bool mg_regular(const Grid& g, const Grid& gc) {
    for (int e = 0; e < g.D; ++e)
        if (2 * gc.pr[e] != g.n[e] - 2) return false;
    return true;
}
// A periodic dimension with an odd number of cells (possible on the finest level only) puts two cells of one
// colour next to each other across the wrap.  A half-sweep there runs in passes: cells are told apart by the
// set of such dimensions in whose last plane they lie, and neighbours across a wrap differ in that set.
__host__ __device__ inline int wrap_conflicts(const Grid& g) {
    int m = 0;
    for (int e = 0; e < g.D; ++e)
        if (g.isper(e) && (g.n[e] & 1) && g.n[e] > 3) m |= 1 << e;
    return m;
}
__device__ __forceinline__ int wrap_class(const Grid& g, int conflicts, int x, int y, int z) {
    return (((conflicts & 1) && x == g.n[0] - 2) ? 1 : 0) | (((conflicts & 2) && y == g.n[1] - 2) ? 2 : 0) |
           (((conflicts & 4) && z == g.n[2] - 2) ? 4 : 0);
}

// Coarse face coefficients: Σ over the fine faces covering each coarse face times ratio[e][c], the distance of
// the fine cells beside face c along e over that of the coarse cells (½ between coarse cells of two fine ones);
// all coarse faces 1..n-1 along i, interior elsewhere.
template <class T>
__global__ void restrict_L_k(Grid gc, Grid gf, const T* __restrict__ Lf, const double* __restrict__ ratio,
                             T* __restrict__ Lc) {
    const int x = blockIdx.x * blockDim.x + threadIdx.x, y = blockIdx.y * blockDim.y + threadIdx.y;
    const int z = blockIdx.z;
    if (x >= gc.n[0] || y >= gc.n[1]) return;
    const int c[3] = {x, y, z};
    const long long Ic = lin(gc, x, y, z);
    for (int i = 0; i < gc.D; ++i) {
        bool ok = true;
        for (int e = 0; e < gc.D; ++e) {
            const int hi = (e == i) ? gc.n[e] - 1 : gc.n[e] - 2;
            if (c[e] < 1 || c[e] > hi) ok = false;
        }
        if (!ok) continue;
        // fine base cell of the face: the first child in every dimension
        int fb[3] = {mg_child(gc, 0, c[0]), mg_child(gc, 1, c[1]), gc.D == 3 ? mg_child(gc, 2, c[2]) : 0};
        T s = T(0);
        const int o1 = (i == 0) ? 1 : 0, o2 = (i == 2) ? 1 : 2;   // the other dimensions
        const int n1 = mg_children(gc, o1, c[o1]), n2 = (gc.D == 3) ? mg_children(gc, o2, c[o2]) : 1;
        for (int b = 0; b < n2; ++b)
            for (int a = 0; a < n1; ++a) {
                int q[3] = {fb[0], fb[1], fb[2]};
                q[o1] += a;
                if (gc.D == 3) q[o2] += b;
                s += Lf[lin(gf, q[0], q[1], q[2]) + i * gf.N];
            }
        Lc[Ic + i * gc.N] = T(ratio[(i > 0 ? gc.n[0] : 0) + (i > 1 ? gc.n[1] : 0) + c[i]]) * s;
    }
}

// Red-black Gauss-Seidel half-sweep, one thread per cell of the colour: thread tx takes the pair of
// interior cells (1 + 2tx, 2 + 2tx) of its row and updates the one of this colour, so no
// lane idles; in FP32 the diagonal comes from the face coefficients the update reads anyway
// (same value and zero-diagonal rule as set_diag_k).  In FP64 the inverse diagonal is read (set_diag_k) and the
// update is a chain of 8 multiply-adds: with the diagonal's sums and the division it was about 30 FP64
// instructions a cell, at 16 cycles a warp each the whole cost (100x200x100, mean over the levels: 18.2 -> 8.1 us).
// With PROL (over-relaxed first red half-sweep of a post-smoothing whose prolongation is fused
// into the sweeps) the cell's previous value is x + the injected coarse correction.
// In 3D a thread takes its pair in RB_ZT consecutive z planes and reads every plane's operands before
// it stores: a half-sweep reads only the other colour, so no plane's store changes what another plane
// reads, and the loads of all planes are in flight at once (the z neighbours of one plane are the x
// neighbours of the next, a repeated address).  The values are those of one plane per thread.
constexpr int RB_ZT = 2;
template <class T, int D, bool PROL = false, class TL = T, bool REG = true>
__global__ void rbgs_pair_k(Grid g, int y0, int y1, const TL* __restrict__ L, const T* __restrict__ b,
                            const T* __restrict__ iD, T* __restrict__ xv, int color, T omega, int conflicts, int cls,
                            Grid gc = Grid(), const T* __restrict__ xc = nullptr) {
    int pair, y;
    plane_cell<T>((g.n[0] - 1) / 2, pair, y);
    y += y0;   // rows [y0, y1) of the interior
    if (y >= y1) return;
    const int xp = 1 + 2 * pair;
    const int z0 = D == 3 ? 1 + RB_ZT * int(blockIdx.z) : 0;
    const T eps = sizeof(T) == 8 ? T(2.220446049250313e-16) : T(1.1920929e-7);
    // plane k's cell of this colour and its operands: the off-diagonal sum, the diagonal, b and
    // (over-relaxed) the previous value
    auto cell_of = [&](int z) {
        int x = xp;
        if (((x + y + z) & 1) != color) ++x;
        // with wrap conflicts, a pass takes the cells of its class alone (any x past the row is no cell)
        if (conflicts && wrap_class(g, conflicts, x, y, z) != cls) x = g.n[0];
        return x;
    };
    auto load = [&](int x, int z, int& I, T& off, T& dd, T& bv, T& xo) {
        I = x + y * int(g.s[1]) + z * int(g.s[2]);
        const Nb o = nb_of<D>(g, x, y, z);
        if constexpr (sizeof(T) == 8) {
            off = T(0);
            dd = iD[I];
            bv = resid7<D>(g, L, b[I], xv, I, o);
        } else {
            off = off7<D>(g, L, xv, I, o);
            dd = diag7<D>(g, L, I);
            bv = b[I];
        }
        if (!is_one(omega)) {
            xo = xv[I];
            if (PROL) xo += xc[mg_parent_cell<REG>(gc, x, y, z)];
        }
    };
    auto store = [&](int I, T off, T dd, T bv, T xo) {
        if constexpr (sizeof(T) == 8) {
            xv[I] = is_one(omega) ? bv * dd : fma(omega, fma(bv, dd, -xo), xo);
            return;
        }
        const T iD = (dd * dd < T(2) * eps) ? T(0) : T(1) / dd;
        const T gs = (bv - off) * iD;
        if (is_one(omega)) xv[I] = gs;
        else xv[I] = xo + omega * (gs - xo);   // over-relaxation: x + ω (x_GS - x)
    };
    const int xmax = g.n[0] - 2;
    if (D == 3 && z0 + RB_ZT - 1 <= g.n[2] - 2) {
        int I[RB_ZT];
        T off[RB_ZT], dd[RB_ZT], bv[RB_ZT], xo[RB_ZT];
        bool ok[RB_ZT];
#pragma unroll
        for (int k = 0; k < RB_ZT; ++k) {
            const int x = cell_of(z0 + k);
            ok[k] = x <= xmax;
            xo[k] = T(0);
            if (ok[k]) load(x, z0 + k, I[k], off[k], dd[k], bv[k], xo[k]);
        }
#pragma unroll
        for (int k = 0; k < RB_ZT; ++k)
            if (ok[k]) store(I[k], off[k], dd[k], bv[k], xo[k]);
        return;
    }
    for (int k = 0; k < (D == 3 ? RB_ZT : 1); ++k) {
        const int z = z0 + k;
        if (D == 3 && z > g.n[2] - 2) break;
        const int x = cell_of(z);
        if (x > xmax) continue;
        int I;
        T off, dd, bv, xo = T(0);
        load(x, z, I, off, dd, bv, xo);
        store(I, off, dd, bv, xo);
    }
}

// ---- first half-sweep of a smoothing, fused with the pass before it.  A red update reads only
// black neighbours, so the red values that precede a smoothing's first (black) half-sweep are
// consumed by that half-sweep alone: they are computed here where read, b (1/D) for the
// pre-smoothing from x = 0 (the first red sweep, whose neighbours are zero) and x + the
// injected coarse correction for the post-smoothing (prolong_k's values, interior cells only).  The red cells are written only for
// a pre-smoothing of one sweep (write_red), whose red values are part of its result.
template <class T, bool PROL, bool REG>
__device__ __forceinline__ T first_nb(const Grid& g, const Grid& gc, const T* __restrict__ b,
                                      const T* __restrict__ iD, const T* __restrict__ xc, const T* xv, int J,
                                      int cx, int cy, int cz, T omega) {
    // J, (cx, cy, cz): index and (periodically wrapped) coordinates of the neighbour
    const bool in = cx >= 1 && cx <= g.n[0] - 2 && cy >= 1 && cy <= g.n[1] - 2 &&
                    (g.D == 2 || (cz >= 1 && cz <= g.n[2] - 2));
    if (!in) return xv[J];
    if (!PROL && sizeof(T) == 8) return b[J] * iD[J];   // the caller's sum takes the factor omega
    if (PROL) return xv[J] + xc[mg_parent_cell<REG>(gc, cx, cy, cz)];
    return is_one(omega) ? b[J] * iD[J] : omega * (b[J] * iD[J]);
}

template <class T, int D, bool PROL, class TL = T, bool REG = true>
__global__ void rbgs_first_k(Grid g, int y0, int y1, Grid gc, const TL* __restrict__ L, const T* __restrict__ b,
                             const T* __restrict__ iD, const T* __restrict__ xc, T* __restrict__ xv, int write_red,
                             T omega) {
    int pair, y;
    plane_cell<T>((g.n[0] - 1) / 2, pair, y);
    y += y0;   // rows [y0, y1) of the interior
    const int z = D == 3 ? 1 + int(blockIdx.z) : 0;
    if (y >= y1) return;
    const int x0 = 1 + 2 * pair;
    const bool blk0 = ((x0 + y + z) & 1) == 1;
    const int x = blk0 ? x0 : x0 + 1, xr = blk0 ? x0 + 1 : x0;   // black and red cell of the pair
    const int s1 = int(g.s[1]), s2 = int(g.s[2]);
    if (!PROL && write_red && xr <= g.n[0] - 2) {
        const int Ir = xr + y * s1 + z * s2;
        xv[Ir] = is_one(omega) ? b[Ir] * iD[Ir] : omega * (b[Ir] * iD[Ir]);
    }
    if (x > g.n[0] - 2) return;
    const int I = x + y * s1 + z * s2;
    const TL* L1 = L + g.N;
    const TL* L2 = L1 + g.N;
    // the six neighbour values, then one shared accumulation (the same sums in the same order
    // whichever way the values were found)
    T v[6] = {T(0), T(0), T(0), T(0), T(0), T(0)};
    if (x >= 2 && x <= g.n[0] - 3 && y >= 2 && y <= g.n[1] - 3 && (D == 2 || (z >= 2 && z <= g.n[2] - 3))) {
        // every neighbour interior, no wrap
        const int J[6] = {I - 1, I + 1, I - s1, I + s1, I - s2, I + s2};
        if (PROL) {
            const int g1 = int(gc.s[1]), g2 = int(gc.s[2]);
            const int px = mg_up<REG>(gc, 0, x), py = mg_up<REG>(gc, 1, y) * g1, pz = D == 3 ? mg_up<REG>(gc, 2, z) * g2 : 0;
            const int P = px + py + pz;
            int Pn[6];
            if (REG) {   // the cell's own parent, or the one below (above) when the coordinate is odd (even)
                Pn[0] = P - ((x & 1) ? 1 : 0);
                Pn[1] = P + ((x & 1) ? 0 : 1);
                Pn[2] = P - ((y & 1) ? g1 : 0);
                Pn[3] = P + ((y & 1) ? 0 : g1);
                Pn[4] = P - ((z & 1) ? g2 : 0);
                Pn[5] = P + ((z & 1) ? 0 : g2);
            } else {
                Pn[0] = P - px + mg_up<REG>(gc, 0, x - 1);
                Pn[1] = P - px + mg_up<REG>(gc, 0, x + 1);
                Pn[2] = P - py + mg_up<REG>(gc, 1, y - 1) * g1;
                Pn[3] = P - py + mg_up<REG>(gc, 1, y + 1) * g1;
                Pn[4] = P - pz + (D == 3 ? mg_up<REG>(gc, 2, z - 1) * g2 : 0);
                Pn[5] = P - pz + (D == 3 ? mg_up<REG>(gc, 2, z + 1) * g2 : 0);
            }
#pragma unroll
            for (int q = 0; q < 2 * D; ++q) v[q] = xv[J[q]] + xc[Pn[q]];
        } else {
#pragma unroll
            for (int q = 0; q < 2 * D; ++q)
                v[q] = is_one(omega) || sizeof(T) == 8 ? b[J[q]] * iD[J[q]] : omega * (b[J[q]] * iD[J[q]]);
        }
    } else {
        const Nb o = nb_of<D>(g, x, y, z);
        const int xl = (g.isper(0) && x == 1) ? g.n[0] - 2 : x - 1, xh = (g.isper(0) && x == g.n[0] - 2) ? 1 : x + 1;
        const int yl = (g.isper(1) && y == 1) ? g.n[1] - 2 : y - 1, yh = (g.isper(1) && y == g.n[1] - 2) ? 1 : y + 1;
        v[0] = first_nb<T, PROL, REG>(g, gc, b, iD, xc, xv, I + o.xl, xl, y, z, omega);
        v[1] = first_nb<T, PROL, REG>(g, gc, b, iD, xc, xv, I + o.xh, xh, y, z, omega);
        v[2] = first_nb<T, PROL, REG>(g, gc, b, iD, xc, xv, I + o.yl, x, yl, z, omega);
        v[3] = first_nb<T, PROL, REG>(g, gc, b, iD, xc, xv, I + o.yh, x, yh, z, omega);
        if (D == 3) {
            const int zl = (g.isper(2) && z == 1) ? g.n[2] - 2 : z - 1, zh = (g.isper(2) && z == g.n[2] - 2) ? 1 : z + 1;
            v[4] = first_nb<T, PROL, REG>(g, gc, b, iD, xc, xv, I + o.zl, x, y, zl, omega);
            v[5] = first_nb<T, PROL, REG>(g, gc, b, iD, xc, xv, I + o.zh, x, y, zh, omega);
        }
    }
    if constexpr (sizeof(T) == 8) {
        T a = fma(L[I], v[0], L[I + 1] * v[1]);
        a = fma(L1[I], v[2], a);
        a = fma(L1[I + s1], v[3], a);
        if (D == 3) {
            a = fma(L2[I], v[4], a);
            a = fma(L2[I + s2], v[5], a);
        }
        if (PROL) {
            const T gs = (b[I] - a) * iD[I];
            const T xo = is_one(omega) ? T(0) : xv[I] + xc[mg_parent_cell<REG>(gc, x, y, z)];
            xv[I] = is_one(omega) ? gs : fma(omega, gs - xo, xo);
        } else {
            xv[I] = omega * (fma(-omega, a, b[I]) * iD[I]);
        }
        return;
    }
    T a = cf(L[I]) * v[0] + cf(L[I + 1]) * v[1];
    a += cf(L1[I]) * v[2] + cf(L1[I + s1]) * v[3];
    if (D == 3) a += cf(L2[I]) * v[4] + cf(L2[I + s2]) * v[5];
    const T dd = diag7<D>(g, L, I);
    const T eps = sizeof(T) == 8 ? T(2.220446049250313e-16) : T(1.1920929e-7);
    const T iDI = (dd * dd < T(2) * eps) ? T(0) : T(1) / dd;
    const T gs = (b[I] - a) * iDI;
    if (is_one(omega)) {
        xv[I] = gs;
    } else if (PROL) {   // over-relaxation from the prolongated value of this (black) cell
        const T xo = xv[I] + xc[mg_parent_cell<REG>(gc, x, y, z)];
        xv[I] = xo + omega * (gs - xo);
    } else {             // from x = 0
        xv[I] = omega * gs;
    }
}

#include "poisson_regular.cuh"

// ---- temporally blocked red-black Gauss-Seidel (3D, FP32): S half-sweeps in one launch.
// A block owns a TB_X x TB_Y column of interior cells and a range of z-planes and marches up
// z as a wavefront: at step t half-sweep s works on plane t - s over the column widened by
// S-1-s cells on every side, so that half-sweep s+1 finds every neighbour it reads in shared
// memory (three planes per half-sweep).  The widened parts are recomputed by every block that
// needs them, from the same inputs with the same arithmetic, so a cell has one value whichever
// block computes it; only its owner writes it.  Half-sweep s updates colour (c0 + s) & 1 with
// rbgs_pair_k's sums in rbgs_pair_k's order and the stored inverse diagonal (set_diag_k, the
// same formula).  A cell ends in x_out with the value of the last half-sweep of its colour.
// The input is zero (pre-smoothing: the V-cycle starts from x = 0) or x_in plus the injection
// prolongation of a coarse correction (post-smoothing).  Periodic dimensions wrap the widened
// column onto the grid (an even number of interior cells keeps the colouring); along a wall
// the cells outside the interior hold zero and their face coefficients are zero.
constexpr int TB_X = 32, TB_Y = 16, TB_T = 256;

struct TbArgs {
    Grid g, gc;            // level, coarse level (prolongation)
    const float* L;
    const float* b;
    const float* iD;
    const float* xin;      // post-smoothing input (null: start from zero)
    const float* xc;       // coarse correction added to xin (or null)
    float* xout;
    int c0;                // colour of the first half-sweep
    int zchunk;            // z-planes owned by a block
};

// grid coordinate of the logical coordinate l along e: periodic images wrap onto the
// interior, wall cells outside the interior are not valid
__device__ __forceinline__ int tb_wrap(const Grid& g, int e, int l, bool& ok) {
    const int m = g.n[e] - 2;
    if (g.isper(e)) {
        int p = l;
        while (p < 1) p += m;
        while (p > m) p -= m;
        ok = true;
        return p;
    }
    ok = l >= 1 && l <= m;
    return l;
}

__device__ __forceinline__ int tb_slot(int zl) { return (zl + 3 * 64) % 3; }

template <int S, bool ZERO>
__global__ void __launch_bounds__(TB_T, 4) rbgs_tb_k(TbArgs a) {
    // frame position (fx, fy) <-> logical cell (ox - S + fx, oy - S + fy).  A frame row is
    // stored as its even-fx half then its odd-fx half, so that the cells of one colour in a row
    // are contiguous.  Threads own pairs (2p, 2p+1) of a row: the frame starts on an odd logical
    // x and every level has an even number of interior cells per dimension, so the two cells of
    // a pair are both interior or both not, and a periodic wrap never falls between them.
    constexpr int FX = TB_X + 2 * S, FY = TB_Y + 2 * S, FN = FX * FY, HX = FX / 2;
    constexpr int RIN = ZERO ? 0 : 1;                 // ring 0 holds the input planes (post)
    constexpr int NIN = (FN + TB_T - 1) / TB_T;       // input cells per thread
    constexpr int F_VALID = 1, F_OWNED = 2, F_PAR = 4, F_LO = 8, F_HI = 16, F_USE = 32;
    __shared__ float ring[RIN + S - 1][3][FN];
    const Grid& g = a.g;
    const int tid = threadIdx.x;
    const int ox = 1 + int(blockIdx.x) * TB_X, oy = 1 + int(blockIdx.y) * TB_Y;
    const int nzi = g.n[2] - 2;
    const int z0 = 1 + int(blockIdx.z) * a.zchunk;
    if (z0 > nzi) return;
    const int z1 = min(z0 + a.zchunk, nzi + 1);
    const int s1 = int(g.s[1]), s2 = int(g.s[2]);
    const float* __restrict__ L0 = a.L;
    const float* __restrict__ L1 = a.L + g.N;
    const float* __restrict__ L2 = a.L + 2 * g.N;

    // pair slots of each half-sweep: frame index of the even cell, grid offset (x, y) of the
    // even cell, flags (valid, owned by this block, (x + y) parity, region edge pairs)
    int sq[S][2], sxy[S][2], sfl[S][2];
#pragma unroll
    for (int s = 0; s < S; ++s) {
        const int hs = S - 1 - s;
        const int plo = (S - hs) / 2, phi = (S + TB_X + hs + 1) / 2;
        const int np = phi - plo, rows = TB_Y + 2 * hs;
#pragma unroll
        for (int k = 0; k < 2; ++k) {
            const int it = tid + k * TB_T;
            sfl[s][k] = 0;
            sq[s][k] = 0;
            sxy[s][k] = 0;
            if (it >= np * rows) continue;
            const int r = it / np, p = plo + (it - r * np);
            const int fy = S - hs + r;
            const int x0 = ox - S + 2 * p, y = oy - S + fy;
            bool okx, oky;
            const int px = tb_wrap(g, 0, x0, okx), py = tb_wrap(g, 1, y, oky);
            int fl = F_USE | (((x0 + y) & 1) ? F_PAR : 0);
            if (okx && oky) fl |= F_VALID;
            if (fy >= S && fy < S + TB_Y && 2 * p >= S && 2 * p < S + TB_X && x0 <= g.n[0] - 2 && y <= g.n[1] - 2)
                fl |= F_OWNED;
            if (2 * p < S - hs) fl |= F_LO;                   // only the odd cell is in the region
            if (2 * p + 1 >= S + TB_X + hs) fl |= F_HI;       // only the even cell is in the region
            sfl[s][k] = fl;
            sq[s][k] = fy * FX + p;
            sxy[s][k] = px + py * s1;
        }
    }
    // input cells of this thread: grid offset (x, y) (-1: outside a wall) and coarse offset
    int ixy[NIN], icxy[NIN];
#pragma unroll
    for (int k = 0; k < NIN; ++k) {
        const int e = tid + k * TB_T;
        ixy[k] = -1;
        icxy[k] = 0;
        if (ZERO || e >= FN) continue;
        const int fy = e / FX, fx = e - fy * FX;
        bool okx, oky;
        const int px = tb_wrap(g, 0, ox - S + fx, okx), py = tb_wrap(g, 1, oy - S + fy, oky);
        if (okx && oky) {
            ixy[k] = px + py * s1;
            icxy[k] = (px + 1) / 2 + ((py + 1) / 2) * int(a.gc.s[1]);
        }
    }

    auto stage_in = [&](int zl) {
        bool okz;
        const int pz = tb_wrap(g, 2, zl, okz);
        float* dst = ring[0][tb_slot(zl)];
        const int cz = ((pz + 1) / 2) * int(a.gc.s[2]);
#pragma unroll
        for (int k = 0; k < NIN; ++k) {
            const int e = tid + k * TB_T;
            if (e >= FN) continue;
            float v = 0.f;
            if (okz && ixy[k] >= 0) {
                v = a.xin[ixy[k] + pz * s2];
                if (a.xc) v += a.xc[icxy[k] + cz];
            }
            const int fy = e / FX, fx = e - fy * FX;
            dst[fy * FX + (fx & 1) * HX + (fx >> 1)] = v;
        }
    };

    const int T0 = z0 - S + 1, T1 = z1 + S - 2;
    if (!ZERO) {
        stage_in(T0 - 1);
        stage_in(T0);
    }
    for (int t = T0; t <= T1; ++t) {
        if (!ZERO) stage_in(t + 1);
        __syncthreads();
#pragma unroll
        for (int s = 0; s < S; ++s) {
            if (t >= T0 + 2 * s) {
                const int zl = t - s;
                const int col = (a.c0 + s) & 1;
                bool okz;
                const int pz = tb_wrap(g, 2, zl, okz);
                const bool own_z = zl >= z0 && zl < z1;
                const int zo = pz * s2;
                float* outp = ZERO ? ring[s < S - 1 ? s : 0][tb_slot(zl)] : ring[s < S - 1 ? s + 1 : 0][tb_slot(zl)];
                const int pin = ZERO ? (s > 0 ? s - 1 : 0) : s;
                const float* pc = ring[pin][tb_slot(zl)];
                const float* pd = ring[pin][tb_slot(zl - 1)];
                const float* pu = ring[pin][tb_slot(zl + 1)];
#pragma unroll
                for (int k = 0; k < 2; ++k) {
                    const int fl = sfl[s][k];
                    if (!(fl & F_USE)) continue;
                    const int e = ((fl & F_PAR ? 1 : 0) + zl + col) & 1;   // which cell of the pair
                    if ((fl & F_LO) && e == 0) continue;
                    if ((fl & F_HI) && e == 1) continue;
                    const int q = sq[s][k] + e * HX;
                    float v = 0.f;
                    if ((fl & F_VALID) && okz) {
                        const int I = sxy[s][k] + e + zo;
                        if (ZERO && s == 0) {
                            v = a.b[I] * a.iD[I];
                        } else {
                            const int qxl = q + (e ? -HX : HX - 1);
                            const float vxl = pc[qxl], vxh = pc[qxl + 1];
                            const float vyl = pc[q - FX], vyh = pc[q + FX];
                            const float vzl = pd[q], vzh = pu[q];
                            float off = L0[I] * vxl + L0[I + 1] * vxh;
                            off += L1[I] * vyl + L1[I + s1] * vyh;
                            off += L2[I] * vzl + L2[I + s2] * vzh;
                            v = (a.b[I] - off) * a.iD[I];
                        }
                        if (s >= S - 2 && (fl & F_OWNED) && own_z) a.xout[I] = v;
                    }
                    if (s < S - 1) outp[q] = v;
                }
            }
            __syncthreads();
        }
    }
}


template <class T, int D>
__global__ void residual_k(Grid g, const T* __restrict__ L, const T* __restrict__ b, const T* __restrict__ xv,
                           T* __restrict__ r) {
    CELL_INTERIOR(g)
    const Nb o = nb_of<D>(g, x, y, z);
    r[I] = b[I] - (off7<D>(g, L, xv, I, o) + diag7<D>(g, L, I) * xv[I]);
}

// residual of the (at most 2^D) fine children of each coarse cell, summed straight into the coarse
// right-hand side (no fine residual array); diag: the level's diagonal, read in FP64 only (7 multiply-adds a cell
// instead of 17 FP64 operations)
template <class T, int D, class TL = T, bool REG = true>
__global__ void resid_restrict_k(Grid gc, int yc0, int yc1, Grid gf, const TL* __restrict__ L,
                                 const T* __restrict__ diag, const T* __restrict__ b, const T* __restrict__ xv, T* __restrict__ bc) {
    int xc, yc;
    plane_cell<T>(gc.n[0] - 2, xc, yc);
    xc += 1;
    yc += yc0;   // coarse rows [yc0, yc1)
    const int zc = D == 3 ? 1 + int(blockIdx.z) : 0;
    if (xc > gc.n[0] - 2 || yc >= yc1) return;
    const int s1 = int(gf.s[1]), s2 = int(gf.s[2]);
    T sum = T(0);
    const int fx = REG ? 2 * xc - 1 : mg_child(gc, 0, xc), fy = REG ? 2 * yc - 1 : mg_child(gc, 1, yc);
    const int fz = D == 3 ? (REG ? 2 * zc - 1 : mg_child(gc, 2, zc)) : 0;
    const int mx = REG ? 2 : mg_children(gc, 0, xc), my = REG ? 2 : mg_children(gc, 1, yc);
    const int mz = D == 3 ? (REG ? 2 : mg_children(gc, 2, zc)) : 1;
    for (int k = 0; k < mz; ++k)
        for (int j = 0; j < my; ++j)
            for (int i = 0; i < mx; ++i) {
                const int x = fx + i, y = fy + j, z = fz + k;
                const int I = x + y * s1 + z * s2;
                const Nb o = nb_of<D>(gf, x, y, z);
                if constexpr (sizeof(T) == 8) sum += resid7<D>(gf, L, fma(-diag[I], xv[I], b[I]), xv, I, o);
                else sum += b[I] - (off7<D>(gf, L, xv, I, o) + diag7<D>(gf, L, I) * xv[I]);
            }
    bc[xc + yc * int(gc.s[1]) + zc * int(gc.s[2])] = sum;
}

template <class T>
__global__ void prolong_k(Grid gf, Grid gc, const T* __restrict__ xc, T* __restrict__ xf) {
    const Grid& g = gf;
    INTERIOR_XYZ
    xf[I] += xc[mg_parent_cell<false>(gc, c[0], c[1], c[2])];
}

// The small levels of the V-cycle in one launch: a single block runs the whole cycle below (and on) the first
// level of at most tail_pairs<T>() pairs of cells, with a block barrier between the stages.  The stages are those of
// the levels above (relaxed red-black half-sweeps from zero, residual restriction, prolongation); the coarsest level
// is solved by nuc symmetric sweeps on its mean-free right-hand side (a colour swept twice in a row keeps its
// values, so those sweeps are skipped).
// Shared memory holds, for each level, x on the ghost-padded grid, and by pairs of x-neighbours (thread t of the
// level has pair t, its red and its black cell) the right-hand side, the 2D face coefficients and the inverse
// diagonal, and the cells' indices.  Ghosts across a periodic wrap are kept as copies by the thread that writes their
// cell, so that a cell's neighbours lie at the same distances everywhere.
// What bounds it: latency, a chain of about 40 stages of 0.4 us, where a launch of its own takes 2 to 3 us.
// A level's sizes are kept in registers (keep): read from the kernel's parameters, which the compiler otherwise does
// again in every stage, they cost more than the stage's arithmetic (1000 cycles a stage, of which 130 the update).
constexpr int TAIL_MAX = 16, TAIL_THREADS = 1024, TAIL_PAIRS = 2, TAIL_WORDS = 4;
// v, as a value that the compiler can only keep
__device__ __forceinline__ int keep(int v) {
    asm volatile("" : "+r"(v));
    return v;
}
template <class T>
__device__ __forceinline__ T* keep(T* v) {
    asm volatile("" : "+l"(v));
    return v;
}
template <class T>
struct TailArgs {
    int nl;                                          // levels; 0 is the largest
    Grid g[TAIL_MAX];
    const T* L[TAIL_MAX];
    const T* iD[TAIL_MAX];
    int np[TAIL_MAX];                                // pairs
    int xo[TAIL_MAX], bo[TAIL_MAX], co[TAIL_MAX];    // x, right-hand side, coefficients (offsets in values)
    int io[TAIL_MAX];                                // TAIL_WORDS a pair (offset in words behind the values)
    int ro, values, words;                           // residual scratch; sizes in all
    int nu1[TAIL_MAX], nu2[TAIL_MAX];
    int nuc;
    T omega;
    const T* b;                                      // right-hand side and result of level 0
    T* x;
    size_t bytes() const { return sizeof(T) * (size_t)values + 4 * (size_t)words; }
};
// flags of a cell: copies to keep at x + n, x - n, y + n, ... (bits 0-5); its wrap_class (bits 6-8); two children
// along x, y, z (bits 9-11)
template <int D>
__device__ __forceinline__ unsigned tail_flags(const Grid& g, int conflicts, int x, int y, int z) {
    const int c[3] = {x, y, z};
    unsigned f = unsigned(wrap_class(g, conflicts, x, y, z)) << 6;
#pragma unroll
    for (int e = 0; e < D; ++e) {
        if (g.isper(e)) f |= (c[e] == 1 ? 1u << 2 * e : 0u) | (c[e] == g.n[e] - 2 ? 2u << 2 * e : 0u);
        if (c[e] <= g.pr[e]) f |= 512u << e;
    }
    return f;
}
// distances to the copies across the wraps
struct Wraps {
    int w0, w1, w2;
    __device__ Wraps(const Grid& g) : w0(keep(g.n[0] - 2)), w1(keep((g.n[1] - 2) * int(g.s[1]))), w2(keep((g.n[2] - 2) * int(g.s[2]))) {}
};
template <class T, int D>
__device__ __forceinline__ void tail_store(const Wraps& w, T* x, int I, unsigned f, T v) {
    x[I] = v;
    if (f & 63u) {
        if (f & 1u) x[I + w.w0] = v;
        if (f & 2u) x[I - w.w0] = v;
        if (f & 4u) x[I + w.w1] = v;
        if (f & 8u) x[I - w.w1] = v;
        if (D == 3) {
            if (f & 16u) x[I + w.w2] = v;
            if (f & 32u) x[I - w.w2] = v;
        }
    }
}
template <int D>
__device__ __forceinline__ void tail_pair(const Grid& g, int t, int& x, int& y, int& z) {
    const int hx = (g.n[0] - 1) / 2, ny = g.n[1] - 2, r = t / hx, rz = r / ny;
    x = 1 + 2 * (t - r * hx);
    y = 1 + r - rz * ny;
    z = D == 3 ? 1 + rz : 0;
}
// Pair t of level g in TAIL_WORDS words at w (with a stride): its first cell with bit 30 when that is the red one and
// bit 31 when there is a second; the flags of both (16 bits each); their parents on gc; the first child of the first
// cell on gf (that of the second lies 2 on, or 1 behind a single child).  gc, gf: null where there is no such level.
template <int D>
__device__ __forceinline__ void tail_words(const Grid& g, const Grid* gc, const Grid* gf, int t, unsigned* w, int step) {
    int x, y, z;
    tail_pair<D>(g, t, x, y, z);
    const int conflicts = wrap_conflicts(g);
    const bool two = x < g.n[0] - 2;
    w[0] = unsigned(x + y * int(g.s[1]) + z * int(g.s[2])) | (((x + y + z) & 1) ? 0u : 1u << 30) | (two ? 1u << 31 : 0u);
    w[step] = tail_flags<D>(g, conflicts, x, y, z) | (two ? tail_flags<D>(g, conflicts, x + 1, y, z) << 16 : 0u);
    w[2 * step] = gc ? unsigned(mg_parent_cell<false>(*gc, x, y, z)) | (two ? unsigned(mg_parent_cell<false>(*gc, x + 1, y, z)) << 16 : 0u) : 0u;
    w[3 * step] = gf ? unsigned(lin(*gf, mg_child(g, 0, x), mg_child(g, 1, y), D == 3 ? mg_child(g, 2, z) : 0)) : 0u;
}
// the words by colour: cells (0: none), flags, parents (red in the low half words)
struct PairCells {
    unsigned red = 0, black = 0, fl = 0;
    bool swap = false;   // the first cell is black
    __device__ PairCells() {}
    __device__ PairCells(unsigned w0, unsigned w1) {
        const unsigned I = w0 & 0x3FFFFFFFu, J = w0 >> 31 ? I + 1 : 0u;
        swap = !(w0 >> 30 & 1u);
        red = swap ? J : I;
        black = swap ? I : J;
        fl = order(w1);
    }
    __device__ unsigned order(unsigned v) const { return swap ? v >> 16 | v << 16 : v; }
};
// Σ of the children of a coarse cell with flags f, the first at r
template <class T, int D>
__device__ __forceinline__ T tail_children(const T* r, unsigned f, int s1, int s2) {
    const bool bx = f & 512u, by = f & 1024u, bz = D == 3 && (f & 2048u);
    T v[8];
#pragma unroll
    for (int q = 0; q < (D == 3 ? 8 : 4); ++q) {
        const bool in = (!(q & 1) || bx) && (!(q & 2) || by) && (!(q & 4) || bz);
        v[q] = in ? r[(q & 1 ? 1 : 0) + (q & 2 ? s1 : 0) + (q & 4 ? s2 : 0)] : T(0);
    }
    T sum = v[0];
#pragma unroll
    for (int q = 1; q < (D == 3 ? 8 : 4); ++q) sum += v[q];
    return sum;
}

// coefficients and cell words of every level into shared memory
template <class T, int D>
__device__ void tail_setup(const TailArgs<T>& a, T* sm) {
    const int tid = threadIdx.x;
    unsigned* w = reinterpret_cast<unsigned*>(sm + a.values);
    for (int k = 0; k < a.nl; ++k) {
        const Grid& g = a.g[k];
        const int np = keep(a.np[k]), N = keep(int(g.N)), s1 = keep(int(g.s[1])), s2 = keep(int(g.s[2])), co = keep(a.co[k]), io = keep(a.io[k]);
        const T* __restrict__ L0 = keep(a.L[k]);
        const T* __restrict__ iD = keep(a.iD[k]);
        for (int t = tid; t < np; t += TAIL_THREADS) {
            tail_words<D>(g, k + 1 < a.nl ? &a.g[k + 1] : nullptr, k > 0 ? &a.g[k - 1] : nullptr, t, w + io + t, np);
            const PairCells pc(w[io + t], 0u);
#pragma unroll
            for (int c = 0; c < 2; ++c) {
                const int I = c ? pc.black : pc.red;
                const T* L = L0 + I;
                T v[7] = {};
                if (I) {
                    v[0] = __ldg(L);
                    v[1] = __ldg(L + 1);
                    v[2] = __ldg(L + N);
                    v[3] = __ldg(L + N + s1);
                    v[4] = __ldg(iD + I);
                    if (D == 3) {
                        v[5] = __ldg(L + 2 * N);
                        v[6] = __ldg(L + 2 * N + s2);
                    }
                }
#pragma unroll
                for (int q = 0; q < 2 * D + 1; ++q) sm[co + (2 * q + c) * np + t] = v[q];
            }
        }
    }
}

// one V-cycle on the levels (after tail_setup); mean_s: shared
template <class T, int D>
__device__ __forceinline__ void tail_cycle(const TailArgs<T>& a, T* sm, T& mean_s) {
    const int tid = threadIdx.x, last = keep(a.nl) - 1;
    const unsigned* w = reinterpret_cast<const unsigned*>(sm + keep(a.values));
    T* scratch = sm + keep(a.ro);
    // A visit of a level: nh half-sweeps x += om (x_GS - x) of alternating colours from color0 on.
    //  mode 0: from x = 0 (nh >= 1), then the restriction of the residual into the next level's right-hand side
    //  mode 1: after x += P(x of the next level)
    //  mode 2: the coarsest level, from x = 0
    auto visit = [&](int l, int nh, int color0, T om, int mode) {
        const Grid& g = a.g[l];
        const int np = keep(a.np[l]), s1 = keep(int(g.s[1])), s2 = keep(int(g.s[2])), conflicts = keep(wrap_conflicts(g));
        const int bo = keep(a.bo[l]), co = keep(a.co[l]), step = 2 * np;
        const Wraps wr(g);
        T* x = sm + keep(a.xo[l]);
        const unsigned* id = w + keep(a.io[l]);
        PairCells pc[TAIL_PAIRS];
#pragma unroll
        for (int k = 0; k < TAIL_PAIRS; ++k) {
            const int t = tid + k * TAIL_THREADS;
            if (t < np) pc[k] = PairCells(id[t], id[np + t]);
        }
        // b - Σ c x_nb of cell I, coefficients at c; Σ c when asked for
        auto gather = [&](int c, int I, T r, T* dd) {
            const T c0 = sm[c], c1 = sm[c + step], c2 = sm[c + 2 * step], c3 = sm[c + 3 * step];
            const T x0 = x[I - 1], x1 = x[I + 1], x2 = x[I - s1], x3 = x[I + s1];
            T c4 = T(0), c5 = T(0), x4 = T(0), x5 = T(0);
            if (D == 3) {
                c4 = sm[c + 5 * step];
                c5 = sm[c + 6 * step];
                x4 = x[I - s2];
                x5 = x[I + s2];
            }
            if (dd) *dd = (c0 + c1) + (c2 + c3) + (c4 + c5);
            r = fma(-c0, x0, r);
            r = fma(-c1, x1, r);
            r = fma(-c2, x2, r);
            r = fma(-c3, x3, r);
            if (D == 3) {
                r = fma(-c4, x4, r);
                r = fma(-c5, x5, r);
            }
            return r;
        };
        if (mode == 1) {
            const T* xc = sm + keep(a.xo[l + 1]);
#pragma unroll
            for (int k = 0; k < TAIL_PAIRS; ++k) {
                const int t = tid + k * TAIL_THREADS;
                if (t >= np) continue;
                const unsigned par = pc[k].order(id[2 * np + t]);
                const int r = pc[k].red, b = pc[k].black;
                const T vr = r ? x[r] + xc[par & 0xFFFFu] : T(0), vb = b ? x[b] + xc[par >> 16] : T(0);
                if (r) tail_store<T, D>(wr, x, r, pc[k].fl & 0xFFFFu, vr);
                if (b) tail_store<T, D>(wr, x, b, pc[k].fl >> 16, vb);
            }
            __syncthreads();
        }
        for (int s = 0; s < nh; ++s) {
            const int color = (color0 + s) & 1, sh = 16 * color;
            for (int cls = 0; cls <= conflicts; ++cls) {
                if (cls & ~conflicts) continue;
                // the operands of every pair are read before the first store
                T nv[TAIL_PAIRS];
#pragma unroll
                for (int k = 0; k < TAIL_PAIRS; ++k) {
                    const int t = tid + k * TAIL_THREADS, I = color ? pc[k].black : pc[k].red;
                    if (!I) continue;
                    const int c = co + color * np + t;
                    const T xo = x[I], d = sm[c + 4 * step], r = gather(c, I, sm[bo + color * np + t], nullptr);
                    nv[k] = om == T(1) ? r * d : fma(om, fma(r, d, -xo), xo);
                }
#pragma unroll
                for (int k = 0; k < TAIL_PAIRS; ++k) {
                    const int I = color ? pc[k].black : pc[k].red;
                    const unsigned f = pc[k].fl >> sh & 0xFFFFu;
                    if (I && int(f >> 6 & 7u) == cls) tail_store<T, D>(wr, x, I, f, nv[k]);
                }
                __syncthreads();
            }
        }
        if (mode != 0) return;
#pragma unroll
        for (int k = 0; k < TAIL_PAIRS; ++k)
#pragma unroll
            for (int c = 0; c < 2; ++c) {
                const int t = tid + k * TAIL_THREADS, I = c ? pc[k].black : pc[k].red;
                if (!I) continue;
                T dd;
                const T r = gather(co + c * np + t, I, sm[bo + c * np + t], &dd);
                scratch[I] = fma(dd, x[I], r);
            }
        __syncthreads();
        const int npc = keep(a.np[l + 1]), bc = keep(a.bo[l + 1]), ic = keep(a.io[l + 1]);
        for (int t = tid; t < npc; t += TAIL_THREADS) {
            const unsigned w0 = w[ic + t], f = w[ic + npc + t];
            const T* r = scratch + w[ic + 3 * npc + t];
            const int first = bc + (w0 >> 30 & 1u ? 0 : npc) + t, second = bc + (w0 >> 30 & 1u ? npc : 0) + t;   // slots
            sm[first] = tail_children<T, D>(r, f & 0xFFFFu, s1, s2);
            if (w0 >> 31) sm[second] = tail_children<T, D>(r + (f & 512u ? 2 : 1), f >> 16, s1, s2);
        }
        __syncthreads();
    };
    // level 0's right-hand side; x = 0 everywhere, and the right-hand sides of no cell
    {
        const int np = keep(a.np[0]), bo = keep(a.bo[0]);
        const unsigned* id = w + keep(a.io[0]);
        const T* b = keep(a.b);
        for (int t = tid; t < np; t += TAIL_THREADS) {
            const PairCells pc(id[t], 0u);
            const T r = pc.red ? b[pc.red] : T(0), k = pc.black ? b[pc.black] : T(0);
            sm[bo + t] = r;
            sm[bo + np + t] = k;
        }
    }
    for (int k = 0; k <= last; ++k) {
        const int n = keep(int(a.g[k].N)), xo = keep(a.xo[k]);
        for (int q = tid; q < n; q += TAIL_THREADS) sm[xo + q] = T(0);
    }
    {
        const int np = keep(a.np[last]), bo = keep(a.bo[last]);
        if (last > 0)
            for (int t = tid; t < 2 * np; t += TAIL_THREADS) sm[bo + t] = T(0);
    }
    __syncthreads();
    for (int l = 0; l < last; ++l) visit(l, 2 * keep(a.nu1[l]), 0, a.omega, 0);
    {
        const Grid& g = a.g[last];
        const int np = keep(a.np[last]), bo = keep(a.bo[last]);
        const unsigned* id = w + keep(a.io[last]);
        // FP64 sum by one warp (the slots of no cell are zero): an FP64 instruction occupies the pipe for 16 cycles
        // a warp, whatever its lanes do
        if (tid < 32) {
            double acc = 0.0;
            for (int q = tid; q < 2 * np; q += 32) acc += double(sm[bo + q]);
            for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
            if (tid == 0) mean_s = T(acc / double((g.n[0] - 2) * (g.n[1] - 2) * (D == 3 ? g.n[2] - 2 : 1)));
        }
        __syncthreads();
        const T mean = mean_s;
        for (int t = tid; t < np; t += TAIL_THREADS) {
            const PairCells pc(id[t], 0u);
            if (pc.red) sm[bo + t] -= mean;
            if (pc.black) sm[bo + np + t] -= mean;
        }
        __syncthreads();
        // R B, B R, R B, ...: a colour following itself changes nothing
        visit(last, keep(a.nuc) + 1, 0, T(1), 2);
    }
    for (int l = last - 1; l >= 0; --l) visit(l, 2 * keep(a.nu2[l]), 1, a.omega, 1);
    // the result (its ghost entries stay zero)
    {
        const int np = keep(a.np[0]), xo = keep(a.xo[0]);
        const unsigned* id = w + keep(a.io[0]);
        T* x = keep(a.x);
        for (int t = tid; t < np; t += TAIL_THREADS) {
            const int I = id[t] & 0x3FFFFFFFu;
            x[I] = sm[xo + I];
            if (id[t] >> 31) x[I + 1] = sm[xo + I + 1];
        }
    }
}
template <class T, int D>
__global__ void __launch_bounds__(TAIL_THREADS) mg_tail_k(const __grid_constant__ TailArgs<T> a) {
    extern __shared__ __align__(16) unsigned char tail_raw[];
    __shared__ T mean_s;
    T* sm = reinterpret_cast<T*>(tail_raw);
    tail_setup<T, D>(a, sm);
    __syncthreads();
    tail_cycle<T, D>(a, sm, mean_s);
}

// Pairs of cells in the largest level that the one-block kernel takes.  FP32: TAIL_PAIRS for each thread (16^3
// cells).  FP64: 256, since a multiprocessor issues FP64 at 1/64 of the FP32 rate and a half-sweep on more cells is
// faster spread over the device.
template <class T> constexpr long long tail_pairs() { return sizeof(T) == 4 ? TAIL_PAIRS * TAIL_THREADS : 256; }

// ---- the one-launch solver of small grids (poisson_cluster.cuh)
// Interior cells up to which it is used, and pairs of cells of its tail's largest level.  Measured on GB300, a step
// with the multi-launch solver and on this path: FP32 (mixed) 41x35x30 4.3 and 2.8 ms, 32x64x32 4.9 and 4.2 ms.  The FP64
// limit is from before x lay in shared memory in 2D and the iteration in one cluster (128x64 2.4 and 2.6 ms then; 16
// multiprocessors have a tenth of the device's FP64 pipes) and is low by now: 128x64 2.32 and 2.15 ms, 128x128 2.50 and
// 2.27, 192x128 2.20 and 2.25, 256x192 2.91 and 3.36; 24x20x16 3.16 and 2.41, 32x32x16 3.72 and 2.95.
template <class T> constexpr long long cluster_cells() { return sizeof(T) == 4 ? 65536 : 4096; }
constexpr int CL_ITERATIONS = 2000;   // a launch: up to 0.3 s
template <class T> constexpr long long cluster_tail_pairs() { return sizeof(T) == 4 ? 512 : 128; }

// ------------------------------------------------------------------ Krylov kernels
// Row loops: a block takes whole x-rows of interior cells (rows dealt round-robin over a
// grid of at most KBLOCKS blocks), so the reductions end in one warp-shuffle block sum per
// block and the cross-block sums read only gridDim.x partials.
constexpr int KTHREADS = 256;
constexpr int KBLOCKS = 1216;   // 8 blocks on each of 152 SMs

// Row loops: block b takes rows b, b + G, b + 2G, ... (G blocks) of the interior; the row's
// (y, z) advance incrementally (a grid holds < 2^31 cells, so 32-bit row numbers suffice)
#define ROWS_FOR(g, DD)                                                                              \
    const int nxi_ = (g).n[0] - 2, nyi_ = (g).n[1] - 2;                                              \
    const int nrows_ = nyi_ * ((DD) == 3 ? (g).n[2] - 2 : 1);                                        \
    const int dy_ = int(gridDim.x) % nyi_, dz_ = int(gridDim.x) / nyi_;                              \
    int y = 1 + int(blockIdx.x) % nyi_, z = ((DD) == 3 ? 1 : 0) + int(blockIdx.x) / nyi_;           \
    for (int rw_ = blockIdx.x; rw_ < nrows_;                                                         \
         rw_ += gridDim.x, y += dy_, z += dz_ + (y > nyi_ ? 1 : 0), y -= (y > nyi_ ? nyi_ : 0))
#define ROWS_BEGIN(g)                                                                      \
    {                                                                                      \
        ROWS_FOR(g, (g).D) {                                                               \
            for (int x = 1 + threadIdx.x; x <= nxi_; x += blockDim.x) {                    \
                [[maybe_unused]] const int c[3] = {x, y, z};                               \
                const long long I = lin(g, x, y, z);
#define ROWS_END \
    }            \
    }            \
    }

// the same with a 32-bit cell index and the dimension fixed at compile time
#define ROWS_BEGIN_D(g)                                                                    \
    {                                                                                      \
        const int s1_ = int((g).s[1]), s2_ = int((g).s[2]);                                \
        ROWS_FOR(g, D) {                                                                   \
            const int row_ = y * s1_ + z * s2_;                                            \
            for (int x = 1 + threadIdx.x; x <= nxi_; x += blockDim.x) {                    \
                const int I = row_ + x;

// Blocks of the whole-array vector kernels: two float4 a thread on small grids (every further block only adds a partial
// to the last block's sum), on large ones as many as are resident at once (update32_k and dot2_32_k at 128x192x160:
// 12.1 and 14.3 us with 4 an SM, 12.8 and 20.0 with 8, of which 6 and 4 were resident; 8 of 32 registers 17.3 and 19.7).
constexpr int VB_RESIDENT = 4;
inline int vblocks(const Grid& g, int nsm) {
    const long long b = (g.N / 4 + 2 * KTHREADS - 1) / (2 * KTHREADS);
    return int(std::max<long long>(1, std::min<long long>(b, std::min(VB_RESIDENT * std::max(nsm, 1), KBLOCKS))));
}
inline int kblocks(const Grid& g) {
    const long long rows = (long long)(g.n[1] - 2) * (g.D == 3 ? g.n[2] - 2 : 1);
    return int(rows < KBLOCKS ? rows : KBLOCKS);
}

__device__ __forceinline__ double warp_sum(double v) {
    for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
    return v;
}
__device__ __forceinline__ unsigned long long warp_max(unsigned long long v) {
    for (int o = 16; o > 0; o >>= 1) {
        const unsigned long long w = __shfl_down_sync(0xffffffffu, v, o);
        v = w > v ? w : v;
    }
    return v;
}
// block sums of a and b, valid in thread 0 (fixed order: deterministic)
__device__ __forceinline__ void block_sum2(double& a, double& b) {
    __shared__ double sa[32], sb[32];
    a = warp_sum(a);
    b = warp_sum(b);
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    if (lane == 0) {
        sa[w] = a;
        sb[w] = b;
    }
    __syncthreads();
    if (w == 0) {
        const int nw = blockDim.x >> 5;
        a = warp_sum(lane < nw ? sa[lane] : 0.0);
        b = warp_sum(lane < nw ? sb[lane] : 0.0);
    }
}
__device__ __forceinline__ unsigned long long block_max(unsigned long long m) {
    __shared__ unsigned long long sm[32];
    m = warp_max(m);
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    if (lane == 0) sm[w] = m;
    __syncthreads();
    if (w == 0) m = warp_max(lane < (int)(blockDim.x >> 5) ? sm[lane] : 0ull);
    return m;
}

// diagonal D_I = -Σ_i (L[I,i] + L[I+δi,i]) of the FP64 operator
__device__ __forceinline__ double diag_of(const Grid& g, const double* L, long long I) {
    double dd = 0.0;
    for (int i = 0; i < g.D; ++i) dd -= L[I + i * g.N] + L[I + g.s[i] + i * g.N];
    return dd;
}
// diag_of (same sums, same order) out of line, with scalar arguments, for kernels whose common path
// must not carry its FP64 additions (inlined in a branch of pure arithmetic, the compiler if-converts
// it into every thread)
template <int D>
__device__ __noinline__ double diag_of_cold(const double* L, long long I, long long s1, long long s2, long long N) {
    double dd = 0.0;
    dd -= L[I] + L[I + 1];
    dd -= L[I + N] + L[I + s1 + N];
    if (D == 3) dd -= L[I + 2 * N] + L[I + s2 + 2 * N];
    return dd;
}

__global__ void set_diag64_k(Grid g, const double* __restrict__ L, double* __restrict__ diag) {
    ROWS_BEGIN(g)
    diag[I] = diag_of(g, L, I);
    ROWS_END
}

// Finest-level set-up of the mixed solver in one pass over the FP64 face coefficients L (one
// thread per cell of the ghost-inclusive grid):
//  - the FP32 copy L32 of every coefficient (and its FP16 copy L16, when given), = float(L);
//  - on interior cells the FP64 diagonal D_I = -Σ_i (L[I,i] + L[I+δi,i]) in diag_of's order, and the
//    FP32 inverse diagonal of the FP32 copy with set_diag_k's sums and zero rule.
// Where the 2D coefficients of a cell are bit-identical (pure-phase cells away from walls), the
// FP64 sum ((0 - 2a) - 2a) - 2a (3D; (0 - 2a) - 2a in 2D) is exactly fma(-2D, a, 0): the partial
// sums are exact multiples of a and only the last one rounds, as the fma does; both give +0 for a = ±0.
template <int D>
__global__ void setup_fine_k(Grid g, const double* __restrict__ L, double* __restrict__ diag,
                             float* __restrict__ L32, __half* __restrict__ L16, float* __restrict__ iD32) {
    const int x = blockIdx.x * blockDim.x + threadIdx.x, y = blockIdx.y * blockDim.y + threadIdx.y;
    const int z = D == 3 ? int(blockIdx.z) : 0;
    if (x >= g.n[0] || y >= g.n[1]) return;
    const long long I = lin(g, x, y, z);
    double a[D];
    float fa[D];
#pragma unroll
    for (int i = 0; i < D; ++i) {
        a[i] = L[I + i * g.N];
        fa[i] = f32_rn(a[i]);
        L32[I + i * g.N] = fa[i];
        if (L16) L16[I + i * g.N] = __float2half_rn(fa[i]);
    }
    if (x < 1 || y < 1 || x > g.n[0] - 2 || y > g.n[1] - 2) return;
    if (D == 3 && (z < 1 || z > g.n[2] - 2)) return;
    double b[D];
    bool same = true;
    const unsigned long long a0 = (unsigned long long)__double_as_longlong(a[0]);
#pragma unroll
    for (int i = 0; i < D; ++i) {
        b[i] = L[I + g.s[i] + i * g.N];
        same = same && (unsigned long long)__double_as_longlong(a[i]) == a0 &&
               (unsigned long long)__double_as_longlong(b[i]) == a0;
    }
    diag[I] = same ? fma(-2.0 * D, a[0], 0.0) : diag_of_cold<D>(L, I, g.s[1], g.s[2], g.N);
    float df = 0.0f;
#pragma unroll
    for (int i = 0; i < D; ++i) df -= fa[i] + f32_rn(b[i]);
    const float eps = 1.1920929e-7f;
    iD32[I] = (df * df < 2.0f * eps) ? 0.0f : 1.0f / df;
}

// z planes per block of the tiled stencil kernels: 8, and 1 where 8 would leave fewer than two blocks for a
// multiprocessor (a thread's planes are then a chain of loads on an idle device)
constexpr int MV_ZT = 8;
inline int mv_planes(const Grid& g, int nsm) {
    const long long tiles = ((g.n[0] - 2 + 31) / 32) * (long long)((g.n[1] - 2 + 7) / 8);
    return g.D == 3 && tiles * ((g.n[2] - 2 + MV_ZT - 1) / MV_ZT) < 2ll * nsm ? 1 : MV_ZT;
}
inline dim3 mv_tile_grid(const Grid& g, int zt) {
    return dim3((g.n[0] - 2 + 31) / 32, (g.n[1] - 2 + 7) / 8, g.D == 3 ? (g.n[2] - 2 + zt - 1) / zt : 1);
}
// launch K<D, planes per block> for the grid's dimension and the solver's tile depth
#define LAUNCH_TILE(gg, K, ...)                                                                      \
    do {                                                                                             \
        const dim3 tg_ = mv_tile_grid(gg, mg->zt);                                                   \
        if ((gg).D == 2) K<2, MV_ZT><<<tg_, KTHREADS, 0, st>>>(__VA_ARGS__);                         \
        else if (mg->zt == 1) K<3, 1><<<tg_, KTHREADS, 0, st>>>(__VA_ARGS__);                        \
        else K<3, MV_ZT><<<tg_, KTHREADS, 0, st>>>(__VA_ARGS__);                                     \
        ia::note_launch();                                                                           \
    } while (0)

// z_I - D_I x_I - Σ L x_nb as one FMA chain: 2D + 1 FP64 operations where pairwise sums take 3D + 1
// (the residual kernels are bound by the FP64 pipe)
template <int D>
__device__ __forceinline__ double resid_cell(const Grid& g, const double* __restrict__ L, double dd,
                                             const double* __restrict__ zz, const double* __restrict__ xv, int I,
                                             const Nb& o) {
    const int s1 = int(g.s[1]), s2 = int(g.s[2]);
    const double* L1 = L + g.N;
    double v = fma(-dd, xv[I], zz[I]);
    v = fma(-L[I], xv[I + o.xl], v);
    v = fma(-L[I + 1], xv[I + o.xh], v);
    v = fma(-L1[I], xv[I + o.yl], v);
    v = fma(-L1[I + s1], xv[I + o.yh], v);
    if (D == 3) {
        const double* L2 = L1 + g.N;
        v = fma(-L2[I], xv[I + o.zl], v);
        v = fma(-L2[I + s2], xv[I + o.zh], v);
    }
    return v;
}

// r = z - A x over interior cells, L∞(r) into *linf (zeroed by the caller); diag precomputed (or NULL:
// from L).  Row loop over a grid of at most KBLOCKS blocks (no per-block scratch).
template <int D>
__global__ void true_resid_k(Grid g, const double* __restrict__ L, const double* __restrict__ diag,
                             const double* __restrict__ zz, const double* __restrict__ xv, double* __restrict__ r,
                             unsigned long long* linf) {
    unsigned long long m = 0ull;
    ROWS_BEGIN_D(g)
    const Nb o = nb_of<D>(g, x, y, z);
    const double v = resid_cell<D>(g, L, diag ? diag[I] : diag7<D>(g, L, I), zz, xv, I, o);
    r[I] = v;
    const unsigned long long b = abs_bits(v);
    m = b > m ? b : m;
    ROWS_END
    m = block_max(m);
    if (threadIdx.x == 0) atomicMax(linf, m);
}

// The same on the x-y tiles of matvec32_tile_k (32 x 8 cells, MV_ZT z planes per block of 256 threads) with
// the precomputed diagonal; each block's L∞ (as the bit pattern of |r|) into pmax[block], reduced by
// finalize_max_k.
// With r32 given, also the next inner solve's start: r32 = float(r) (integer rounding, no FP64-pipe
// conversion in this FP64-bound kernel) and e32 = 0 on the same interior cells (their ghost entries stay
// zero from the allocation: the whole-array vector updates only ever add zero there).
template <int D, int ZT>
__global__ void __launch_bounds__(256) true_resid_tile_k(Grid g, const double* __restrict__ L,
                                                         const double* __restrict__ diag,
                                                         const double* __restrict__ zz,
                                                         const double* __restrict__ xv, double* __restrict__ r,
                                                         unsigned long long* __restrict__ pmax,
                                                         float* __restrict__ r32, float* __restrict__ e32) {
    const int x = 1 + int(blockIdx.x) * 32 + int(threadIdx.x & 31), y = 1 + int(blockIdx.y) * 8 + int(threadIdx.x >> 5);
    const int z0 = D == 3 ? 1 + ZT * int(blockIdx.z) : 0;
    unsigned long long m = 0ull;
    auto cell = [&](int z) {
        const int I = x + y * int(g.s[1]) + z * int(g.s[2]);
        const Nb o = nb_of<D>(g, x, y, z);
        const double v = resid_cell<D>(g, L, diag[I], zz, xv, I, o);
        r[I] = v;
        if (r32) {
            r32[I] = f32_rn(v);
            e32[I] = 0.f;
        }
        const unsigned long long b = abs_bits(v);
        m = b > m ? b : m;
    };
    if (x <= g.n[0] - 2 && y <= g.n[1] - 2) {
        if (D == 3 && z0 + ZT - 1 <= g.n[2] - 2) {
#pragma unroll
            for (int k = 0; k < ZT; ++k) cell(z0 + k);   // a full tile (see matvec32_tile_k)
        } else {
            for (int k = 0; k < (D == 3 ? ZT : 1); ++k) {
                if (D == 3 && z0 + k > g.n[2] - 2) break;
                cell(z0 + k);
            }
        }
    }
    m = block_max(m);
    if (threadIdx.x == 0) pmax[blockIdx.x + gridDim.x * (blockIdx.y + gridDim.y * blockIdx.z)] = m;
}
__global__ void finalize_max_k(const unsigned long long* __restrict__ pmax, long long n, unsigned long long* out) {
    unsigned long long m = 0ull;
    for (long long i = threadIdx.x; i < n; i += blockDim.x) m = pmax[i] > m ? pmax[i] : m;
    m = block_max(m);
    if (threadIdx.x == 0) *out = m;
}

// fixed-order sum of `n` partials for `k` quantities → out[0..k)
// Σ partial[qd·n + i] over i in a fixed order, valid in thread 0 (a block of 1024 threads)
__device__ double finalize_sum(const double* __restrict__ partial, long long n, int qd) {
    __shared__ double sm[1024];
    double acc = 0.0;
    for (long long i = threadIdx.x; i < n; i += blockDim.x) acc += partial[qd * n + i];
    sm[threadIdx.x] = acc;
    __syncthreads();
    for (int w = blockDim.x / 2; w > 0; w >>= 1) {
        if (threadIdx.x < w) sm[threadIdx.x] += sm[threadIdx.x + w];
        __syncthreads();
    }
    const double v = sm[0];
    __syncthreads();
    return v;
}
__global__ void finalize_k(const double* __restrict__ partial, long long n, int k, double* out) {
    for (int qd = 0; qd < k; ++qd) {
        const double v = finalize_sum(partial, n, qd);
        if (threadIdx.x == 0) out[qd] = v;
    }
}
// Σ p[i] and Σ q[i] over n partials by one block of 256 threads in a fixed order, valid in thread 0: strands of
// 256, a shuffle tree in each warp, then the eight warp sums by the first thread.  One barrier instead of the ten
// of a tree over shared memory: with few partials the barriers were most of the reduction's tail.
// Out of line: only the last block of a reduction calls it, and inlined it would raise the streaming
// loop's register count.
__device__ __noinline__ void sum2_by256(const double* p, const double* q, long long n, double& sp, double& sq) {
    __shared__ double wp[8], wq[8];
    double a = 0.0, b = 0.0;
#pragma unroll 4
    for (long long i = threadIdx.x; i < n; i += 256) {
        a += __ldcg(p + i);
        if (q) b += __ldcg(q + i);
    }
    a = warp_sum(a);
    if (q) b = warp_sum(b);
    if ((threadIdx.x & 31) == 0) {
        wp[threadIdx.x >> 5] = a;
        wq[threadIdx.x >> 5] = b;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        for (int w = 1; w < 8; ++w) {
            a += wp[w];
            if (q) b += wq[w];
        }
        sp = a;
        sq = b;
    }
}
// After thread 0 of every block has written the block's partials: true in the last block to finish,
// which then sees every partial (each block's write is fenced before its count); the counter is reset
// for the next launch by that block.
__device__ bool last_block(unsigned int* done, unsigned int nblocks) {
    __shared__ bool am_last;
    if (threadIdx.x == 0) {
        __threadfence();
        am_last = atomicAdd(done, 1u) == nblocks - 1;
    }
    __syncthreads();
    if (am_last && threadIdx.x == 0) *done = 0u;
    return am_last;
}
// The inner FCG's scalars on the device, in the host's former FP64 operations: β from s·q and s·r (β = 0
// on the first step), then α = (s·r)/(p·q) with the breakdown test; on a breakdown the update is skipped
// and α, s·r are not carried to the next step.
__device__ void fcg_beta(FcgDev* S, double sq, double sr, int first) {
    const double beta = first ? 0.0 : (-S->alpha_prev * sq) / S->rho_prev;
    S->sr = sr;
    S->beta = beta;
    S->beta32 = float(beta);
}
__device__ void fcg_alpha(FcgDev* S, double pq) {
    const double sr = S->sr;
    const bool stop = !(pq != 0.0) || !isfinite(pq) || !isfinite(sr) || !isfinite(S->beta);
    const double alpha = sr / pq;
    S->alpha32 = float(alpha);
    S->stop = stop ? 1 : 0;
    S->rin = 0u;
    S->rin64 = 0ull;
    if (!stop) {
        S->rho_prev = sr;
        S->alpha_prev = alpha;
    }
}

// ---- FP64 Krylov kernels (IA_POISSON_FP64).  As the FP32 ones below, with the scalars on the device; the vectors
// are the library's, whose ghost entries are zero here, so they are streamed whole.
// q = A p and partial sums of p·q, ZT planes a thread, one chain of multiply-adds a cell; the rows follow one another
// through the lanes
template <int D, int ZT>
__global__ void __launch_bounds__(256) matvec64_k(Grid g, const double* __restrict__ L, const double* __restrict__ diag,
                                                       const double* __restrict__ pv, double* __restrict__ q,
                                                       double* __restrict__ partial, FcgDev* S) {
    const int nx = g.n[0] - 2, t = int(blockIdx.x) * 256 + int(threadIdx.x), x = 1 + t % nx, y = 1 + t / nx;   // (see plane_cell)
    const int z0 = D == 3 ? 1 + ZT * int(blockIdx.z) : 0;
    double acc = 0.0, unused = 0.0;
    if (y <= g.n[1] - 2) {
#pragma unroll
        for (int k = 0; k < (D == 3 ? ZT : 1); ++k) {
            const int z = z0 + k;
            if (D == 3 && z > g.n[2] - 2) break;
            const int I = x + y * int(g.s[1]) + z * int(g.s[2]);
            const double v = product7<D>(g, L, diag[I] * pv[I], pv, I, nb_of<D>(g, x, y, z));
            q[I] = v;
            acc = fma(pv[I], v, acc);
        }
    }
    acc = warp_sum(acc);
    __shared__ double ws[8];
    if ((threadIdx.x & 31) == 0) ws[threadIdx.x >> 5] = acc;
    __syncthreads();
    const unsigned int nb = gridDim.x * gridDim.z;
    if (threadIdx.x == 0) {
        for (int w = 1; w < 8; ++w) acc += ws[w];
        partial[blockIdx.x + gridDim.x * blockIdx.z] = acc;
    }
    if (!last_block(&S->done_mv, nb)) return;
    double pq = 0.0;
    sum2_by256(partial, nullptr, nb, pq, unused);
    if (threadIdx.x == 0) fcg_alpha(S, pq);
}
__global__ void __launch_bounds__(256) dot2_64_k(long long n, const double* __restrict__ sv, const double* __restrict__ q,
                                                 const double* __restrict__ r, double* __restrict__ partial, FcgDev* S, int first) {
    double a1 = 0.0, a2 = 0.0;
    const long long stride = (long long)gridDim.x * blockDim.x;
#pragma unroll 4
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += stride) {
        const double s = sv[i];
        a1 = fma(s, q[i], a1);
        a2 = fma(s, r[i], a2);
    }
    block_sum2(a1, a2);
    if (threadIdx.x == 0) {
        partial[blockIdx.x] = a1;
        partial[gridDim.x + blockIdx.x] = a2;
    }
    if (!last_block(&S->done_dot, gridDim.x)) return;
    double sq = 0.0, sr = 0.0;
    sum2_by256(partial, partial + gridDim.x, gridDim.x, sq, sr);
    if (threadIdx.x == 0) fcg_beta(S, sq, sr, first);
}
__global__ void __launch_bounds__(256) xpby64_k(long long n, const double* __restrict__ sv, const FcgDev* __restrict__ S,
                                                double* __restrict__ pv) {
    const double beta = S->beta;
    const long long stride = (long long)gridDim.x * blockDim.x;
#pragma unroll 4
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += stride)
        pv[i] = beta == 0.0 ? sv[i] : fma(beta, pv[i], sv[i]);
}
// x += α p (x's ghost entries, the caller's, take the direction's zeros) ; r -= α q ; L∞(r) bits into S->rin64
// (nothing after a breakdown)
__global__ void __launch_bounds__(256) update64_k(long long n, FcgDev* __restrict__ S, const double* __restrict__ pv,
                                                  const double* __restrict__ q, double* __restrict__ xv, double* __restrict__ r) {
    if (S->stop) return;
    const double alpha = S->alpha_prev;
    unsigned long long m = 0ull;
    const long long stride = (long long)gridDim.x * blockDim.x;
#pragma unroll 4
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += stride) {
        xv[i] = fma(alpha, pv[i], xv[i]);
        const double v = fma(-alpha, q[i], r[i]);
        r[i] = v;
        const unsigned long long b = abs_bits(v);
        m = b > m ? b : m;
    }
    m = block_max(m);
    if (threadIdx.x == 0) atomicMax(&S->rin64, m);
}

// ---- FP32 inner Krylov kernels (mixed / learned): FP32 products, per-thread sums in FP32
// over its cells, FP64 block and cross-block sums.
// The x-y tiles of a matrix product: 32 x 8 cells of zt consecutive planes, x fastest
struct MvTiles {
    int nx, ny, n, zt;
    __host__ __device__ MvTiles(const Grid& g, int planes) : zt(planes) {
        nx = (g.n[0] - 2 + 31) / 32;
        ny = (g.n[1] - 2 + 7) / 8;
        n = nx * ny * (g.D == 3 ? (g.n[2] - 2 + zt - 1) / zt : 1);
    }
    __device__ __forceinline__ void origin(int t, int& x, int& y, int& z) const {
        const int r = t / nx;
        x = 1 + (t - r * nx) * 32;
        z = r / ny;
        y = 1 + (r - z * ny) * 8;
        z = 1 + z * zt;
    }
};
constexpr int MV_RESIDENT = 5;   // blocks on a multiprocessor
inline unsigned mv_blocks(const Grid& g, int zt, int nsm) {
    return unsigned(std::min(MvTiles(g, zt).n, MV_RESIDENT * std::max(nsm, 1)));
}

// q = A p and per-block partial sums of p·q on x-y tiles: a block of 256 threads takes 32 x 8 cells of MV_ZT consecutive
// z planes (one plane in 2D) at a time, so that the stencil's x and y neighbours come from L1 and every load of a cell
// issues at once (a row loop, one row per block and step, waits for each row's loads and fetches the y neighbours from
// other SMs' rows through L2).  As many blocks as the device holds go through all tiles: a block of its own for each
// tile ended in a fence and a count, and the last one summed 16384 partials (256x512x256: 183 us so, 166 with 32-bit
// byte offsets, 141 with 5 resident blocks an SM, 146 with 4, 150 with 6).  The partials are summed in a fixed order.
// IX: unsigned below RB_CELLS cells, else size_t.
template <int D, int ZT, class IX>
__global__ void __launch_bounds__(256, MV_RESIDENT) matvec32_tile_k(Grid g, Ends ends, const float* __restrict__ L,
                                                                 const float* __restrict__ pv, float* __restrict__ q,
                                                                 double* __restrict__ partial, FcgDev* S) {
    const int s1 = int(g.s[1]), s2 = D == 3 ? int(g.s[2]) : 0;
    const MvTiles tiles(g, ZT);
    double sum = 0.0;
    for (int t = blockIdx.x; t < tiles.n; t += gridDim.x) {
        int x, y, z0;
        tiles.origin(t, x, y, z0);
        x += int(threadIdx.x & 31);
        y += int(threadIdx.x >> 5);
        if (D == 2) z0 = 0;
        const int xl = x == 1 ? ends.lo[0] : -1, xh = x == g.n[0] - 2 ? ends.hi[0] : 1;
        const int yl = y == 1 ? ends.lo[1] : -s1, yh = y == g.n[1] - 2 ? ends.hi[1] : s1;
        float acc = 0.f;
        auto cell = [&](int z) {
            const IX I = x + y * s1 + z * s2;
            const int zl = z == 1 ? ends.lo[2] : -s2, zh = z == g.n[2] - 2 ? ends.hi[2] : s2;
            const float c = at(pv, I);
            const Star s = star7<D>(L, g.N, I, s1, s2, at(pv, I + xl), at(pv, I + xh), at(pv, I + yl), at(pv, I + yh),
                                    D == 3 ? at(pv, I + zl) : 0.f, D == 3 ? at(pv, I + zh) : 0.f);
            const float v = s.off + s.dd * c;
            *(float*)((char*)q + I * (IX)4) = v;
            acc += c * v;
        };
        if (x <= g.n[0] - 2 && y <= g.n[1] - 2) {
            if (D == 3 && z0 + ZT - 1 <= g.n[2] - 2) {
                // a full tile: no bound test between the planes, so that their loads can be issued early
                // and a plane's values reused as the next plane's z neighbours
#pragma unroll
                for (int k = 0; k < ZT; ++k) cell(z0 + k);
            } else {
                for (int k = 0; k < (D == 3 ? ZT : 1); ++k) {
                    if (D == 3 && z0 + k > g.n[2] - 2) break;
                    cell(z0 + k);
                }
            }
        }
        // a warp's sum over a tile in FP32 (a fixed shuffle tree), over its tiles in FP64 by one lane: a per-thread
        // FP64 reduction costs more FP64-pipe time than the stencil itself
        for (int o = 16; o > 0; o >>= 1) acc += __shfl_down_sync(0xffffffffu, acc, o);
        if ((threadIdx.x & 31) == 0) sum += double(acc);
    }
    __shared__ double ws[8];
    if ((threadIdx.x & 31) == 0) ws[threadIdx.x >> 5] = sum;
    __syncthreads();
    if (threadIdx.x == 0) {
        double a = 0.0;
        for (int w = 0; w < 8; ++w) a += ws[w];
        partial[blockIdx.x] = a;
    }
    // the last block: p·q in a fixed order, then α
    if (!last_block(&S->done_mv, gridDim.x)) return;
    double pq = 0.0, unused = 0.0;
    sum2_by256(partial, nullptr, gridDim.x, pq, unused);
    if (threadIdx.x == 0) fcg_alpha(S, pq);
}

// Whole-array FP32 vector kernels of the inner solve.  Only interior cells of these vectors are
// written (the one-launch solver's copies in ghosts are cleared: clear_wrap_copies), so their ghost
// entries stay zero and sums and updates over all N entries equal those over the interior; the arrays are streamed as 16-byte vectors (cudaMalloc alignment),
// the N mod 4 tail by the first threads.
__global__ void __launch_bounds__(256, VB_RESIDENT) dot2_32_k(long long n, const float* __restrict__ sv, const float* __restrict__ q,
                          const float* __restrict__ r, double* __restrict__ partial, FcgDev* S, int first) {
    double b1 = 0.0, b2 = 0.0;
    const long long n4 = n / 4, stride = (long long)gridDim.x * blockDim.x;
    const long long t0 = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    const float4* s4 = reinterpret_cast<const float4*>(sv);
    const float4* q4 = reinterpret_cast<const float4*>(q);
    const float4* r4 = reinterpret_cast<const float4*>(r);
    auto add = [&](const float4& a, const float4& bq, const float4& br, float& a1, float& a2) {
        a1 += a.x * bq.x + a.y * bq.y + a.z * bq.z + a.w * bq.w;
        a2 += a.x * br.x + a.y * br.y + a.z * br.z + a.w * br.w;
    };
    // four vectors of each array in flight; their products are summed in FP32, a thread's sums in FP64
    long long i = t0;
    for (; i + 3 * stride < n4; i += 4 * stride) {
        float4 a[4], bq[4], br[4];
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            a[k] = s4[i + k * stride];
            bq[k] = q4[i + k * stride];
            br[k] = r4[i + k * stride];
        }
        float a1 = 0.f, a2 = 0.f;
#pragma unroll
        for (int k = 0; k < 4; ++k) add(a[k], bq[k], br[k], a1, a2);
        b1 += double(a1);
        b2 += double(a2);
    }
    float a1 = 0.f, a2 = 0.f;
    for (; i < n4; i += stride) add(s4[i], q4[i], r4[i], a1, a2);
    if (t0 < n - 4 * n4) {
        const long long k = 4 * n4 + t0;
        a1 += sv[k] * q[k];
        a2 += sv[k] * r[k];
    }
    b1 += double(a1);
    b2 += double(a2);
    block_sum2(b1, b2);
    if (threadIdx.x == 0) {
        partial[blockIdx.x] = b1;
        partial[gridDim.x + blockIdx.x] = b2;
    }
    // the last block: s·q and s·r in a fixed order, then β
    if (!last_block(&S->done_dot, gridDim.x)) return;
    double sq = 0.0, sr = 0.0;
    sum2_by256(partial, partial + gridDim.x, gridDim.x, sq, sr);
    if (threadIdx.x == 0) fcg_beta(S, sq, sr, first);
}

// p = s + β p; β = 0 restarts from s without reading the old direction (which a rejected
// preconditioner output may have left non-finite)
__global__ void __launch_bounds__(256, VB_RESIDENT) xpby32_k(long long n, const float* __restrict__ sv, const FcgDev* __restrict__ S,
                         float* __restrict__ pv) {
    const float beta = S->beta32;
    const long long n4 = n / 4, stride = (long long)gridDim.x * blockDim.x;
    const long long t0 = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    const float4* s4 = reinterpret_cast<const float4*>(sv);
    float4* p4 = reinterpret_cast<float4*>(pv);
    const bool restart = beta == 0.f;
#pragma unroll 4
    for (long long i = t0; i < n4; i += stride) {
        const float4 a = s4[i];
        if (restart) {
            p4[i] = a;
        } else {
            const float4 p = p4[i];
            p4[i] = make_float4(a.x + beta * p.x, a.y + beta * p.y, a.z + beta * p.z, a.w + beta * p.w);
        }
    }
    if (t0 < n - 4 * n4) {
        const long long i = 4 * n4 + t0;
        pv[i] = restart ? sv[i] : sv[i] + beta * pv[i];
    }
}

// e += α p ; r -= α q ; L∞(r) as float bits into S->rin (nothing after a breakdown)
__global__ void __launch_bounds__(256, VB_RESIDENT) update32_k(long long n, FcgDev* __restrict__ S, const float* __restrict__ pv,
                           const float* __restrict__ q, float* __restrict__ e, float* __restrict__ r) {
    if (S->stop) return;
    const float alpha = S->alpha32;
    unsigned int* linf = &S->rin;
    unsigned long long m = 0ull;
    const long long n4 = n / 4, stride = (long long)gridDim.x * blockDim.x;
    const long long t0 = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    const float4* p4 = reinterpret_cast<const float4*>(pv);
    const float4* q4 = reinterpret_cast<const float4*>(q);
    float4* e4 = reinterpret_cast<float4*>(e);
    float4* r4 = reinterpret_cast<float4*>(r);
    auto mx = [&](float v) {
        const unsigned long long b = __float_as_uint(v) & 0x7FFFFFFFu;
        m = b > m ? b : m;
    };
#pragma unroll 4
    for (long long i = t0; i < n4; i += stride) {
        const float4 p = p4[i], qq = q4[i];
        float4 ee = e4[i], rr = r4[i];
        ee.x += alpha * p.x; ee.y += alpha * p.y; ee.z += alpha * p.z; ee.w += alpha * p.w;
        rr.x -= alpha * qq.x; rr.y -= alpha * qq.y; rr.z -= alpha * qq.z; rr.w -= alpha * qq.w;
        e4[i] = ee;
        r4[i] = rr;
        mx(rr.x); mx(rr.y); mx(rr.z); mx(rr.w);
    }
    if (t0 < n - 4 * n4) {
        const long long i = 4 * n4 + t0;
        e[i] += alpha * pv[i];
        const float v = r[i] - alpha * q[i];
        r[i] = v;
        mx(v);
    }
    m = block_max(m);
    if (threadIdx.x == 0) atomicMax(linf, (unsigned int)m);
}

// ---- learned hybrid preconditioner: partial dots n·t and n·An for the energy-optimal step
// ω = (n·t)/(n·An), which minimises the A-norm of the error e - ω n left behind the V-cycle
// (t = A e); A is negative semi-definite here, so both dots carry the same sign.
template <int D>
__global__ void energy_dots_k(Grid g, const float* __restrict__ L, const float* __restrict__ n,
                              const float* __restrict__ t, double* __restrict__ partial) {
    float a1 = 0.f, a2 = 0.f;
    ROWS_BEGIN_D(g)
    const Nb o = nb_of<D>(g, x, y, z);
    const float an = off7<D>(g, L, n, I, o) + diag7<D>(g, L, I) * n[I];
    a1 += n[I] * t[I];
    a2 += n[I] * an;
    ROWS_END
    double b1 = a1, b2 = a2;
    block_sum2(b1, b2);
    if (threadIdx.x == 0) {
        partial[blockIdx.x] = b1;
        partial[gridDim.x + blockIdx.x] = b2;
    }
}

// s += ω n with ω = (n·t)/(n·An) from the device dots (0 unless both are finite and n·An ≠ 0)
__global__ void add_scaled_k(Grid g, const double* __restrict__ dots, const float* __restrict__ nv,
                             float* __restrict__ sv) {
    const double tn = dots[0], nan_ = dots[1];
    const bool ok = nan_ != 0.0 && nan_ == nan_ && tn == tn && fabs(nan_) < 1e300 && fabs(tn) < 1e300;
    const float w = float(ok ? tn / nan_ : 0.0);
    ROWS_BEGIN(g)
    sv[I] += w * nv[I];
    ROWS_END
}

// x += e (FP64 += FP32), interior cells
// double(v) with integer operations for zeros, normal numbers, inf and NaN (the conversion instruction
// issues on the FP64 pipe); FP32 subnormals take the conversion, out of line
__device__ __noinline__ double widen_cold(float v) { return double(v); }
__device__ __forceinline__ double widen_exact(float v) {
    const unsigned b = __float_as_uint(v);
    return (((b >> 23) & 0xFFu) != 0u || (b << 1) == 0u) ? ff_widen(v) : widen_cold(v);
}

// x += e over interior cells, on the tiles of matvec32_tile_k (one cell per thread and plane)
template <int D, int ZT>
__global__ void __launch_bounds__(256) add_correction_k(Grid g, const float* __restrict__ e, double* __restrict__ xv) {
    const int x = 1 + int(blockIdx.x) * 32 + int(threadIdx.x & 31), y = 1 + int(blockIdx.y) * 8 + int(threadIdx.x >> 5);
    const int z0 = D == 3 ? 1 + ZT * int(blockIdx.z) : 0;
    if (x > g.n[0] - 2 || y > g.n[1] - 2) return;
#pragma unroll
    for (int k = 0; k < (D == 3 ? ZT : 1); ++k) {
        const int z = z0 + k;
        if (D == 3 && z > g.n[2] - 2) break;
        const int I = x + y * int(g.s[1]) + z * int(g.s[2]);
        xv[I] += widen_exact(e[I]);
    }
}

// periodic ghost of a scalar (WaterLily perBC!) at number t of the boundary planes' cells; reads only positions that
// no thread writes: the mapped position has no periodic ghost coordinate left
__device__ __forceinline__ void perbc_cell(const Grid& g, double* a, long long t) {
    int c[3];
    if (!bc_plane_cell(g, t, c)) return;
    const int x = c[0], y = c[1], z = c[2];
    bool any = false;
    for (int e = 0; e < g.D; ++e)
        if (g.isper(e) && (c[e] == 0 || c[e] == g.n[e] - 1)) {
            c[e] = bc_src(g, e, c[e]);
            any = true;
        }
    if (any) a[lin(g, x, y, z)] = a[lin3(g, c)];
}
// one thread per cell of the boundary planes
__global__ void perbc_k(Grid g, double* a) { perbc_cell(g, a, blockIdx.x * (long long)blockDim.x + threadIdx.x); }

}  // namespace
}  // namespace ia
#include "poisson_cluster.cuh"
namespace ia {

// ------------------------------------------------------------------ host side

// z-planes per block of the blocked smoother: about eight blocks per multiprocessor in all,
// each block marching at least 4 S planes
static int tb_zchunk(const Grid& g, int S, int nsm) {
    const int tiles = ((g.n[0] - 2 + TB_X - 1) / TB_X) * ((g.n[1] - 2 + TB_Y - 1) / TB_Y);
    const int nzi = g.n[2] - 2;
    const int want = std::max(1, (8 * std::max(nsm, 1)) / std::max(tiles, 1));
    int zc = (nzi + want - 1) / want;
    zc = std::max(zc, std::min(nzi, 4 * S));
    return std::max(zc, 1);
}

// the blocked smoother runs the FP32 V-cycle of a 3D level whose next coarser level (gc) halves every
// dimension, for nu1, nu2 in {1, 2}
static bool tb_usable(const PoissonMG* mg, const Grid& g, const Grid& gc) {
    if (mg->smoother != IA_SMOOTHER_BLOCKED || g.D != 3 || mg->omega != 1.0) return false;
    if (mg->nu1 < 1 || mg->nu1 > 2 || mg->nu2 < 1 || mg->nu2 > 2) return false;
    return mg_regular(g, gc);
}

static void tb_launch(const PoissonMG* mg, const TbArgs& a, int S, cudaStream_t st) {
    TbArgs b = a;
    b.zchunk = tb_zchunk(a.g, S, mg->nsm);
    const dim3 grid((a.g.n[0] - 2 + TB_X - 1) / TB_X, (a.g.n[1] - 2 + TB_Y - 1) / TB_Y,
                    (a.g.n[2] - 2 + b.zchunk - 1) / b.zchunk);
    const bool zero = a.xin == nullptr;
    if (S == 4) {
        if (zero) rbgs_tb_k<4, true><<<grid, TB_T, 0, st>>>(b);
        else rbgs_tb_k<4, false><<<grid, TB_T, 0, st>>>(b);
    } else {
        if (zero) rbgs_tb_k<2, true><<<grid, TB_T, 0, st>>>(b);
        else rbgs_tb_k<2, false><<<grid, TB_T, 0, st>>>(b);
    }
    ia::note_launch();
}

constexpr int TAIL_BYTES = 200 * 1024;   // shared memory of the one-block V-cycle
constexpr int CL_BYTES = 210 * 1024;     // and, with what is static, of a block of the one-launch solver
// shared-memory layout of the one-block V-cycle from level l0 on
template <class T>
static TailArgs<T> tail_layout(const PoissonMG* mg, int l0) {
    TailArgs<T> a;
    a.nl = mg->nlev - l0;
    int v = 0, w = 0;
    for (int k = 0; k < a.nl && k < TAIL_MAX; ++k) {
        const Grid& g = mg->lev[l0 + k].g;
        const int np = (g.n[0] - 1) / 2 * (g.n[1] - 2) * (g.D == 3 ? g.n[2] - 2 : 1);
        a.g[k] = g;
        a.np[k] = np;
        a.xo[k] = v;
        a.bo[k] = v += int(g.N);
        a.co[k] = v += 2 * np;
        v += (2 * g.D + 1) * 2 * np;
        a.io[k] = w;
        w += TAIL_WORDS * np;
    }
    a.ro = v;
    a.values = v + int(a.g[0].N);
    a.words = w;
    return a;
}
// first level of the one-block V-cycle; the coarsest level (at most 512 cells) always fits
template <class T>
static int tail_level(const PoissonMG* mg, long long most = tail_pairs<T>()) {
    int l = mg->nlev - 1;
    while (l > 0 && mg->nlev - l < TAIL_MAX) {
        const Grid& g = mg->lev[l - 1].g;
        const long long pairs = (long long)((g.n[0] - 1) / 2) * (g.n[1] - 2) * (g.D == 3 ? g.n[2] - 2 : 1);
        if (pairs > most || mg->lev[l].g.N > 0xFFFF || tail_layout<T>(mg, l - 1).bytes() > (size_t)TAIL_BYTES) break;
        --l;
    }
    return l;
}
template <class T>
static TailArgs<T> tail_args(PoissonMG* mg, int l0, int nu1, int nu2, int nuc) {
    TailArgs<T> a = tail_layout<T>(mg, l0);
    for (int k = 0; k < a.nl; ++k) {
        MGLevel& L = mg->lev[l0 + k];
        a.L[k] = L.template L_<T>();
        a.iD[k] = L.template iD_<T>();
        a.nu1[k] = (l0 + k == 0 && mg->nu1f > 0) ? mg->nu1f : nu1;
        a.nu2[k] = (l0 + k == 0 && mg->nu2f > 0) ? mg->nu2f : nu2;
    }
    a.nuc = nuc;
    a.omega = T(mg->omega);
    a.b = mg->lev[l0].template b_<T>();
    a.x = mg->lev[l0].template x_<T>();
    return a;
}

template <class T>
static cudaError_t vcycle(ia_handle* h, PoissonMG* mg, int l, cudaStream_t st, int nu1, int nu2, int nuc) {
    auto& L = mg->lev[l];
    T* x = L.template x_<T>();
    T* b = L.template b_<T>();
    const T* Lc = L.template L_<T>();
    const T* iD = L.template iD_<T>();
    if (l >= tail_level<T>(mg)) {
        const TailArgs<T> a = tail_args<T>(mg, l, nu1, nu2, nuc);
        const size_t bytes = a.bytes();
        if (L.g.D == 3) mg_tail_k<T, 3><<<1, TAIL_THREADS, bytes, st>>>(a);
        else mg_tail_k<T, 2><<<1, TAIL_THREADS, bytes, st>>>(a);
        ia::note_launch();
        return cudaGetLastError();
    }
    if constexpr (sizeof(T) == 4) {
        if (tb_usable(mg, L.g, mg->lev[l + 1].g)) {
            // pre-smoothing from zero into the level's scratch vector, residual restriction
            // from it, then post-smoothing of scratch + prolongated correction into x
            auto& C = mg->lev[l + 1];
            TbArgs ta;
            ta.g = L.g;
            ta.gc = C.g;
            ta.L = Lc;
            ta.b = b;
            ta.iD = iD;
            ta.xin = nullptr;
            ta.xc = nullptr;
            ta.xout = L.r32;
            ta.c0 = 0;
            ta.zchunk = 1;
            int tk = (l == 0) ? timing_begin(h, TK_MG_FINE) : -1;
            tb_launch(mg, ta, 2 * nu1, st);
            timing_end(h, tk);
            { resid_restrict_k<T, 3><<<cell_grid(C.g), blk(), 0, st>>>(C.g, 1, C.g.n[1] - 1, L.g, Lc, (const T*)nullptr, b, L.r32, C.template b_<T>()); ia::note_launch(); }
            cudaError_t e = vcycle<T>(h, mg, l + 1, st, nu1, nu2, nuc);
            if (e != cudaSuccess) return e;
            ta.xin = L.r32;
            ta.xc = C.x32;
            ta.xout = x;
            ta.c0 = 1;
            tk = (l == 0) ? timing_begin(h, TK_MG_FINE) : -1;
            tb_launch(mg, ta, 2 * nu2, st);
            timing_end(h, tk);
            return cudaGetLastError();
        }
    }
    // the finest level may smooth a different number of times than the coarser ones (ia_poisson_mg_fine);
    // the recursion below passes the coarse counts on
    const int nu1_here = (l == 0 && mg->nu1f > 0) ? mg->nu1f : nu1;
    const int nu2_here = (l == 0 && mg->nu2f > 0) ? mg->nu2f : nu2;
    // the finest mixed level's half-sweeps and residual restriction read the FP16 coefficient copy
    const __half* L16 = nullptr;
    if constexpr (sizeof(T) == 4) L16 = (l == 0 && mg->coef16) ? L.L16 : nullptr;
    auto& C = mg->lev[l + 1];
    const T om = T(mg->omega);
    const bool reg = mg_regular(L.g, C.g);
    // 3D levels in FP32 that halve evenly: the kernels of poisson_regular.cuh
    const bool even = sizeof(T) == 4 && L.g.D == 3 && reg && L.g.N < RB_CELLS;
    auto with_even = [&](auto&& launch) {
        if constexpr (sizeof(T) == 4) {
            const float* xc = C.x32;
            if (L16) launch(rb_args(L.g, C.g, L16, b, iD, x, xc, om));
            else launch(rb_args(L.g, C.g, Lc, b, iD, x, xc, om));
        }
        ia::note_launch();
    };
    // each launch takes the interior rows [y0, y1)
    const int pairs = (L.g.n[0] - 1) / 2;
    // cells of one colour that touch across a wrap are updated in passes, one per class of such cells
    const int conf = wrap_conflicts(L.g);
    auto half = [&](int color, int y0, int y1) {
        const int tk = (l == 0) ? timing_begin(h, TK_MG_FINE) : -1;
        const dim3 gr = plane_grid<T>(pairs, y1 - y0, L.g.D == 3 ? (L.g.n[2] - 2 + RB_ZT - 1) / RB_ZT : 1);
        if (even) {
            with_even([&](auto a) {
                a.y0 = y0;
                a.y1 = y1;
                a.color = color;
                rb_half_k<std::decay_t<decltype(*a.L)>, false><<<gr, blk(), 0, st>>>(a);
            });
            timing_end(h, tk);
            return;
        }
        for (int cls = 0; cls <= conf; ++cls) {
            if (cls & ~conf) continue;
            auto go = [&](const auto* coef) {
                using TL = std::decay_t<decltype(*coef)>;
                if (L.g.D == 3) rbgs_pair_k<T, 3, false, TL><<<gr, blk(), 0, st>>>(L.g, y0, y1, coef, b, iD, x, color, om, conf, cls);
                else rbgs_pair_k<T, 2, false, TL><<<gr, blk(), 0, st>>>(L.g, y0, y1, coef, b, iD, x, color, om, conf, cls);
            };
            if constexpr (sizeof(T) == 4) {
                if (L16) go(L16);
            }
            if (!L16) go(Lc);
            ia::note_launch();
        }
        timing_end(h, tk);
    };
    // the relaxed first red half-sweep of a post-smoothing: the red cells still hold x without the
    // coarse correction, which it adds to the value it reads
    auto half_prol = [&](int y0, int y1) {
        const int tk = (l == 0) ? timing_begin(h, TK_MG_FINE) : -1;
        const dim3 gr = plane_grid<T>(pairs, y1 - y0, L.g.D == 3 ? (L.g.n[2] - 2 + RB_ZT - 1) / RB_ZT : 1);
        if (even) {
            with_even([&](auto a) {
                a.y0 = y0;
                a.y1 = y1;
                rb_half_k<std::decay_t<decltype(*a.L)>, true><<<gr, blk(), 0, st>>>(a);
            });
            timing_end(h, tk);
            return;
        }
        const T* xc = C.template x_<T>();
        auto go = [&](auto REG, const auto* coef) {
            using TL = std::decay_t<decltype(*coef)>;
            constexpr bool R = decltype(REG)::value;
            if (L.g.D == 3) rbgs_pair_k<T, 3, true, TL, R><<<gr, blk(), 0, st>>>(L.g, y0, y1, coef, b, iD, x, 0, om, 0, 0, C.g, xc);
            else rbgs_pair_k<T, 2, true, TL, R><<<gr, blk(), 0, st>>>(L.g, y0, y1, coef, b, iD, x, 0, om, 0, 0, C.g, xc);
        };
        if constexpr (sizeof(T) == 4) {
            if (L16) reg ? go(std::true_type{}, L16) : go(std::false_type{}, L16);
        }
        if (!L16) reg ? go(std::true_type{}, Lc) : go(std::false_type{}, Lc);
        ia::note_launch();
        timing_end(h, tk);
    };
    // over-relaxed updates read the cell's own previous value: the red values of the first sweep
    // are then stored, and the post-smoothing's first red half-sweep adds the coarse correction
    // to the value it reads
    const bool relax = mg->omega != 1.0;
    const int write_red = (nu1_here == 1 || relax) ? 1 : 0;
    // first black half-sweep: from x = 0 (pre) or from x + P(x_coarse) (post)
    auto first = [&](bool prol, int y0, int y1) {
        const int tk = (l == 0) ? timing_begin(h, TK_MG_FIRST) : -1;
        const dim3 gr = plane_grid<T>(pairs, y1 - y0, L.g.D == 3 ? L.g.n[2] - 2 : 1);
        const int wr = prol ? 0 : write_red;
        if (even) {
            with_even([&](auto a) {
                using TL = std::decay_t<decltype(*a.L)>;
                a.y0 = y0;
                a.y1 = y1;
                a.write_red = wr;
                if (prol) rb_first_k<TL, true><<<gr, blk(), 0, st>>>(a);
                else rb_first_k<TL, false><<<gr, blk(), 0, st>>>(a);
            });
            timing_end(h, tk);
            return;
        }
        const T* xc = C.template x_<T>();
        auto go = [&](auto PROL, auto REG, const auto* coef) {
            using TL = std::decay_t<decltype(*coef)>;
            constexpr bool P = decltype(PROL)::value, R = decltype(REG)::value;
            if (L.g.D == 3) rbgs_first_k<T, 3, P, TL, R><<<gr, blk(), 0, st>>>(L.g, y0, y1, C.g, coef, b, iD, xc, x, wr, om);
            else rbgs_first_k<T, 2, P, TL, R><<<gr, blk(), 0, st>>>(L.g, y0, y1, C.g, coef, b, iD, xc, x, wr, om);
        };
        auto pick = [&](const auto* coef) {
            if (!prol) go(std::false_type{}, std::true_type{}, coef);   // no coarse parent is read
            else if (reg) go(std::true_type{}, std::true_type{}, coef);
            else go(std::true_type{}, std::false_type{}, coef);
        };
        if constexpr (sizeof(T) == 4) {
            if (L16) pick(L16);
        }
        if (!L16) pick(Lc);
        ia::note_launch();
        timing_end(h, tk);
    };
    // residual restriction of the coarse rows [yc0, yc1)
    auto restrict_rows = [&](int yc0, int yc1) {
        const dim3 gr = plane_grid<T>(C.g.n[0] - 2, yc1 - yc0, C.g.D == 3 ? C.g.n[2] - 2 : 1);
        T* bc = C.template b_<T>();
        if (even) {
            with_even([&](auto a) {
                a.y0 = yc0;
                a.y1 = yc1;
                if constexpr (sizeof(T) == 4) rb_restrict_k<<<gr, blk(), 0, st>>>(a, bc);
            });
            return;
        }
        const T* dg = nullptr;   // FP64: the diagonal is kept in the level's scratch vector
        if constexpr (sizeof(T) == 8) dg = L.r;
        auto go = [&](auto REG, const auto* coef) {
            using TL = std::decay_t<decltype(*coef)>;
            constexpr bool R = decltype(REG)::value;
            if (L.g.D == 3) resid_restrict_k<T, 3, TL, R><<<gr, blk(), 0, st>>>(C.g, yc0, yc1, L.g, coef, dg, b, x, bc);
            else resid_restrict_k<T, 2, TL, R><<<gr, blk(), 0, st>>>(C.g, yc0, yc1, L.g, coef, dg, b, x, bc);
        };
        if constexpr (sizeof(T) == 4) {
            if (L16) reg ? go(std::true_type{}, L16) : go(std::false_type{}, L16);
        }
        if (!L16) reg ? go(std::true_type{}, Lc) : go(std::false_type{}, Lc);
        ia::note_launch();
    };
    // A smoothing is a chain of stages, each a half-sweep of one colour that reads the previous
    // stage's values in rows y-1 .. y+1 (and its own colour's values from two stages back).  On the
    // finest FP32 level with walls in y, the chain runs as a wavefront over slabs of slab_rows rows:
    // for slab k the stage s takes rows [a_k - s, a_(k+1) - s), one row behind stage s-1, so every row
    // a stage reads is final for its predecessor and not yet rewritten by its successor (red-black
    // updates read only the other colour).  The results are those of whole-level half-sweeps, bit for
    // bit, while a slab's rows are still in L2 for the next stage.  The restriction follows with the
    // coarse rows whose fine rows (and their neighbours) are final.
    const bool slab = sizeof(T) == 4 && l == 0 && mg->slab_rows > 0 && L.g.D == 3 && !L.g.isper(1) && !conf &&
                      L.g.n[1] - 2 > mg->slab_rows;
    auto chain = [&](int S, auto&& stage, bool with_restrict) {
        const int ny = L.g.n[1] - 2, yend = L.g.n[1] - 1;
        const int R = slab ? std::max(mg->slab_rows, 2 * S) : ny;
        const int K = (ny + R - 1) / R;
        int yc_done = 1;
        for (int k = 0; k < K; ++k) {
            const bool lastk = k + 1 == K;
            const int a0 = 1 + k * R, a1 = lastk ? yend : 1 + (k + 1) * R;
            for (int s = 0; s < S; ++s) {
                const int y0 = (k == 0) ? 1 : a0 - s, y1 = lastk ? yend : a1 - s;
                if (y1 > y0) stage(s, y0, y1);
            }
            if (with_restrict) {
                const int yc1 = lastk ? C.g.n[1] - 1 : std::min(C.g.n[1] - 1, (a1 - S - 1) / 2 + 1);
                if (yc1 > yc_done) {
                    restrict_rows(yc_done, yc1);
                    yc_done = yc1;
                }
            }
        }
    };
    if (conf) {
        // cells of one colour touch across a wrap, and the fused first half-sweep would take a black neighbour there for
        // a red one: (red, black) nu1 times from x = 0
        cudaError_t e = cudaMemsetAsync(x, 0, sizeof(T) * (size_t)L.g.N, st);
        if (e != cudaSuccess) return e;
        for (int s = 0; s < 2 * nu1_here; ++s) half(s & 1, 1, L.g.n[1] - 1);
        restrict_rows(1, C.g.n[1] - 1);
    } else {
        // pre-smoothing: first (black with the red values in place), then (red, black) nu1 - 1 times
        chain(2 * nu1_here - 1, [&](int s, int y0, int y1) {
            if (s == 0) first(false, y0, y1);
            else half((s & 1) ? 0 : 1, y0, y1);
        }, true);
    }
    cudaError_t e = vcycle<T>(h, mg, l + 1, st, nu1, nu2, nuc);
    if (e != cudaSuccess) return e;
    if (nu2_here == 0 || conf) {
        { prolong_k<T><<<grd(L.g), blk(), 0, st>>>(L.g, C.g, C.template x_<T>(), x); ia::note_launch(); }
        // with wrap conflicts the fused prolongation would read cells that it writes: the half-sweeps
        // (black, red) nu2 times follow the separate pass
        for (int s = 0; s < 2 * nu2_here; ++s) half((s & 1) ? 0 : 1, 1, L.g.n[1] - 1);
        return cudaGetLastError();
    }
    // post-smoothing: first (black from x + P(x_coarse)), red (adding the correction when relaxed),
    // then (black, red) nu2 - 1 times
    chain(2 * nu2_here, [&](int s, int y0, int y1) {
        if (s == 0) first(true, y0, y1);
        else if (s == 1 && relax) half_prol(y0, y1);
        else half((s & 1) ? 0 : 1, y0, y1);
    }, false);
    return cudaGetLastError();
}

// The finest-level V-cycle through its CUDA graph (plain launches while per-launch timing is on)
template <class T>
static cudaError_t vcycle_run(ia_handle* h, PoissonMG* mg, cudaStream_t st) {
    if (h->timing.on) return vcycle<T>(h, mg, 0, st, mg->nu1, mg->nu2, mg->nuc);
    const int k = sizeof(T) == 4 ? 0 : 1;
    int* nu = mg->vgraph_nu[k];
    if (mg->vgraph[k] && (nu[0] != mg->nu1 || nu[1] != mg->nu2 || nu[2] != mg->nuc || nu[3] != mg->smoother ||
                          mg->vgraph_omega[k] != mg->omega || mg->vgraph_c16[k] != mg->coef16 ||
                          mg->vgraph_slab[k] != mg->slab_rows || mg->vgraph_fine[k] != mg->nu1f * 64 + mg->nu2f)) {
        cudaGraphExecDestroy(mg->vgraph[k]);
        mg->vgraph[k] = nullptr;
    }
    if (!mg->vgraph[k]) {
        if (!mg->capture && cudaStreamCreateWithFlags(&mg->capture, cudaStreamNonBlocking) != cudaSuccess)
            return vcycle<T>(h, mg, 0, st, mg->nu1, mg->nu2, mg->nuc);
        const long long n0 = launch_count();
        cudaGraph_t gr = nullptr;
        cudaError_t e = cudaStreamBeginCapture(mg->capture, cudaStreamCaptureModeThreadLocal);
        if (e == cudaSuccess) {
            const cudaError_t ek = vcycle<T>(h, mg, 0, mg->capture, mg->nu1, mg->nu2, mg->nuc);
            e = cudaStreamEndCapture(mg->capture, &gr);
            if (e == cudaSuccess) e = ek;
        }
        const long long captured = launch_count() - n0;
        note_launches(-captured);   // captured, not launched
        if (e == cudaSuccess) e = cudaGraphInstantiate(&mg->vgraph[k], gr, 0);
        if (gr) cudaGraphDestroy(gr);
        if (e != cudaSuccess) {
            mg->vgraph[k] = nullptr;
            cudaGetLastError();
            return vcycle<T>(h, mg, 0, st, mg->nu1, mg->nu2, mg->nuc);
        }
        mg->vgraph_kernels[k] = captured;
        nu[0] = mg->nu1;
        nu[1] = mg->nu2;
        nu[2] = mg->nuc;
        nu[3] = mg->smoother;
        mg->vgraph_omega[k] = mg->omega;
        mg->vgraph_c16[k] = mg->coef16;
        mg->vgraph_slab[k] = mg->slab_rows;
        mg->vgraph_fine[k] = mg->nu1f * 64 + mg->nu2f;
    }
    note_launches(mg->vgraph_kernels[k]);
    return cudaGraphLaunch(mg->vgraph[k], st);
}

// the finest-level coefficients L = 1/ρ_face lie in [1/max(λρ,1), 1/min(λρ,1)] (0 on wall faces): FP16
// holds them (relative precision 2^-11) when that interval lies inside its normal range
bool coef16_fits(double lrho) {
    const double lo = lrho < 1.0 ? lrho : 1.0, hi = lrho < 1.0 ? 1.0 : lrho;
    return lo > 0.0 && 1.0 / lo <= 60000.0 && 1.0 / hi >= 1e-4;
}

// Cells of the next coarser level along a dimension of n: half of them rounded up, for a periodic dimension to
// an even number (the red-black colouring has to close across the wrap), or to one.
static long long mg_coarse_cells(long long n, bool periodic) {
    const long long c = (n + 1) / 2;
    return periodic && c > 1 ? c + (c & 1) : c;
}

// Rows per slab of the finest-level wavefront: the bytes a stage touches per interior row (x, b, the
// inverse diagonal and the coefficients) times the rows of a slab within about 3/5 of L2, a multiple of
// 8 rows (measured at 256x512x256: 64 rows 45.7 ms per step, 32 rows 47.0, 16 rows 49.9, whole-level
// half-sweeps 46.3: smaller slabs lose more to launches and partial blocks than they gain in L2 hits).
// 0 (whole-level half-sweeps) where the wavefront does not apply.
int mg_create(ia_handle* h) {
    PoissonMG* mg = new PoissonMG();
    h->mg = mg;
    const Grid& g0 = h->g;
    long long Nint[3] = {g0.n[0] - 2, g0.n[1] - 2, g0.D == 3 ? g0.n[2] - 2 : 1};
    const bool mixed = h->cfg.poisson_mode != IA_POISSON_FP64;
    mg->coef16 = (mixed && coef16_fits(h->cfg.lrho)) ? 1 : 0;
    int nl = 0;
    int pr[3] = {0, 0, 0};
    std::vector<double> width[3];   // cell widths of the current level in finest cells
    for (int d = 0; d < g0.D; ++d) width[d].assign((size_t)Nint[d], 1.0);
    std::vector<double> ratio;
    while (nl < MG_MAX_LEVELS) {
        int64_t N[3] = {Nint[0], Nint[1], Nint[2]};
        MGLevel& L = mg->lev[nl];
        L.g = make_grid(g0.D, g0.per, N);
        for (int d = 0; d < 3; ++d) L.g.pr[d] = pr[d];
        const size_t n = (size_t)L.g.N;
        cudaError_t e = cudaSuccess;
        // FP64 levels always exist for level 0 (fine operator copies) and for the FP64 mode
        if (!mixed) {
            e = e ? e : cudaMalloc(&L.x, 8 * n);
            e = e ? e : cudaMalloc(&L.b, 8 * n);
            e = e ? e : cudaMalloc(&L.r, 8 * n);
            e = e ? e : cudaMalloc(&L.L, 8 * n * g0.D);
            e = e ? e : cudaMalloc(&L.iD, 8 * n);
            if ((long long)mg->lev[0].g.N <= 2 * cluster_cells<float>()) e = e ? e : cudaMalloc(&L.t, 8 * n);
            if (!e) {
                cudaMemset(L.x, 0, 8 * n);
                cudaMemset(L.b, 0, 8 * n);
                cudaMemset(L.r, 0, 8 * n);
                cudaMemset(L.iD, 0, 8 * n);
                cudaMemset(L.L, 0, 8 * n * g0.D);
            }
        } else {
            e = e ? e : cudaMalloc(&L.x32, 4 * n);
            e = e ? e : cudaMalloc(&L.b32, 4 * n);
            e = e ? e : cudaMalloc(&L.r32, 4 * n);
            e = e ? e : cudaMalloc(&L.L32, 4 * n * g0.D);
            e = e ? e : cudaMalloc(&L.iD32, 4 * n);
            if (nl == 0) e = e ? e : cudaMalloc(&L.L16, 2 * n * g0.D);
            if (!e) {
                cudaMemset(L.x32, 0, 4 * n);
                cudaMemset(L.b32, 0, 4 * n);
                cudaMemset(L.r32, 0, 4 * n);
                cudaMemset(L.iD32, 0, 4 * n);
                cudaMemset(L.L32, 0, 4 * n * g0.D);
            }
        }
        if (nl > 0) {
            e = e ? e : cudaMalloc(&L.ratio, 8 * ratio.size());
            if (!e) e = cudaMemcpy(L.ratio, ratio.data(), 8 * ratio.size(), cudaMemcpyHostToDevice);
        }
        if (e != cudaSuccess) return IA_ERR_CUDA;
        ++nl;
        long long cells = 1;
        for (int d = 0; d < g0.D; ++d) cells *= Nint[d];
        // the coarsest level: few cells, and short enough that its sweeps reach across it
        long long side = 0;
        for (int d = 0; d < g0.D; ++d) side = std::max(side, Nint[d]);
        if (cells <= 512 && side <= 8) break;
        bool coarser = false;
        ratio.clear();
        for (int d = 0; d < g0.D; ++d) {
            const long long n = Nint[d], nc = mg_coarse_cells(n, g0.isper(d));
            pr[d] = int(n - nc);
            coarser = coarser || nc < n;
            // widths of the coarse cells and, for coarse face c = 1 .. nc + 1 (entry c, entry 0 unused), the
            // distance of the cell centres beside it on this level over that on the coarse one
            std::vector<double> wc;
            for (long long c = 0, q = 0; c < nc; ++c, ++q) {
                double w = width[d][(size_t)q];
                if (c < pr[d]) w += width[d][(size_t)++q];
                wc.push_back(w);
            }
            auto dist = [](const std::vector<double>& w, long long lo, long long hi) { return 0.5 * (w[(size_t)lo] + w[(size_t)hi]); };
            ratio.push_back(0.5);
            for (long long c = 0; c <= nc; ++c) {
                const long long q = c < pr[d] ? 2 * c : c + pr[d];   // first child of coarse cell c (0-based)
                // the outer faces: across the wrap, or a wall (whose coefficient is zero)
                const bool edge = c == 0 || c == nc;
                if (nc == 1) ratio.push_back(0.0);
                else ratio.push_back(dist(width[d], edge ? n - 1 : q - 1, edge ? 0 : q) / dist(wc, edge ? nc - 1 : c - 1, edge ? 0 : c));
            }
            width[d] = wc;
            Nint[d] = nc;
        }
        if (!coarser) break;
    }
    mg->nlev = nl;
    if (cudaFuncSetAttribute(mg_tail_k<float, 2>, cudaFuncAttributeMaxDynamicSharedMemorySize, TAIL_BYTES) != cudaSuccess ||
        cudaFuncSetAttribute(mg_tail_k<float, 3>, cudaFuncAttributeMaxDynamicSharedMemorySize, TAIL_BYTES) != cudaSuccess ||
        cudaFuncSetAttribute(mg_tail_k<double, 2>, cudaFuncAttributeMaxDynamicSharedMemorySize, TAIL_BYTES) != cudaSuccess ||
        cudaFuncSetAttribute(mg_tail_k<double, 3>, cudaFuncAttributeMaxDynamicSharedMemorySize, TAIL_BYTES) != cudaSuccess)
        return IA_ERR_CUDA;
    const size_t N = (size_t)g0.N;
    cudaError_t e = cudaSuccess;
    // FP64: the finest level's right-hand side is the Krylov residual; mixed: the FP64 true residual
    if (!mixed) mg->r = mg->lev[0].b;
    else e = e ? e : cudaMalloc(&mg->r, 8 * N);
    e = e ? e : cudaMalloc(&mg->p, 8 * N);
    e = e ? e : cudaMalloc(&mg->q, 8 * N);
    mg->kb = kblocks(g0);
    {
        int dev = 0;
        cudaGetDevice(&dev);
        cudaDeviceGetAttribute(&mg->nsm, cudaDevAttrMultiProcessorCount, dev);
        mg->vb = vblocks(g0, mg->nsm);
        mg->zt = mv_planes(g0, mg->nsm);
        const dim3 mv = mv_tile_grid(g0, mg->zt);
        mg->mvb = (long long)mv.x * mv.y * mv.z;
    }
    e = e ? e : cudaMalloc(&mg->partial, 8 * std::max<size_t>(2 * (size_t)KBLOCKS, (size_t)mg->mvb));
    e = e ? e : cudaMalloc(&mg->diag64, 8 * N);
    if (!e) cudaMemset(mg->diag64, 0, 8 * N);
    if (mixed) {
        e = e ? e : cudaMalloc(&mg->p32, 4 * N);
        e = e ? e : cudaMalloc(&mg->q32, 4 * N);
        e = e ? e : cudaMalloc(&mg->e32, 4 * N);
        if (!e) {
            cudaMemset(mg->p32, 0, 4 * N);
            cudaMemset(mg->q32, 0, 4 * N);
            cudaMemset(mg->e32, 0, 4 * N);
        }
    }
    if (h->cfg.poisson_mode == IA_POISSON_LEARNED) {
        e = e ? e : cudaMalloc(&mg->rl32, 4 * N);
        e = e ? e : cudaMalloc(&mg->nl32, 4 * N);
        e = e ? e : cudaMalloc(&mg->t32, 4 * N);
        if (!e) {   // ghosts stay zero: only interior cells are written
            cudaMemset(mg->rl32, 0, 4 * N);
            cudaMemset(mg->nl32, 0, 4 * N);
            cudaMemset(mg->t32, 0, 4 * N);
        }
    }
    e = e ? e : cudaMalloc(&mg->dsc, 8 * 16);
    e = e ? e : cudaMalloc(&mg->fcg, sizeof(FcgDev));
    if (!e) cudaMemset(mg->fcg, 0, sizeof(FcgDev));
    e = e ? e : cudaMallocHost(&mg->hsc, 8 * 16);
    if (e != cudaSuccess) return IA_ERR_CUDA;
    cudaMemset(mg->r, 0, 8 * N);
    cudaMemset(mg->p, 0, 8 * N);
    cudaMemset(mg->q, 0, 8 * N);
    mg->nu1 = 2;
    mg->nu2 = 2;
    mg->nuc = 16;
    // whole-level half-sweeps by default: with two z planes per half-sweep thread the y-slab wavefront
    // (ia_poisson_slab_rows) no longer shortens the step
    mg->slab_rows = 0;
    return IA_OK;
}

void mg_destroy(ia_handle* h) {
    PoissonMG* mg = h->mg;
    if (!mg) return;
    for (int l = 0; l < MG_MAX_LEVELS; ++l) {
        MGLevel& L = mg->lev[l];
        cudaFree(L.x); cudaFree(L.b); cudaFree(L.r); cudaFree(L.L); cudaFree(L.iD); cudaFree(L.t);
        cudaFree(L.x32); cudaFree(L.b32); cudaFree(L.r32); cudaFree(L.L32); cudaFree(L.iD32); cudaFree(L.L16);
        cudaFree(L.ratio);
    }
    if (mg->r != mg->lev[0].b) cudaFree(mg->r);
    cudaFree(mg->p); cudaFree(mg->q);
    cudaFree(mg->p32); cudaFree(mg->q32); cudaFree(mg->e32);
    cudaFree(mg->rl32); cudaFree(mg->nl32); cudaFree(mg->t32);
    cudaFree(mg->partial); cudaFree(mg->dsc); cudaFree(mg->fcg); cudaFree(mg->diag64);
    for (int k = 0; k < 2; ++k)
        if (mg->vgraph[k]) cudaGraphExecDestroy(mg->vgraph[k]);
    if (mg->capture) cudaStreamDestroy(mg->capture);
    if (mg->hsc) cudaFreeHost(mg->hsc);
    delete mg;
    h->mg = nullptr;
}

// build every level's operator from the fine coefficients L0 (μ₀, FP64)
static cudaError_t mg_setup(ia_handle* h, const double* L0) {
    PoissonMG* mg = h->mg;
    cudaStream_t st = h->stream;
    const bool mixed = h->cfg.poisson_mode != IA_POISSON_FP64;
    MGLevel& F = mg->lev[0];
    const long long nv = F.g.N * F.g.D;
    if (!mixed) { set_diag64_k<<<mg->kb, KTHREADS, 0, st>>>(F.g, L0, mg->diag64); ia::note_launch(); }
    if (!mixed) {
        cudaMemcpyAsync(F.L, L0, 8 * nv, cudaMemcpyDeviceToDevice, st);
        { set_diag_k<double><<<grd(F.g), blk(), 0, st>>>(F.g, F.L, F.iD, F.r); ia::note_launch(); }
        for (int l = 1; l < mg->nlev; ++l) {
            { restrict_L_k<double><<<grd(mg->lev[l].g), blk(), 0, st>>>(mg->lev[l].g, mg->lev[l - 1].g,
                                                                       mg->lev[l - 1].L, mg->lev[l].ratio, mg->lev[l].L); ia::note_launch(); }
            { set_diag_k<double><<<grd(mg->lev[l].g), blk(), 0, st>>>(mg->lev[l].g, mg->lev[l].L, mg->lev[l].iD, mg->lev[l].r); ia::note_launch(); }
        }
    } else {
        // FP64 diagonal, FP32 (and FP16) coefficient copies and the FP32 inverse diagonal in one pass
        const dim3 gg((F.g.n[0] + 31) / 32, (F.g.n[1] + 7) / 8, F.g.D == 3 ? F.g.n[2] : 1);
        __half* l16 = mg->coef16 ? F.L16 : nullptr;
        LAUNCH_D(F.g, setup_fine_k, gg, blk(), F.g, L0, mg->diag64, F.L32, l16, F.iD32);
        for (int l = 1; l < mg->nlev; ++l) {
            { restrict_L_k<float><<<grd(mg->lev[l].g), blk(), 0, st>>>(mg->lev[l].g, mg->lev[l - 1].g,
                                                                      mg->lev[l - 1].L32, mg->lev[l].ratio, mg->lev[l].L32); ia::note_launch(); }
            { set_diag_k<float><<<grd(mg->lev[l].g), blk(), 0, st>>>(mg->lev[l].g, mg->lev[l].L32, mg->lev[l].iD32, nullptr); ia::note_launch(); }
        }
    }
    return cudaGetLastError();
}

// r = z - A x with the FP64 operator and the precomputed diagonal; L∞(r), as the bit pattern of |r|,
// into *dlinf
static void true_residual(PoissonMG* mg, const Grid& g, const double* L, const double* zz, const double* xv,
                          unsigned long long* dlinf, cudaStream_t st, float* r32 = nullptr, float* e32 = nullptr) {
    unsigned long long* pmax = reinterpret_cast<unsigned long long*>(mg->partial);
    LAUNCH_TILE(g, true_resid_tile_k, g, L, mg->diag64, zz, xv, mg->r, pmax, r32, e32);
    { finalize_max_k<<<1, 1024, 0, st>>>(pmax, mg->mvb, dlinf); ia::note_launch(); }
}

static double read_linf(ia_handle* h, unsigned long long* dlinf) {
    unsigned long long v = 0;
    cudaMemcpyAsync(&h->mg->hsc[0], dlinf, 8, cudaMemcpyDeviceToHost, h->stream);
    cudaStreamSynchronize(h->stream);
    std::memcpy(&v, &h->mg->hsc[0], 8);
    double d;
    std::memcpy(&d, &v, 8);
    return d;
}

// Mixed precision: FP64 defect correction x += e, e from an inner flexible CG run
// entirely in FP32 (operator, preconditioner, vectors) on A e = r, started from the FP64
// true residual; inner dot products are block sums in FP32 reduced across blocks in
// FP64 and the CG scalars are FP64.  The inner preconditioner is the FP32 V-cycle
// (IA_POISSON_MIXED) or, for IA_POISSON_LEARNED, the mode set by ia_poisson_precond.
static int poisson_solve_mixed(ia_handle* h, double* xv, const double* zz, const double* L, double tol, int itmx,
                               int* iters, double* resid) {
    PoissonMG* mg = h->mg;
    cudaStream_t st = h->stream;
    const Grid& g = h->g;
    MGLevel& F = mg->lev[0];
    const long long N = g.N;
    unsigned long long* dlinf = reinterpret_cast<unsigned long long*>(mg->dsc + 8);
    double* hdots = mg->dsc + 12;                                  // hybrid n·t, n·An
    const bool learned = h->cfg.poisson_mode == IA_POISSON_LEARNED;
    // inner residual: the V-cycle reads its right-hand side from F.b32, so the plain mixed
    // mode keeps the residual there; the learned modes keep it apart
    float* rr = learned ? mg->rl32 : F.b32;
    int mode = learned ? mg->precond : IA_PRECOND_VCYCLE;
    auto vcyc = [&]() -> cudaError_t {
        const int tk = timing_begin(h, TK_MG_SMOOTH);
        const cudaError_t e = vcycle_run<float>(h, mg, st);
        timing_end(h, tk);
        mg->stats[1]++;
        return e;
    };
    auto net = [&](const float* in) -> bool {
        const int tk = timing_begin(h, TK_NN);
        const int rc = nn_apply(h, in, F.L32, mg->nl32, g.n[0] - 2, g.n[1] - 2, g.n[2] - 2, N);
        timing_end(h, tk);
        mg->stats[0]++;
        return rc == IA_OK;
    };
    // sv ≈ A⁻¹ rr
    auto precond = [&](float*& sv) -> bool {
        if (mode == IA_PRECOND_NONE) {
            sv = rr;
            return true;
        }
        if (mode == IA_PRECOND_NET) {
            sv = mg->nl32;
            return net(rr);
        }
        if (rr != F.b32) cudaMemcpyAsync(F.b32, rr, 4 * N, cudaMemcpyDeviceToDevice, st);
        sv = F.x32;
        if (vcyc() != cudaSuccess) return false;
        if (mode != IA_PRECOND_HYBRID) return true;
        // hybrid: the net corrects what the V-cycle left, s += ω net(t) with t = r - A s and
        // ω = (n·t)/(n·An), the energy-optimal step along n = net(t)
        int tk = timing_begin(h, TK_KRYLOV);
        if (g.D == 3) { residual_k<float, 3><<<cell_grid(g), blk(), 0, st>>>(g, F.L32, rr, F.x32, mg->t32); ia::note_launch(); }
        else { residual_k<float, 2><<<cell_grid(g), blk(), 0, st>>>(g, F.L32, rr, F.x32, mg->t32); ia::note_launch(); }
        timing_end(h, tk);
        if (!net(mg->t32)) return false;
        tk = timing_begin(h, TK_KRYLOV);
        LAUNCH_D(g, energy_dots_k, mg->kb, KTHREADS, g, F.L32, mg->nl32, mg->t32, mg->partial);
        { finalize_k<<<1, 1024, 0, st>>>(mg->partial, mg->kb, 2, hdots); ia::note_launch(); }
        { add_scaled_k<<<mg->kb, KTHREADS, 0, st>>>(g, hdots, mg->nl32, F.x32); ia::note_launch(); }
        timing_end(h, tk);
        return cudaGetLastError() == cudaSuccess;
    };
    int total = 0;
    int tk = timing_begin(h, TK_KRYLOV);
    // every FP64 residual also starts the next inner solve: rr = float(r), e32 = 0
    true_residual(mg, g, L, zz, xv, dlinf, st, rr, mg->e32);
    timing_end(h, tk);
    double res = read_linf(h, dlinf);
    while (!(res <= tol) && total < itmx) {
        const double target = std::fmax(0.5 * tol / res, mg->inner_rtol) * res;
        FcgDev* S = mg->fcg;
        // the reductions' last-block counters start from zero in every inner solve (each launch leaves
        // them at zero, but not one that an error cut short)
        cudaMemsetAsync(&S->done_dot, 0, 2 * sizeof(unsigned int), st);
        for (int it = 0; it < mg->inner_max && total < itmx; ++it) {
            float* sv = nullptr;
            if (!precond(sv)) return IA_ERR_CUDA;
            // β, the direction, q = A p, α and the update without a host round trip; one read-back of
            // the inner residual and the breakdown flag per step
            tk = timing_begin(h, TK_KRYLOV);
            { dot2_32_k<<<mg->vb, KTHREADS, 0, st>>>(N, sv, mg->q32, rr, mg->partial, S, it == 0 ? 1 : 0); ia::note_launch(); }
            { xpby32_k<<<mg->vb, KTHREADS, 0, st>>>(N, sv, S, mg->p32); ia::note_launch(); }
            auto matvec = [&](auto IX) {
                using I = decltype(IX);
                const unsigned gr = mv_blocks(g, mg->zt, mg->nsm);
                const Ends e = ends_of(g);
                if (g.D == 2) matvec32_tile_k<2, MV_ZT, I><<<gr, KTHREADS, 0, st>>>(g, e, F.L32, mg->p32, mg->q32, mg->partial, S);
                else if (mg->zt == 1) matvec32_tile_k<3, 1, I><<<gr, KTHREADS, 0, st>>>(g, e, F.L32, mg->p32, mg->q32, mg->partial, S);
                else matvec32_tile_k<3, MV_ZT, I><<<gr, KTHREADS, 0, st>>>(g, e, F.L32, mg->p32, mg->q32, mg->partial, S);
                ia::note_launch();
            };
            if (g.N < RB_CELLS) matvec(0u);
            else matvec(size_t(0));
            { update32_k<<<mg->vb, KTHREADS, 0, st>>>(N, S, mg->p32, mg->q32, mg->e32, rr); ia::note_launch(); }
            timing_end(h, tk);
            cudaMemcpyAsync(mg->hsc + 2, &S->rin, 8, cudaMemcpyDeviceToHost, st);
            if (cudaStreamSynchronize(st) != cudaSuccess) return IA_ERR_CUDA;
            unsigned int rin_bits = 0;
            int stop = 0;
            std::memcpy(&rin_bits, reinterpret_cast<const char*>(mg->hsc + 2), 4);
            std::memcpy(&stop, reinterpret_cast<const char*>(mg->hsc + 2) + 4, 4);
            ++total;
            mg->stats[3]++;
            if (stop) break;
            float rinf;
            std::memcpy(&rinf, &rin_bits, 4);
            if (double(rinf) <= target) break;
        }
        tk = timing_begin(h, TK_KRYLOV);
        LAUNCH_TILE(g, add_correction_k, g, mg->e32, xv);
        true_residual(mg, g, L, zz, xv, dlinf, st, rr, mg->e32);
        timing_end(h, tk);
        const double res_old = res;
        res = read_linf(h, dlinf);
        mg->stats[4]++;
        // fallback: a correction that fails to halve the FP64 true residual (or a net
        // kernel that reported a timeout) hands the rest of the solve to the V-cycle
        if (learned && mode != IA_PRECOND_VCYCLE && (!(res <= 0.5 * res_old) || nn_error_flag(h))) {
            mode = IA_PRECOND_VCYCLE;
            mg->stats[2]++;
        }
    }
    { perbc_k<<<unsigned((bc_plane_cells(g) + 255) / 256), 256, 0, st>>>(g, xv); ia::note_launch(); }
    if (cudaGetLastError() != cudaSuccess) return IA_ERR_CUDA;
    *iters = total;
    *resid = res;
    return (res <= tol) ? IA_OK : IA_WARN_NOT_CONVERGED;
}

// ---- the one-launch solver of small grids (poisson_cluster.cuh)
// Two-dimensional grids with an odd extent and a long side are solved on one level, by the coarsest level's sweeps, while
// one cluster holds them: these stop at the same residual as the multigrid with 10 to 20 times its error, on 161 x 97 cells
// up to 5e-9 of the pressure, and their results are to stay within 1e-9 of what they were.  (On sides of up to 96 cells,
// and on the three-dimensional grids that fit this path, the two are below 1e-9 apart, and the multigrid runs; it does on
// larger grids, too, and ends what one level does not: see poisson_solve.)  The rule asks for the grid alone: recording of
// times and the smoother's settings, which the coarsest level's sweeps don't have, change nothing.
// 161 x 97, mixed, a step: 249 ms with one block sweeping, 11.7 ms here, 1.9 ms with the multigrid.
static bool one_level(const Grid& g) {
    return g.D == 2 && ((g.n[0] & 1) || (g.n[1] & 1)) && std::max(g.n[0], g.n[1]) - 2 > 96 &&
           (long long)((g.n[0] - 1) / 2) * (g.n[1] - 2) <= (long long)CL_PAIRS * CL_MAX * TAIL_THREADS;
}

template <class T, int D>
static int cluster_blocks(PoissonMG* mg, long long pairs) {
    int& most = mg->cluster;   // the largest cluster that the device can place; -1: not asked yet
    if (most < 0) {
        int got = 0;
        const auto k = solve_cluster_k<T, D>;
        if (cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, CL_BYTES) == cudaSuccess &&
            cudaFuncSetAttribute(k, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) == cudaSuccess)
            for (int c = CL_MAX; c >= 1 && !got; c /= 2) {
                cudaLaunchConfig_t cfg = {};
                cudaLaunchAttribute at = {};
                at.id = cudaLaunchAttributeClusterDimension;
                at.val.clusterDim.x = c;
                at.val.clusterDim.y = at.val.clusterDim.z = 1;
                cfg.gridDim = dim3(c);
                cfg.blockDim = dim3(TAIL_THREADS);
                cfg.dynamicSmemBytes = CL_BYTES;
                cfg.attrs = &at;
                cfg.numAttrs = 1;
                int n = 0;
                if (cudaOccupancyMaxActiveClusters(&n, k, &cfg) == cudaSuccess && n >= 1) got = c;
            }
        cudaGetLastError();
        most = got;
    }
    return most >= 1 && pairs <= (long long)CL_PAIRS * most * TAIL_THREADS ? most : 0;
}

// the words of the levels above the tail and of its first one: pairs a thread keeps of each, offsets; bytes in all
template <int D>
static size_t cl_layout(const PoissonMG* mg, int nd, int C, int* kp, int* wo) {
    int off = 0;
    for (int l = 0; l <= nd; ++l) {
        const int share = (cl_pairs<D>(mg->lev[l].g) + C - 1) / C, k = (share + TAIL_THREADS - 1) / TAIL_THREADS;
        if (kp) {
            kp[l] = k;
            wo[l] = off;
        }
        off += k * CL_WORDS * TAIL_THREADS;
    }
    if (wo) wo[nd + 1] = off;
    return 4 * (size_t)off;
}

// Solves on the cluster path when it applies: *done says whether it did.  flat: on one level.
template <class T, int D>
static cudaError_t cluster_solve(ia_handle* h, bool flat, double* xv, const double* zz, const double* L, double tol, int itmx,
                                 int* iters, double* resid, bool* done) {
    PoissonMG* mg = h->mg;
    const Grid& g = h->g;
    *done = false;
    const long long cells = (long long)(g.n[0] - 2) * (g.n[1] - 2) * (D == 3 ? g.n[2] - 2 : 1);
    // (relaxation factor 1, at which the half-sweeps and the blocked smoother do the same arithmetic, stays on the
    // kernels that share it)
    if (!flat && (h->timing.on || mg->smoother != IA_SMOOTHER_HALFSWEEP || mg->omega == 1.0 || cells > cluster_cells<T>()))
        return cudaSuccess;
    if (sizeof(T) == 8 && !mg->lev[0].t) return cudaSuccess;
    const int lt = flat ? 0 : tail_level<T>(mg, cluster_tail_pairs<T>());
    const long long pairs = (long long)((g.n[0] - 1) / 2) * (g.n[1] - 2) * (D == 3 ? g.n[2] - 2 : 1);
    const int C = cluster_blocks<T, D>(mg, pairs);
    // (on one level the tail, which then has the coarsest level alone, is not used)
    const int l0 = flat ? mg->nlev - 1 : lt;
    if (!C || lt > CL_LEVELS || (mg->nlev > 1 && mg->lev[1].g.N > 0xFFFF) ||
        tail_layout<T>(mg, l0).bytes() + cl_layout<D>(mg, lt, C, nullptr, nullptr) > (size_t)CL_BYTES)
        return cudaSuccess;
    *done = true;
    mg->wrap_copies = true;
    SolveArgs<T> a;
    const size_t words = cl_layout<D>(mg, lt, C, a.kp, a.wo);
    a.tail = tail_args<T>(mg, l0, mg->nu1, mg->nu2, mg->nuc);
    a.nd = lt;
    a.flat = flat ? 1 : 0;
    for (int l = 0; l <= lt; ++l) {
        MGLevel& V = mg->lev[l];
        a.g[l] = V.g;
        a.x[l] = V.template x_<T>();
        a.b[l] = V.template b_<T>();
        a.L[l] = V.template L_<T>();
        a.iD[l] = V.template iD_<T>();
        if (l == lt) break;
        if constexpr (sizeof(T) == 8) a.r[l] = V.t;
        else a.r[l] = V.r32;
        a.nu1[l] = (l == 0 && mg->nu1f > 0) ? mg->nu1f : mg->nu1;
        a.nu2[l] = (l == 0 && mg->nu2f > 0) ? mg->nu2f : mg->nu2;
    }
    a.omega = T(mg->omega);
    if constexpr (sizeof(T) == 4) {
        a.p = mg->p32;
        a.q = mg->q32;
        a.e = mg->e32;
        a.L0 = mg->lev[0].L32;
    } else {
        a.p = mg->p;
        a.q = mg->q;
        a.e = nullptr;
        a.L0 = L;
    }
    a.xs = xv;
    a.z = zz;
    a.L64 = L;
    a.diag64 = mg->diag64;
    a.tol = tol;
    a.inner_rtol = mg->inner_rtol;
    a.inner_max = mg->inner_max;
    a.partial = mg->partial;
    a.out = reinterpret_cast<SolveOut*>(mg->dsc);
    // each level's window, where they fit beside the rest
    const int tops = lt + a.flat;
    size_t bytes = a.tail.bytes() + words;
    a.win[0] = -1;
    a.win_values = 0;
    if (D == 2 && bytes % sizeof(T) == 0) {
        int off = 0;
        for (int l = 0; l < tops && l < CL_LEVELS; ++l) {
            a.win[l] = off;
            int most = 0;
            for (int r = 0; r < C; ++r) {
                int lo, hi;
                cl_window<D>(a.g[l], C, r, lo, hi);
                most = std::max(most, hi - lo + 1);
            }
            off += most;
        }
        if (tops > 0 && bytes + sizeof(T) * (size_t)off <= (size_t)CL_BYTES) {
            a.win_values = off;
            bytes += sizeof(T) * (size_t)off;
        } else {
            a.win[0] = -1;
        }
    }
    cudaLaunchConfig_t cfg = {};
    cudaLaunchAttribute at = {};
    at.id = cudaLaunchAttributeClusterDimension;
    at.val.clusterDim.x = C;
    at.val.clusterDim.y = at.val.clusterDim.z = 1;
    cfg.gridDim = dim3(C);
    cfg.blockDim = dim3(TAIL_THREADS);
    cfg.dynamicSmemBytes = bytes;
    cfg.stream = h->stream;
    cfg.attrs = &at;
    cfg.numAttrs = 1;
    // at most CL_ITERATIONS a launch: a solve that is allowed any number of them and does not converge must not hold the
    // device in one kernel
    SolveOut o;
    *iters = 0;
    do {
        a.itmx = std::min(itmx - *iters, CL_ITERATIONS);
        const int tk = timing_begin(h, TK_MG_SMOOTH);   // (on one level: all of the solve)
        cudaError_t e = cudaLaunchKernelEx(&cfg, solve_cluster_k<T, D>, a);
        ia::note_launch();
        timing_end(h, tk);
        if (e == cudaSuccess) e = cudaMemcpyAsync(mg->hsc, a.out, sizeof(SolveOut), cudaMemcpyDeviceToHost, h->stream);
        if (e == cudaSuccess) e = cudaStreamSynchronize(h->stream);
        if (e != cudaSuccess) return e;
        std::memcpy(&o, mg->hsc, sizeof(o));
        mg->stats[1] += o.vcycles;
        if (sizeof(T) == 4) {
            mg->stats[3] += o.total;
            mg->stats[4] += o.outer;
        }
        *iters += o.total;
    } while (!(o.res <= tol) && *iters < itmx && o.total == a.itmx);   // (less: a breakdown)
    *resid = o.res;
    return cudaSuccess;
}

// r = z - A x over interior cells; L∞(r) to the host
int poisson_residual(ia_handle* h, double* r, const double* x, const double* z, const double* L, double* linf) {
    cudaStream_t st = h->stream;
    unsigned long long* d = reinterpret_cast<unsigned long long*>(h->dscalar + 60);
    cudaMemsetAsync(d, 0, 8, st);
    LAUNCH_D(h->g, true_resid_k, kblocks(h->g), KTHREADS, h->g, L, nullptr, z, x, r, d);
    unsigned long long v = 0;
    cudaMemcpyAsync(&v, d, 8, cudaMemcpyDeviceToHost, st);
    if (cudaStreamSynchronize(st) != cudaSuccess) return IA_ERR_CUDA;
    if (linf) std::memcpy(linf, &v, 8);
    return IA_OK;
}

// Solve A x = z to L∞(z - A x) <= tol (x holds the initial guess); L = μ₀.
// The many-launch solvers stream whole vectors, whose ghost entries have to be zero.  The one-launch solver keeps copies of
// cells across a wrap in the ghosts of x and takes them into p and e: they are cleared when the other form follows (a copy
// of an infinity or a NaN would otherwise stay in its sums for good).
static cudaError_t clear_wrap_copies(ia_handle* h) {
    PoissonMG* mg = h->mg;
    if (!mg->wrap_copies) return cudaSuccess;
    const bool fp64 = h->cfg.poisson_mode == IA_POISSON_FP64;
    cudaError_t e = cudaSuccess;
    auto clear = [&](void* v, size_t bytes) { e = e ? e : cudaMemsetAsync(v, 0, bytes, h->stream); };
    for (int l = 0; l < mg->nlev; ++l) {
        const size_t n = (size_t)mg->lev[l].g.N;
        if (fp64) clear(mg->lev[l].x, 8 * n);
        else clear(mg->lev[l].x32, 4 * n);
    }
    const size_t N = (size_t)h->g.N;
    if (fp64) {
        clear(mg->p, 8 * N);
    } else {
        clear(mg->p32, 4 * N);
        clear(mg->e32, 4 * N);
    }
    if (e == cudaSuccess) mg->wrap_copies = false;
    return e;
}

static cudaError_t one_launch_solve(ia_handle* h, bool flat, double* xv, const double* zz, const double* L, double tol, int itmx,
                                    int* iters, double* resid, bool* done) {
    if (h->cfg.poisson_mode == IA_POISSON_FP64)
        return h->g.D == 3 ? cluster_solve<double, 3>(h, flat, xv, zz, L, tol, itmx, iters, resid, done)
                           : cluster_solve<double, 2>(h, flat, xv, zz, L, tol, itmx, iters, resid, done);
    return h->g.D == 3 ? cluster_solve<float, 3>(h, flat, xv, zz, L, tol, itmx, iters, resid, done)
                       : cluster_solve<float, 2>(h, flat, xv, zz, L, tol, itmx, iters, resid, done);
}

// on the hierarchy, after mg_setup
static int hierarchy_solve(ia_handle* h, double* xv, const double* zz, const double* L, double tol, int itmx, int* iters,
                           double* resid) {
    PoissonMG* mg = h->mg;
    bool done = false;
    if (one_launch_solve(h, false, xv, zz, L, tol, itmx, iters, resid, &done) != cudaSuccess) return IA_ERR_CUDA;
    if (done) return (*resid <= tol) ? IA_OK : IA_WARN_NOT_CONVERGED;
    if (clear_wrap_copies(h) != cudaSuccess) return IA_ERR_CUDA;
    if (h->cfg.poisson_mode != IA_POISSON_FP64) return poisson_solve_mixed(h, xv, zz, L, tol, itmx, iters, resid);
    cudaStream_t st = h->stream;
    const Grid& g = h->g;
    unsigned long long* dlinf = reinterpret_cast<unsigned long long*>(mg->dsc + 8);
    MGLevel& F = mg->lev[0];
    // the residual is the V-cycle's right-hand side and the preconditioned residual its result, in place
    double* r = mg->r;
    int tk = timing_begin(h, TK_KRYLOV);
    true_residual(mg, g, L, zz, xv, dlinf, st);
    timing_end(h, tk);
    double res = read_linf(h, dlinf);
    FcgDev* S = mg->fcg;
    cudaMemsetAsync(&S->done_dot, 0, 2 * sizeof(unsigned int), st);   // as in poisson_solve_mixed
    int it = 0;
    while (!(res <= tol) && it < itmx) {
        tk = timing_begin(h, TK_MG_SMOOTH);
        const cudaError_t e = vcycle_run<double>(h, mg, st);
        timing_end(h, tk);
        if (e != cudaSuccess) return IA_ERR_CUDA;
        // flexible CG: β = s_k·(r_k - r_{k-1}) / (s_{k-1}·r_{k-1}) with r_k - r_{k-1} = -α q_{k-1}
        tk = timing_begin(h, TK_KRYLOV);
        { dot2_64_k<<<mg->vb, KTHREADS, 0, st>>>(g.N, F.x, mg->q, r, mg->partial, S, it == 0 ? 1 : 0); ia::note_launch(); }
        { xpby64_k<<<mg->vb, KTHREADS, 0, st>>>(g.N, F.x, S, mg->p); ia::note_launch(); }
        {
            // (never more blocks than the 32 x 8 tiles that the partials are allocated for)
            const dim3 gr(plane_grid<double>(g.n[0] - 2, g.n[1] - 2, mv_tile_grid(g, mg->zt).z));
            if (g.D == 2) matvec64_k<2, MV_ZT><<<gr, KTHREADS, 0, st>>>(g, L, mg->diag64, mg->p, mg->q, mg->partial, S);
            else if (mg->zt == 1) matvec64_k<3, 1><<<gr, KTHREADS, 0, st>>>(g, L, mg->diag64, mg->p, mg->q, mg->partial, S);
            else matvec64_k<3, MV_ZT><<<gr, KTHREADS, 0, st>>>(g, L, mg->diag64, mg->p, mg->q, mg->partial, S);
            ia::note_launch();
        }
        { update64_k<<<mg->vb, KTHREADS, 0, st>>>(g.N, S, mg->p, mg->q, xv, r); ia::note_launch(); }
        timing_end(h, tk);
        cudaMemcpyAsync(mg->hsc + 2, &S->rin64, 16, cudaMemcpyDeviceToHost, st);
        if (cudaStreamSynchronize(st) != cudaSuccess) return IA_ERR_CUDA;
        int stop = 0;
        std::memcpy(&stop, reinterpret_cast<const char*>(mg->hsc + 3) + offsetof(FcgDev, stop) - offsetof(FcgDev, rin), 4);
        if (stop) break;
        std::memcpy(&res, mg->hsc + 2, 8);
        ++it;
    }
    { perbc_k<<<unsigned((bc_plane_cells(g) + 255) / 256), 256, 0, st>>>(g, xv); ia::note_launch(); }
    if (cudaGetLastError() != cudaSuccess) return IA_ERR_CUDA;
    *iters = it;
    *resid = res;
    return (res <= tol) ? IA_OK : IA_WARN_NOT_CONVERGED;
}

int poisson_solve(ia_handle* h, double* xv, const double* zz, const double* L, double tol, int itmx, int* iters,
                  double* resid) {
    if (!h->mg) return IA_ERR_INVALID;
    if (mg_setup(h, L) != cudaSuccess) return IA_ERR_CUDA;
    if (h->cfg.poisson_mode == IA_POISSON_LEARNED) return poisson_solve_mixed(h, xv, zz, L, tol, itmx, iters, resid);
    if (!one_level(h->g)) return hierarchy_solve(h, xv, zz, L, tol, itmx, iters, resid);
    // A solve that three quarters of its iterations on one level do not end goes on with the hierarchy from there (density
    // ratio 1000, mixed, to 1e-10: 161 x 97 cells take 2247 iterations of one level, 255 x 255 more than 20000).
    bool done = false;
    if (one_launch_solve(h, true, xv, zz, L, tol, itmx - itmx / 4, iters, resid, &done) != cudaSuccess) return IA_ERR_CUDA;
    if (done && (*resid <= tol || *iters >= itmx)) return (*resid <= tol) ? IA_OK : IA_WARN_NOT_CONVERGED;
    const int used = done ? *iters : 0;
    const int rc = hierarchy_solve(h, xv, zz, L, tol, itmx - used, iters, resid);
    *iters += used;
    return rc;
}

}  // namespace ia
