// Direction-split conservative VOF advection (InterfaceAdvection.jl
// src/advection.jl:17-137 with src/normalEstimation.jl and src/PLIC.jl).
//
// One sweep along d updates f in place, like the reference.  Only interface
// cells change; their new values are staged in a compact buffer and written
// back after every read of the old field has finished.  A sweep is four
// kernels:
//
//  * vof_bulk — one thread per cell of the ghost-inclusive box.  A cell whose
//    three cells along d are all full or all empty, equal to its c̄, and whose
//    face velocities satisfy |u|·δt <= 1/2 leaves the sweep unchanged after
//    cleanWisp!: the face fluxes f·δl and the dilation term cancel to within
//    ~1e-15 < 10 eps.  Those cells are decided with integer compares on the
//    IEEE bit patterns only: on GB300 every FP64 instruction, compares
//    included, issues at 1/64 of the FP32 rate, so the bulk path spends FP64
//    only on the mass flux ρuf.  Cells that need the full update go to a cell
//    list; faces whose donor cell must be reconstructed go to a face list.
//  * vof_faces — one thread per listed face: donor reconstruction (normal
//    scheme + PLIC intercept) and the PLIC slab volume, computed once per face
//    and cached; the face's mass flux ρuf.
//  * vof_cells — one thread per listed cell: the conservative update with the
//    dilation term from the two face fluxes, the fill-error status,
//    cleanWisp!, staged in vals[k].
//  * vof_scatter — f[list[k]] = vals[k].
//
// Ghost cells take the value of their boundary-condition source cell in the
// same sweep, so f leaves the sweep with BCf! applied (src/VOFutil.jl:64-75)
// and the next sweep reads valid ghosts.
#include <cuda_runtime.h>

#include "ff.cuh"
#include "ia_core.cuh"
#include "ia_geom.cuh"
#include "vof.cuh"

namespace ia {

namespace {

constexpr unsigned long long ONE_BITS = 0x3FF0000000000000ull;   // 1.0

__device__ __forceinline__ unsigned long long bits(double v) { return (unsigned long long)__double_as_longlong(v); }
// |v| <= limit, decided on the bit pattern (false for inf / NaN)
__device__ __forceinline__ bool abs_le(double v, unsigned long long lim_bits) { return abs_bits(v) <= lim_bits; }
__device__ __forceinline__ bool is_zero(double v) { return abs_bits(v) == 0ull; }
// v < 1/2 (false for NaN)
__device__ __forceinline__ bool below_half(double v) {
    const unsigned long long b = bits(v);
    return abs_bits(v) <= 0x7FF0000000000000ull && ((b >> 63) || b < 0x3FE0000000000000ull);
}
// f ∈ {+0, 1} exactly
__device__ __forceinline__ bool is_bulk(unsigned long long b) { return b == 0ull || b == ONE_BITS; }

__device__ __forceinline__ double mass_flux(double dl, double F, double lrho) {
    return dl * lrho + (1.0 - lrho) * F;   // fᶠ2ρuf, src/VOFutil.jl:218
}

// getVOFFlux! for one face K whose donor needs reconstruction
// (src/advection.jl:113-137); dl = δt/2 (u1 + u2) is passed in.
template <int D>
__device__ double face_flux_recon(const SweepArgs& a, long long K, int kd, double dl) {
    const long long sd = a.g.s[a.d];
    const bool pos = dl > 0.0;
    const long long C = pos ? K - sd : K;
    const int cd = pos ? kd - 1 : kd;
    const double fC = a.fin[C];
    const int nd = a.g.n[a.d];
    const bool ghost = (cd == 0) || (cd == nd - 1);
    long long R = C;   // periodic ghost donors carry their image's reconstruction (BCVOF!)
    if (ghost) R = (cd == 0) ? C + (long long)(nd - 2) * sd : C - (long long)(nd - 2) * sd;
    Stencil S;
    S.f = a.fin;
    S.c = R;
    S.s[0] = a.g.s[0];
    S.s[1] = a.g.s[1];
    S.s[2] = a.g.s[2];
    double n[3];
    interface_normal<D>(a.scheme, S, n);
    double sa = fabs(n[0]) + fabs(n[1]);
    if (D == 3) sa += fabs(n[2]);
    if (sa == 0.0) return fC * dl;
    const double alpha = get_intercept<D>(n, fC);
    const double b = pos ? alpha - n[a.d] * (1.0 - dl) : alpha;
    n[a.d] *= fabs(dl);
    return get_volume_fraction<D>(n, b) * dl;
}

// Does face K (d-coordinate kd) need the donor reconstruction?  Returns false
// and the flux when the donor is full/empty or a zero-gradient ghost (whose
// α, n̂ the reference never reconstructs: the Σ|n̂| = 0 branch).
__device__ __forceinline__ bool face_simple(const SweepArgs& a, long long K, int kd, double& dl, double& F) {
    const long long sd = a.g.s[a.d];
    dl = a.h * (a.u1[K] + a.u2[K]);
    const unsigned long long db = bits(dl);
    if (is_zero(dl)) {   // δl == 0: no flux, ρuf untouched
        F = 0.0;
        return true;
    }
    const bool pos = !(db >> 63);
    const long long C = pos ? K - sd : K;
    const int cd = pos ? kd - 1 : kd;
    const double fC = a.fin[C];
    const unsigned long long fb = bits(fC);
    const bool zg_ghost = ((cd == 0) || (cd == a.g.n[a.d] - 1)) && !a.g.isper(a.d);
    if (is_bulk(fb)) {
        F = (fb == ONE_BITS) ? dl : 0.0 * dl;
        return true;
    }
    if (zg_ghost || fC == 0.0 || fC == 1.0) {   // -0, or a mixed zero-gradient ghost donor
        F = fC * dl;
        return true;
    }
    return false;
}

// Mass flux ρuf of face K when its donor is full, empty or a zero-gradient
// ghost: with s = u1 + u2 and δl = s·δt/2 the reference's δl λρ + (1-λρ) fᶠ
// is δl for a full donor and δl λρ for an empty one (two FP64 operations;
// the products are re-associated, a relative change below 1e-15).  Returns
// false when the donor needs reconstruction.
__device__ __forceinline__ bool face_mass_simple(const SweepArgs& a, long long K, int kd, double s, double& m) {
    // s = u1[K] + u2[K]
    const long long sd = a.g.s[a.d];
    const unsigned long long sb = bits(s);
    if (is_zero(s)) {   // δl == 0: ρuf stays 0
        m = 0.0;
        return true;
    }
    const bool pos = !(sb >> 63);
    const long long C = pos ? K - sd : K;
    const int cd = pos ? kd - 1 : kd;
    const double fC = a.fin[C];
    const unsigned long long fb = bits(fC);
    if (fb == ONE_BITS) { m = a.h * s; return true; }
    if (fb == 0ull) { m = a.hl * s; return true; }
    const bool zg_ghost = ((cd == 0) || (cd == a.g.n[a.d] - 1)) && !a.g.isper(a.d);
    if (zg_ghost || fC == 0.0 || fC == 1.0) {
        const double dl = a.h * s;
        m = dl * a.lrho + a.one_m_lrho * (fC * dl);
        return true;
    }
    return false;
}

// u1[K] + u2[K] for the rare faces whose sum the caller has not formed (out of line: a call is not
// if-converted into the common path)
__device__ __noinline__ double face_sum_cold(const double* u1, const double* u2, long long K) { return u1[K] + u2[K]; }

template <int D>
__device__ __forceinline__ void coords_of(const Grid& g, long long O, int c[3]) {
    c[0] = int(O % g.n[0]);
    const long long r = O / g.n[0];
    c[1] = int(r % g.n[1]);
    c[2] = (D == 3) ? int(r / g.n[1]) : 0;
}

template <int D>
__device__ __forceinline__ bool in_face_range(const Grid& g, int d, const int c[3]) {
#pragma unroll
    for (int e = 0; e < D; ++e) {
        const int hi = (e == d) ? g.n[e] - 1 : g.n[e] - 2;
        if (c[e] < 1 || c[e] > hi) return false;
    }
    return true;
}

__device__ __forceinline__ void warp_append(unsigned int* list, unsigned int* count, bool pred, unsigned int val) {
    const unsigned int mask = __ballot_sync(0xFFFFFFFFu, pred);
    if (!mask) return;
    const int lane = threadIdx.x & 31;   // blocks are 32 wide in x: one warp per row
    const int leader = __ffs(mask) - 1;
    unsigned int base = 0;
    if (lane == leader) base = atomicAdd(count, (unsigned int)__popc(mask));
    base = __shfl_sync(0xFFFFFFFFu, base, leader);
    if (pred) list[base + __popc(mask & ((1u << lane) - 1u))] = val;
}

// One lane's cell of a bulk pass (a lane without one comes along for the list appends, which are warp-collective)
template <int D, bool FIRST, bool DILA>
__device__ __forceinline__ void bulk_cell(const SweepArgs& a, int x, int y, int z, bool valid) {
    const Grid& g = a.g;
    bool need_cell = false, need_face = false;
    long long O = 0;
    if (valid) {
        O = lin(g, x, y, z);
        const int c[3] = {x, y, z};
        const long long S = lin(g, bc_src(g, 0, x), bc_src(g, 1, y), D == 3 ? bc_src(g, 2, z) : 0);
        const long long sd = g.s[a.d];
        const unsigned long long bm = bits(a.fin[S - sd]), bc = bits(a.fin[S]), bp = bits(a.fin[S + sd]);
        int cb;
        if (FIRST) {
            // c̄ = f < 0.5 ? 0 : 1 over every cell (src/advection.jl:40), on the bit pattern
            a.cbar[O] = below_half(a.fin[O]) ? 0 : 1;
            cb = (bc == ONE_BITS) ? 1 : 0;          // only consulted when bc is bulk
        } else {
            cb = a.cbar[S];
        }
        const bool bulk = (bm == bc) && (bc == bp) && is_bulk(bc) && (cb == (bc == ONE_BITS ? 1 : 0)) &&
                          abs_le(a.u1[S], a.ulim) && abs_le(a.u1[S + sd], a.ulim) &&
                          abs_le(a.u2[S], a.ulim) && abs_le(a.u2[S + sd], a.ulim);
        need_cell = !bulk;
        double sS = 0.0;   // u1[S] + u2[S]: the dilation difference's and an interior face's mass flux sum
        if (DILA) {
            // the momentum update's dilation term of this (ghost-mapped) cell, on FP32 pairs: c̄ of the
            // source cell (in the first sweep from its fraction, as the c̄ pass above computes it)
            int cs;
            if (FIRST) cs = below_half(__longlong_as_double((long long)bc)) ? 0 : 1;
            else cs = cb;
            // the velocity difference in FP64 as (u1 + u2)(S + δd) − (u1 + u2)(S): the second sum is the face
            // mass flux's for an interior cell, so the cell issues two FP64 additions for both instead of
            // four (this pass is bound by its FP64 work), then one split and a pair product
            sS = a.u1[S] + a.u2[S];
            const double du = (a.u1[S + sd] + a.u2[S + sd]) - sS;
            const ff rq = cs ? ff{a.rq_1_hi, a.rq_1_lo} : ff{a.rq_l_hi, a.rq_l_lo};
            const ff dq = ff_mul(rq, ff_split(du));
            a.dila[O] = make_float2(dq.hi, dq.lo);
        }
        // in place a bulk cell keeps its value and only a stale ghost copy needs a write;
        // out of place (the coupled step keeps f_old) every bulk cell is written
        if (bulk && (a.fin != a.fout || ((O != S) && bits(a.fin[O]) != bc)))
            a.fout[O] = (bc == ONE_BITS) ? 1.0 : 0.0;
        if (in_face_range<D>(g, a.d, c)) {
            double m;
            const double sO = DILA ? (O == S ? sS : face_sum_cold(a.u1, a.u2, O)) : a.u1[O] + a.u2[O];
            if (face_mass_simple(a, O, c[a.d], sO, m)) {
                if (a.rhouf_d) a.rhouf_d[O] = m;
            } else {
                need_face = true;
            }
        } else if (a.rhouf_d) {
            a.rhouf_d[O] = 0.0;
        }
    }
    warp_append(a.list, a.list_count, valid && need_cell, (unsigned int)O);
    warp_append(a.flist, a.flist_count, valid && need_face, (unsigned int)O);
}

template <int D, bool FIRST, bool DILA>
__global__ void __launch_bounds__(256) vof_bulk(SweepArgs a) {
    // x in [1, n-2] one cell per lane, so that a row of 32k interior cells fills k warps; the
    // last block column's first warp takes the ghost cells x = 0 and n-1 of the block's 8 rows.
    const Grid& g = a.g;
    const bool gcol = blockIdx.x + 1 == gridDim.x;
    const int x = gcol ? ((threadIdx.x & 1) ? g.n[0] - 1 : 0) : 1 + int(blockIdx.x) * 32 + int(threadIdx.x);
    const int y = gcol ? int(blockIdx.y) * 8 + int(threadIdx.x >> 1) : int(blockIdx.y) * 8 + int(threadIdx.y);
    const bool valid = (gcol ? (threadIdx.y == 0 && threadIdx.x < 16) : x <= g.n[0] - 2) && y < g.n[1];
    bulk_cell<D, FIRST, DILA>(a, x, y, blockIdx.z, valid);
}

// ---- whole-call scan (3D advection alone): the full cells of a call in one pass
// Most tiles of a grid hold one fluid, and then nothing in them changes in any sweep: a cell changes in a sweep along d
// only if its two neighbours along d differ from it, every dimension is swept once a call, so by induction only if some
// cell of the 3 x 3 x 3 box around it (of the box around its source cell, for a ghost) differs from it in the field
// that the call starts from.  vof_scan writes what all sweeps would write into such a tile (ρuf along every direction,
// c̄) and lists the others; the sweeps' bulk passes then go through the listed tiles (vof_bulk_tiles).  A velocity above
// the bulk test's bound anywhere sends every tile to the sweeps.
// What bounds it: HBM and the FP64 pipe alike (81 B and 6 FP64 operations a cell for the three directions, 0.2 ms each
// at 256^3), and before them latency: a block's loads of f end at a barrier, so that eight blocks of 32 registers a
// thread beat four that load two planes of velocities at once (a call 527 us against 559).  A sphere in 256^3 cells:
// 856 us a call with a pass over the whole grid in each of the three sweeps, 527 us with the scan.
constexpr int VT_X = 32, VT_Y = 8, VT_Z = 8;
inline __host__ __device__ int tiles_of(int n, int t) { return (n + t - 1) / t; }
__device__ __forceinline__ void tile_origin(const Grid& g, int t, int& x0, int& y0, int& z0) {
    const int tx = tiles_of(g.n[0], VT_X), ty = tiles_of(g.n[1], VT_Y);
    x0 = t % tx * VT_X;
    t /= tx;
    y0 = t % ty * VT_Y;
    z0 = t / ty * VT_Z;
}

// The coordinates outside a tile [lo, hi] of dimension e whose cells its own can depend on: the one on either side; with
// the upper ghost in the tile the two below it (its source's neighbour; the ghost can have a tile to itself); with a
// periodic ghost in the tile or beside it the three around that ghost's source.  The k-th of them (at most 8).
__device__ __forceinline__ int tile_low(const Grid& g, int e, int lo, int hi) {
    return max(0, hi == g.n[e] - 1 ? min(lo - 1, g.n[e] - 3) : lo - 1);
}
__device__ __forceinline__ bool beside(const Grid& g, int e, int lo, int hi, int k, int& c) {
    const int low = tile_low(g, e, lo, hi);
    if (k < lo - low) { c = low + k; return true; }
    k -= lo - low;
    if (hi < g.n[e] - 1) {
        if (k == 0) { c = hi + 1; return true; }
        --k;
    }
    if (!g.isper(e)) return false;
    if (lo == 0) {
        if (k < 3) { c = g.n[e] - 3 + k; return true; }
        k -= 3;
    }
    if (hi >= g.n[e] - 2 && k < 3) { c = k; return true; }
    return false;
}

__global__ void __launch_bounds__(256, 8) vof_scan(ScanArgs a) {
    const Grid& g = a.g;
    int x0, y0, z0;
    tile_origin(g, blockIdx.x, x0, y0, z0);
    const int tid = threadIdx.x, tx = tid & 31, ty = tid >> 5, x = x0 + tx, y = y0 + ty;
    const int x1 = min(x0 + VT_X, g.n[0]) - 1, y1 = min(y0 + VT_Y, g.n[1]) - 1, z1 = min(z0 + VT_Z, g.n[2]) - 1;
    const long long s1 = g.s[1], s2 = g.s[2];
    const unsigned long long ref = bits(a.f[x0 + y0 * s1 + z0 * s2]);
    const int zl = tile_low(g, 2, z0, z1), zh = min(z1 + 1, g.n[2] - 1);
    bool same = is_bulk(ref);
    auto column = [&](int cx, int cy) {   // (cx, cy) at the tile's depths and those beside it
        const double* f = a.f + cx + cy * s1;
#pragma unroll 5
        for (int z = zl; z <= zh; ++z) same = same & (bits(f[z * s2]) == ref);
        if (g.isper(2)) {
            if (z0 == 0)
                for (int z = max(0, g.n[2] - 3); z < g.n[2]; ++z) same = same & (bits(f[z * s2]) == ref);
            if (z1 >= g.n[2] - 2)
                for (int z = 0; z < 3; ++z) same = same & (bits(f[z * s2]) == ref);
        }
    };
    if (x <= x1 && y <= y1) column(x, y);
    int cx, cy;
    if (ty < 2) {   // two warps: the tile's x in the rows beside it
        for (int k = ty; beside(g, 1, y0, y1, k, cy); k += 2)
            if (x <= x1) column(x, cy);
    } else if (ty < 6) {   // 128 threads: row q % 16 of column q / 16 beside it (rows 8-15: those beside the tile)
        const int q = tid - 64;
        for (int k = q >> 4; beside(g, 0, x0, x1, k, cx); k += 8) {
            if ((q & 15) < 8) {
                if (y0 + (q & 15) <= y1) column(cx, y0 + (q & 15));
            } else if (beside(g, 1, y0, y1, (q & 15) - 8, cy)) {
                column(cx, cy);
            }
        }
    }
    const bool uniform = __syncthreads_and(same);
    if (!uniform && tid == 0) a.tiles[atomicAdd(a.count, 1u)] = blockIdx.x;
    const bool one = ref == ONE_BITS;
    const double c = one ? a.h : a.hl;
    bool fast = true;
    if (x <= x1 && y <= y1) {
        const bool in_x = x >= 1 && x <= g.n[0] - 2, in_y = y >= 1 && y <= g.n[1] - 2;
        const bool lo_x = x >= 1, lo_y = y >= 1;
#pragma unroll 1
        for (int z = z0; z <= z1; ++z) {
            const long long I = x + y * s1 + z * s2;
            const bool in_z = z >= 1 && z <= g.n[2] - 2, lo_z = z >= 1;
            double p[3], q[3];
#pragma unroll
            for (int d = 0; d < 3; ++d) {
                p[d] = a.u1[I + d * g.N];
                q[d] = a.u2[I + d * g.N];
            }
#pragma unroll
            for (int d = 0; d < 3; ++d) fast = fast & abs_le(p[d], a.ulim) & abs_le(q[d], a.ulim);
            if (!uniform) continue;
            a.cbar[I] = one ? 1 : 0;
            if (!a.rhouf) continue;
#pragma unroll
            for (int d = 0; d < 3; ++d) {
                const bool face = (d == 0 ? lo_x : in_x) && (d == 1 ? lo_y : in_y) && (d == 2 ? lo_z : in_z);
                const double s = p[d] + q[d];
                a.rhouf[I + d * g.N] = face && !is_zero(s) ? c * s : 0.0;
            }
        }
    }
    if (!__syncthreads_and(fast) && tid == 0) atomicOr(a.above, 1u);
}

// the bulk pass of a sweep over the listed tiles (every tile when a velocity was above the bound), a plane at a time
template <bool FIRST>
__global__ void __launch_bounds__(256) vof_bulk_tiles(SweepArgs a) {
    const Grid& g = a.g;
    const bool every = *a.above != 0u;
    const long long n = every ? (long long)tiles_of(g.n[0], VT_X) * tiles_of(g.n[1], VT_Y) * tiles_of(g.n[2], VT_Z)
                              : (long long)*a.tile_count;
    for (long long k = blockIdx.x; k < n * VT_Z; k += gridDim.x) {
        int x0, y0, z0;
        tile_origin(g, every ? int(k / VT_Z) : int(a.tiles[k / VT_Z]), x0, y0, z0);
        const int x = x0 + int(threadIdx.x), y = y0 + int(threadIdx.y), z = z0 + int(k % VT_Z);
        if (z < g.n[2]) bulk_cell<3, FIRST, false>(a, x, y, z, x < g.n[0] && y < g.n[1]);
    }
}

template <int D>
// one warp a block: few warps have work, and this spreads them over the SMs (a sphere at 256^3: 540 us a call, 559 with four)
__global__ void __launch_bounds__(32) vof_faces(SweepArgs a) {
    const unsigned int count = *a.flist_count;
    for (unsigned int k = blockIdx.x * blockDim.x + threadIdx.x; k < count; k += gridDim.x * blockDim.x) {
        const long long K = a.flist[k];
        int c[3];
        coords_of<D>(a.g, K, c);
        const double dl = a.h * (a.u1[K] + a.u2[K]);
        const double F = face_flux_recon<D>(a, K, c[a.d], dl);
        a.flux[K] = F;
        if (a.rhouf_d) a.rhouf_d[K] = mass_flux(dl, F, a.lrho);
    }
}

template <int D, bool FIRST>
__global__ void __launch_bounds__(128) vof_cells(SweepArgs a) {
    const unsigned int count = *a.list_count;
    const Grid& g = a.g;
    const long long sd = g.s[a.d];
    for (unsigned int k = blockIdx.x * blockDim.x + threadIdx.x; k < count; k += gridDim.x * blockDim.x) {
        const long long O = a.list[k];
        int c[3];
        coords_of<D>(g, O, c);
        const int sc[3] = {bc_src(g, 0, c[0]), bc_src(g, 1, c[1]), D == 3 ? bc_src(g, 2, c[2]) : 0};
        const long long S = lin(g, sc[0], sc[1], sc[2]);
        double dl, F_lo, F_hi;
        if (!face_simple(a, S, sc[a.d], dl, F_lo)) F_lo = a.flux[S];
        if (!face_simple(a, S + sd, sc[a.d] + 1, dl, F_hi)) F_hi = a.flux[S + sd];
        const double fS = a.fin[S];
        const int cb = FIRST ? ((fS < 0.5) ? 0 : 1) : a.cbar[S];
        const double du = (a.u1[S + sd] - a.u1[S]) + (a.u2[S + sd] - a.u2[S]);
        double v = fS + ((F_lo - F_hi) + double(cb) * du * a.dt / 2.0);
        // reportFillError (src/advection.jl:145-189): judged before cleanWisp!
        if (O == S) {
            if (v != v) {
                atomicOr(&a.st->flags, IA_FLAG_NAN);
            } else if (v - 1.0 > a.tol_rep) {
                atomicOr(&a.st->flags, IA_FLAG_OVERFILL);
                atomicMax(&a.st->max_enc, ord_enc(v));
                const float e = float(v - 1.0);
                atomicMax(&a.st->max_key, ((unsigned long long)__float_as_uint(e) << 32) | (unsigned long long)O);
                a.st->dir = a.d;
            } else if (v < -a.tol_rep) {
                atomicOr(&a.st->flags, IA_FLAG_UNDERFILL);
                atomicMin(&a.st->min_enc, ord_enc(v));
                const float e = float(-v);
                atomicMax(&a.st->min_key, ((unsigned long long)__float_as_uint(e) << 32) | (unsigned long long)O);
                a.st->dir = a.d;
            }
        }
        // cleanWisp! (src/VOFutil.jl:127-136)
        v = (v < a.tol_clean) ? 0.0 : ((v > 1.0 - a.tol_clean) ? 1.0 : v);
        if (a.fin != a.fout) a.fout[O] = v;   // out of place nothing reads it in this sweep
        else a.vals[k] = v;
    }
}

__global__ void __launch_bounds__(256) vof_scatter(SweepArgs a) {
    const unsigned int count = *a.list_count;
    for (unsigned int k = blockIdx.x * blockDim.x + threadIdx.x; k < count; k += gridDim.x * blockDim.x)
        a.fout[a.list[k]] = a.vals[k];
}

template <int D, bool FIRST>
void launch_bulk(const SweepArgs& a, cudaStream_t st) {
    dim3 blk(32, 8, 1);
    dim3 grd((a.g.n[0] - 2 + 31) / 32 + 1, (a.g.n[1] + 7) / 8, a.g.n[2]);
    if (a.tiles) {
        if constexpr (D == 3) { vof_bulk_tiles<FIRST><<<a.tile_blocks, blk, 0, st>>>(a); ia::note_launch(); }
        return;
    }
    if (a.dila) { vof_bulk<D, FIRST, true><<<grd, blk, 0, st>>>(a); ia::note_launch(); }
    else { vof_bulk<D, FIRST, false><<<grd, blk, 0, st>>>(a); ia::note_launch(); }
}

}  // namespace

cudaError_t vof_sweep_bulk(const SweepArgs& a, cudaStream_t st) {
    if (a.g.D == 2) a.first ? launch_bulk<2, true>(a, st) : launch_bulk<2, false>(a, st);
    else a.first ? launch_bulk<3, true>(a, st) : launch_bulk<3, false>(a, st);
    return cudaGetLastError();
}

long long vof_tiles(const Grid& g) {
    return (long long)tiles_of(g.n[0], VT_X) * tiles_of(g.n[1], VT_Y) * tiles_of(g.n[2], VT_Z);
}
cudaError_t vof_scan_call(const ScanArgs& a, cudaStream_t st) {
    { vof_scan<<<unsigned(vof_tiles(a.g)), 256, 0, st>>>(a); ia::note_launch(); }
    return cudaGetLastError();
}

cudaError_t vof_sweep_faces(const SweepArgs& a, cudaStream_t st, int list_blocks) {
    if (a.g.D == 2) { vof_faces<2><<<list_blocks * 4, 32, 0, st>>>(a); ia::note_launch(); }
    else { vof_faces<3><<<list_blocks * 4, 32, 0, st>>>(a); ia::note_launch(); }
    return cudaGetLastError();
}

cudaError_t vof_sweep_scatter(const SweepArgs& a, cudaStream_t st, int list_blocks) {
    { vof_scatter<<<list_blocks / 2, 256, 0, st>>>(a); ia::note_launch(); }
    return cudaGetLastError();
}

cudaError_t vof_sweep_cells(const SweepArgs& a, cudaStream_t st, int list_blocks) {
    if (a.g.D == 2) {
        if (a.first) { vof_cells<2, true><<<list_blocks, 128, 0, st>>>(a); ia::note_launch(); }
        else { vof_cells<2, false><<<list_blocks, 128, 0, st>>>(a); ia::note_launch(); }
    } else {
        if (a.first) { vof_cells<3, true><<<list_blocks, 128, 0, st>>>(a); ia::note_launch(); }
        else { vof_cells<3, false><<<list_blocks, 128, 0, st>>>(a); ia::note_launch(); }
    }
    return cudaGetLastError();
}

}  // namespace ia
