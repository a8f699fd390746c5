// Level-set reinitialisation of src/redistaning.jl: ϕ = 2f - 1 (LevelSet, :13-25), the
// pseudo-time right-hand side L = ϕ_ini (1 - |∇ϕ|) with second-order ENO one-sided
// derivatives (computeL!, :64-83; ∇ϕᵢ², :118-143; the Neumann and periodic boundary
// building blocks :86-110), and the three-stage SSP Runge-Kutta march (redistaning!,
// :42-54; _redistaningStage!, :27-30) with BCf! ghosts after every stage.
//
// One kernel a stage: L, the stage update and the BCf! ghosts (an interior cell writes the ghosts that
// copy it).  The stages alternate between the field and two work arrays of the handle, so that no cell is
// overwritten while a neighbour still reads it.
//
// GB300 issues FP64 at 1/64 of the FP32 rate, compares included, so this is bound by FP64 instructions:
// every comparison is one of integers on the bit patterns (11 FP64 operations a direction remain, of about
// 24), and a direction whose five values are the same bits, or a cell whose gradient vanishes (the field away
// from the interface), takes none.  160 x 128 x 96, ten steps, on GB300: 13.8 ms with separate passes and FP64
// comparisons, 2.8 ms with the latter gone, 2.2 ms with absolute values off the FP64 pipe as well (abs_bits).
#include <cuda_runtime.h>

#include <cmath>

#include "capi_internal.cuh"
#include "ia_bc.cuh"

namespace ia {
namespace {

inline dim3 blk() { return dim3(32, 8, 1); }

constexpr unsigned long long kInfBits = 0x7FF0000000000000ull;

// |a| <= |b| ? a : b (b when either is NaN)
__device__ __forceinline__ double minmod(double a, double b) {
    const unsigned long long ka = abs_bits(a), kb = abs_bits(b);
    return ka <= kb && kb <= kInfBits ? a : b;
}

// The one-sided derivative whose square ∇ϕᵢ²(a,b,c,d,e,s) is (0 where neither side is upwind): ENO2
// (minmod-limited) derivatives dR, dL with w = s·d: dR where wR < 0 and wR + wL < 0, dL where wL > 0 and
// wR + wL > 0.  flip = the sign bit of s (s = ±1); the sign of a sum is that of the comparison with the
// negated term.
__device__ __forceinline__ double upwind(double a, double b, double c, double d, double e, long long flip) {
    // second differences as the reference rounds them, (c + a) - 2b: on two cells between walls two of them are
    // equal but for their rounding, which then decides the minmod
    const double m1 = fma(-2.0, b, c + a), m2 = fma(-2.0, c, d + b), m3 = fma(-2.0, d, e + c);
    const double dR = fma(-0.5, minmod(m3, m2), d - c), dL = fma(0.5, minmod(m2, m1), c - b);
    const double wR = __longlong_as_double(__double_as_longlong(dR) ^ flip);
    const double wL = __longlong_as_double(__double_as_longlong(dL) ^ flip);
    const long long kR = okey(wR), kN = ~okey(wL);   // ~: the key of -wL
    const bool num = abs_bits(dR) <= kInfBits && abs_bits(dL) <= kInfBits;
    const bool r_neg = __double_as_longlong(wR) < 0 && abs_bits(dR) != 0, l_pos = __double_as_longlong(wL) > 0;
    return num && r_neg && kR < kN ? dR : (num && l_pos && kR > kN ? dL : 0.0);
}

// L = ϕini (1 - sqrt(Σ_i ∇ϕᵢ²)) of an interior cell
template <int D>
__device__ __forceinline__ double rhs_cell(const Grid& g, const double* __restrict__ phi, double ini, int I, const int c[3]) {
    const double cc = phi[I];
    const long long kc = __double_as_longlong(cc), ki = __double_as_longlong(ini);
    if (abs_bits(ini) == 0 || abs_bits(ini) > kInfBits) {   // sign 0 (or NaN): no gradient
        return ini * 1.0;
    }
    const long long flip = ki & (1ll << 63);
    double acc = 0.0;
#pragma unroll
    for (int i = 0; i < D; ++i) {
        const int si = int(g.s[i]), ci = c[i], n = g.n[i];
        // beyond the ghost: the periodic image, or the ghost itself at a wall (lowerL!, upperL!)
        const int oa = ci != 1 ? -2 : (g.isper(i) ? n - 3 - ci : -1), oe = ci != n - 2 ? 2 : (g.isper(i) ? 2 - ci : 1);
        const double a = phi[I + oa * si], b = phi[I - si], d = phi[I + si], e = phi[I + oe * si];
        const bool flat = __double_as_longlong(a) == kc && __double_as_longlong(b) == kc && __double_as_longlong(d) == kc &&
                          __double_as_longlong(e) == kc && abs_bits(cc) < kInfBits;
        if (!flat) {
            const double u = upwind(a, b, cc, d, e, flip);
            acc = fma(u, u, acc);
        }
    }
    return __double_as_longlong(acc) == 0 ? ini : ini * (1.0 - sqrt(acc));
}

template <int D>
__device__ __forceinline__ bool interior_of_block(const Grid& g, int c[3], int& I) {
    c[0] = 1 + blockIdx.x * blockDim.x + threadIdx.x;
    c[1] = 1 + blockIdx.y * blockDim.y + threadIdx.y;
    c[2] = D == 3 ? 1 + int(blockIdx.z) : 0;
    I = c[0] + c[1] * int(g.s[1]) + c[2] * int(g.s[2]);
    return c[0] <= g.n[0] - 2 && c[1] <= g.n[1] - 2;
}
inline dim3 igrd(const Grid& g) {
    return dim3((g.n[0] - 2 + 31) / 32, (g.n[1] - 2 + 7) / 8, g.D == 3 ? g.n[2] - 2 : 1);
}

template <int D>
__global__ void __launch_bounds__(256) computeL_k(Grid g, const double* __restrict__ phi, const double* __restrict__ ini,
                                                  double* __restrict__ L) {
    int c[3], I;
    if (interior_of_block<D>(g, c, I)) L[I] = rhs_cell<D>(g, phi, ini[I], I, c);
}

// out = α ϕ⁰ + (1-α)(ϕ + dτ L(ϕ)) with BCf! ghosts; L is kept when Lout is given (the last stage of a march).
// out may be the array of ϕ⁰ (read only at the cell itself), not that of ϕ.
template <int D>
__global__ void __launch_bounds__(256) stage_k(Grid g, const double* __restrict__ phi, const double* phi0,
                                               const double* __restrict__ ini, double dtau, double alpha, double* out,
                                               double* __restrict__ Lout) {
    int c[3], I;
    if (!interior_of_block<D>(g, c, I)) return;
    const double L = rhs_cell<D>(g, phi, ini[I], I, c);
    if (Lout) Lout[I] = L;
    const double w = phi[I] + dtau * L, p0 = phi0[I];
    const double v = alpha == 0.0 && abs_bits(p0) < kInfBits ? w : alpha * p0 + (1.0 - alpha) * w;
    // the ghosts whose source cell this is: along each dimension the cell itself and perhaps one ghost
    int alt[3] = {0, 0, 0};   // offset to the ghost along e (0: none)
    bool edge = false;
#pragma unroll
    for (int e = 0; e < D; ++e) {
        const int n = g.n[e];
        if (c[e] == 1) alt[e] = (g.isper(e) ? n - 2 : -1) * int(g.s[e]);
        else if (c[e] == n - 2) alt[e] = (g.isper(e) ? 2 - n : 1) * int(g.s[e]);
        edge = edge || alt[e] != 0;
    }
    out[I] = v;
    if (!edge) return;
    for (int m = 1; m < (1 << D); ++m) {
        int o = I;
        bool ok = true;
        for (int e = 0; e < D; ++e)
            if ((m >> e) & 1) {
                ok = ok && alt[e] != 0;
                o += alt[e];
            }
        if (ok) out[o] = v;
    }
}

// ϕ = 2f - 1 and ϕini = ϕ on every cell (ghosts included, as the broadcast does)
__global__ void lsinit_k(long long n, const double* __restrict__ f, double* __restrict__ phi,
                         double* __restrict__ ini) {
    for (long long q = blockIdx.x * (long long)blockDim.x + threadIdx.x; q < n; q += (long long)gridDim.x * blockDim.x) {
        const double v = 2.0 * f[q] - 1.0;
        phi[q] = v;
        if (ini) ini[q] = v;
    }
}

}  // namespace
}  // namespace ia

using namespace ia;

extern "C" {

int ia_levelset_init(ia_handle* h, const double* f, double* phi, double* phi_ini) {
    if (!h || !f || !phi) return IA_ERR_INVALID;
    { lsinit_k<<<1216, 256, 0, h->stream>>>(h->g.N, f, phi, phi_ini); ia::note_launch(); }
    return cuda_fail(cudaGetLastError());
}

int ia_levelset_rhs(ia_handle* h, double* L, const double* phi, const double* phi_ini) {
    if (!h || !L || !phi || !phi_ini) return IA_ERR_INVALID;
    cudaMemsetAsync(L, 0, sizeof(double) * (size_t)h->g.N, h->stream);
    if (h->g.D == 3) computeL_k<3><<<igrd(h->g), blk(), 0, h->stream>>>(h->g, phi, phi_ini, L);
    else computeL_k<2><<<igrd(h->g), blk(), 0, h->stream>>>(h->g, phi, phi_ini, L);
    ia::note_launch();
    return cuda_fail(cudaGetLastError());
}

int ia_redistance(ia_handle* h, double* phi, double* phi0, const double* phi_ini, double* L, double d, double dtau) {
    if (!h || !phi || !phi0 || !phi_ini || !L || !(dtau > 0.0) || !(d >= 0.0)) return IA_ERR_INVALID;
    const Grid& g = h->g;
    cudaStream_t st = h->stream;
    const long long itmx = std::llrint(d / dtau);   // Julia round: nearest, ties to even
    const double alphas[3] = {0.0, 3.0 / 4.0, 1.0 / 3.0};
    cudaMemsetAsync(L, 0, sizeof(double) * (size_t)g.N, st);
    for (long long it = 0; it < itmx; ++it) {
        const bool last = it + 1 == itmx;
        if (last) cudaMemcpyAsync(phi0, phi, sizeof(double) * (size_t)g.N, cudaMemcpyDeviceToDevice, st);
        // ϕ → tmp1 → flux → ϕ (ϕ itself is ϕ⁰ until its last stage writes it)
        const double* in[3] = {phi, h->tmp1, h->flux};
        double* out[3] = {h->tmp1, h->flux, phi};
        for (int k = 0; k < 3; ++k) {
            double* Lk = last && k == 2 ? L : nullptr;
            if (g.D == 3) stage_k<3><<<igrd(g), blk(), 0, st>>>(g, in[k], phi, phi_ini, dtau, alphas[k], out[k], Lk);
            else stage_k<2><<<igrd(g), blk(), 0, st>>>(g, in[k], phi, phi_ini, dtau, alphas[k], out[k], Lk);
            ia::note_launch();
        }
    }
    return cuda_fail(cudaGetLastError());
}

}  // extern "C"
