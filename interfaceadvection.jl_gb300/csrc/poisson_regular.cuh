// FP32 smoother, residual restriction and matrix product of 3D levels that halve evenly, included by poisson.cu.
//
// What bounds the general kernels (rbgs_pair_k and the others) on such levels: instructions, not HBM.  An update of six
// neighbours issued 166 instructions for its 14 loads and 30 floating-point operations, and took the same time a cell
// whether the level lies in L2 or not.  On a level whose coarse cells cover two fine ones along each dimension every
// extent is even, so that a pair of cells lies inside as a whole and a pair of planes too, only a pair's outer
// neighbour can lie across a wrap, and at a wall the ghost cells hold zeros and need no case of their own; and below
// 2^30 cells an array is addressed by a 32-bit byte offset that all arrays of an element size share.  The values are
// those of the general kernels, operation for operation.  Time of a launch, general and here: first half-sweep from zero
// 172 and 129 us at 256x512x256, 24.7 and 17.9 at 128x192x160; of a post-smoothing 178 and 132, 25.1 and 13.5; half-sweep
// 106 and 109 (bound by HBM), 11.9 and 9.5; restriction 131 and 127, 12.8 and 12.4.
constexpr long long RB_CELLS = 1ll << 30;

// base[cell + k]; IX: unsigned below RB_CELLS cells, else size_t
template <class V, class IX>
__device__ __forceinline__ V at(const V* base, IX cell, int k = 0) {
    return *(const V*)((const char*)base + cell * (IX)sizeof(V) + k * (int)sizeof(V));
}

// distances to the lower and upper neighbour of the first and last interior cell of each dimension: across the wrap, or
// to the ghost cell
struct Ends {
    int lo[3], hi[3];
};
inline Ends ends_of(const Grid& g) {
    Ends e;
    for (int d = 0; d < 3; ++d) {
        const int s = int(g.s[d]);
        e.lo[d] = g.isper(d) ? (g.n[d] - 3) * s : -s;
        e.hi[d] = g.isper(d) ? (3 - g.n[d]) * s : s;
    }
    return e;
}

template <class TL>
struct RbArgs {
    int n0, n1, n2, s1, s2;      // extents with ghosts, strides
    long long N;
    Ends e, ec;                  // of the level and of the coarse one
    int c1, c2;                  // strides of the coarse level
    int y0, y1;                  // rows [y0, y1) of the interior (coarse rows in the restriction)
    int color;
    float omega;
    int write_red;
    const TL* L;
    const float *b, *iD, *xc;
    float* x;
};

// D_I x = b - off with rbgs_pair_k's order of operations
struct Star {
    float off, dd;
};
template <int D = 3, class TL, class IX>
__device__ __forceinline__ Star star7(const TL* __restrict__ L, long long N, IX I, int s1, int s2, float vxl, float vxh,
                                      float vyl, float vyh, float vzl, float vzh) {
    const TL* L1 = L + N;
    const TL* L2 = L1 + N;
    const float xl = cf(at(L, I)), xh = cf(at(L, I, 1)), yl = cf(at(L1, I)), yh = cf(at(L1, I + s1));
    Star s;
    s.off = xl * vxl + xh * vxh;
    s.off += yl * vyl + yh * vyh;
    s.dd = 0.f;
    s.dd -= xl + xh;
    s.dd -= yl + yh;
    if (D == 3) {
        const float zl = cf(at(L2, I)), zh = cf(at(L2, I + s2));
        s.off += zl * vzl + zh * vzh;
        s.dd -= zl + zh;
    }
    return s;
}
__device__ __forceinline__ float gauss_seidel(const Star& s, float b) {
    const float iD = (s.dd * s.dd < 2.f * 1.1920929e-7f) ? 0.f : 1.f / s.dd;
    return (b - s.off) * iD;
}

// rbgs_pair_k: the pair's cell of the colour in two planes, both planes' operands before the first store
template <class TL, bool PROL>
__global__ void __launch_bounds__(256, 8) rb_half_k(RbArgs<TL> a) {
    const int y = a.y0 + int(blockIdx.y) * 8 + int(threadIdx.y);
    const int x0 = 1 + 2 * (int(blockIdx.x) * 32 + int(threadIdx.x)), z0 = 1 + 2 * int(blockIdx.z);
    if (y >= a.y1 || x0 > a.n0 - 3) return;
    const float* xv = a.x;
    const int e0 = ((x0 + y + z0) & 1) == a.color ? 0 : 1;
    const int ol = x0 == 1 ? a.e.lo[0] : -1, oh = x0 == a.n0 - 3 ? a.e.hi[0] : 1;   // the pair's outer neighbours
    const int yl = y == 1 ? a.e.lo[1] : -a.s1, yh = y == a.n1 - 2 ? a.e.hi[1] : a.s1;
    const unsigned I0 = x0 + y * a.s1 + z0 * a.s2;
    unsigned I[2];
    Star s[2];
    float b[2], xo[2];
#pragma unroll
    for (int k = 0; k < 2; ++k) {
        const int e = k ? 1 - e0 : e0;
        const int zl = k == 0 && z0 == 1 ? a.e.lo[2] : -a.s2, zh = k == 1 && z0 == a.n2 - 3 ? a.e.hi[2] : a.s2;
        I[k] = I0 + e + k * a.s2;
        s[k] = star7(a.L, a.N, I[k], a.s1, a.s2, at(xv, I[k] + (e ? -1 : ol)), at(xv, I[k] + (e ? oh : 1)), at(xv, I[k] + yl), at(xv, I[k] + yh),
                     at(xv, I[k] + zl), at(xv, I[k] + zh));
        b[k] = at(a.b, I[k]);
        xo[k] = at(xv, I[k]);
        if (PROL) xo[k] += at(a.xc, ((x0 + 1) >> 1) + ((y + 1) >> 1) * a.c1 + ((z0 + k + 1) >> 1) * a.c2);
    }
#pragma unroll
    for (int k = 0; k < 2; ++k) {
        const float gs = gauss_seidel(s[k], b[k]);
        a.x[I[k]] = a.omega == 1.f ? gs : xo[k] + a.omega * (gs - xo[k]);
    }
}

// rbgs_first_k
template <class TL, bool PROL>
__global__ void __launch_bounds__(256) rb_first_k(RbArgs<TL> a) {
    const int y = a.y0 + int(blockIdx.y) * 8 + int(threadIdx.y);
    const int x0 = 1 + 2 * (int(blockIdx.x) * 32 + int(threadIdx.x)), z = 1 + int(blockIdx.z);
    if (y >= a.y1 || x0 > a.n0 - 3) return;
    const float* xv = a.x;
    const int e = (x0 + y + z) & 1 ? 0 : 1;   // the pair's black cell; the other is red
    const int ol = x0 == 1 ? a.e.lo[0] : -1, oh = x0 == a.n0 - 3 ? a.e.hi[0] : 1;
    const int yl = y == 1 ? a.e.lo[1] : -a.s1, yh = y == a.n1 - 2 ? a.e.hi[1] : a.s1;
    const int zl = z == 1 ? a.e.lo[2] : -a.s2, zh = z == a.n2 - 2 ? a.e.hi[2] : a.s2;
    const unsigned I = x0 + e + y * a.s1 + z * a.s2, Ir = I + (e ? -1 : 1), Io = I + (e ? oh : ol);
    float vr, vo, vyl, vyh, vzl, vzh, xo = 0.f;   // the pair's red cell, its outer neighbour, and along y and z
    if (PROL) {
        // a pair has one parent, and of the neighbours along a dimension one shares it
        const unsigned P = ((x0 + 1) >> 1) + ((y + 1) >> 1) * a.c1 + ((z + 1) >> 1) * a.c2;
        const float pc = at(a.xc, P);
        const float px = at(a.xc, P + (e ? (x0 == a.n0 - 3 ? a.ec.hi[0] : 1) : (x0 == 1 ? a.ec.lo[0] : -1)));
        const float py = at(a.xc, P + (y & 1 ? (y == 1 ? a.ec.lo[1] : -a.c1) : (y == a.n1 - 2 ? a.ec.hi[1] : a.c1)));
        const float pz = at(a.xc, P + (z & 1 ? (z == 1 ? a.ec.lo[2] : -a.c2) : (z == a.n2 - 2 ? a.ec.hi[2] : a.c2)));
        vr = at(xv, Ir) + pc;
        vo = at(xv, Io) + px;
        vyl = at(xv, I + yl) + (y & 1 ? py : pc);
        vyh = at(xv, I + yh) + (y & 1 ? pc : py);
        vzl = at(xv, I + zl) + (z & 1 ? pz : pc);
        vzh = at(xv, I + zh) + (z & 1 ? pc : pz);
        xo = at(xv, I) + pc;
    } else {
        auto red = [&](unsigned J) {   // the red value after the first red half-sweep from zero
            const float v = at(a.b, J) * at(a.iD, J);
            return a.omega == 1.f ? v : a.omega * v;
        };
        vr = red(Ir);
        vo = red(Io);
        vyl = red(I + yl);
        vyh = red(I + yh);
        vzl = red(I + zl);
        vzh = red(I + zh);
        if (a.write_red) a.x[Ir] = vr;
    }
    const Star s = star7(a.L, a.N, I, a.s1, a.s2, e ? vr : vo, e ? vo : vr, vyl, vyh, vzl, vzh);
    const float gs = gauss_seidel(s, at(a.b, I));
    a.x[I] = a.omega == 1.f ? gs : (PROL ? xo + a.omega * (gs - xo) : a.omega * gs);
}

// resid_restrict_k; bc: the coarse right-hand side
template <class TL>
__global__ void __launch_bounds__(256) rb_restrict_k(RbArgs<TL> a, float* __restrict__ bc) {
    const int xc = 1 + int(blockIdx.x) * 32 + int(threadIdx.x), yc = a.y0 + int(blockIdx.y) * 8 + int(threadIdx.y);
    const int zc = 1 + int(blockIdx.z);
    const int x0 = 2 * xc - 1, y0 = 2 * yc - 1, z0 = 2 * zc - 1;
    if (yc >= a.y1 || x0 > a.n0 - 3) return;
    const float* __restrict__ xv = a.x;
    const int xl = x0 == 1 ? a.e.lo[0] : -1, xh = x0 == a.n0 - 3 ? a.e.hi[0] : 1;
    const int yl = y0 == 1 ? a.e.lo[1] : -a.s1, yh = y0 == a.n1 - 3 ? a.e.hi[1] : a.s1;
    const int zl = z0 == 1 ? a.e.lo[2] : -a.s2, zh = z0 == a.n2 - 3 ? a.e.hi[2] : a.s2;
    const unsigned I0 = x0 + y0 * a.s1 + z0 * a.s2;
    // every value first, so that their loads are in flight together
    float v[2][2][4], vy[2][2][2], vz[2][2][2], b[2][2][2];   // rows along x with their ends; beyond them along y and z
#pragma unroll
    for (int k = 0; k < 2; ++k)
#pragma unroll
        for (int j = 0; j < 2; ++j) {
            const unsigned J = I0 + j * a.s1 + k * a.s2;
            v[k][j][0] = at(xv, J + xl);
            v[k][j][1] = at(xv, J);
            v[k][j][2] = at(xv, J, 1);
            v[k][j][3] = at(xv, J + 1 + xh);
#pragma unroll
            for (int i = 0; i < 2; ++i) {
                vy[k][j][i] = at(xv, J + (j ? yh : yl), i);
                vz[k][j][i] = at(xv, J + (k ? zh : zl), i);
                b[k][j][i] = at(a.b, J, i);
            }
        }
    float sum = 0.f;
#pragma unroll
    for (int k = 0; k < 2; ++k)
#pragma unroll
        for (int j = 0; j < 2; ++j)
#pragma unroll
            for (int i = 0; i < 2; ++i) {
                const Star s = star7(a.L, a.N, I0 + i + j * a.s1 + k * a.s2, a.s1, a.s2, v[k][j][i], v[k][j][i + 2],
                                     j ? v[k][0][i + 1] : vy[k][0][i], j ? vy[k][1][i] : v[k][1][i + 1],
                                     k ? v[0][j][i + 1] : vz[0][j][i], k ? vz[1][j][i] : v[1][j][i + 1]);
                sum += b[k][j][i] - (s.off + s.dd * v[k][j][i + 1]);
            }
    bc[xc + yc * a.c1 + zc * a.c2] = sum;
}

// the level's arguments; gc: the coarse level
template <class TL>
inline RbArgs<TL> rb_args(const Grid& g, const Grid& gc, const TL* L, const float* b, const float* iD, float* x, const float* xc,
                          float omega) {
    RbArgs<TL> a;
    a.n0 = g.n[0];
    a.n1 = g.n[1];
    a.n2 = g.n[2];
    a.s1 = int(g.s[1]);
    a.s2 = int(g.s[2]);
    a.N = g.N;
    a.e = ends_of(g);
    a.ec = ends_of(gc);
    a.c1 = int(gc.s[1]);
    a.c2 = int(gc.s[2]);
    a.y0 = 1;
    a.y1 = g.n[1] - 1;
    a.color = 0;
    a.omega = omega;
    a.write_red = 0;
    a.L = L;
    a.b = b;
    a.iD = iD;
    a.xc = xc;
    a.x = x;
    return a;
}
