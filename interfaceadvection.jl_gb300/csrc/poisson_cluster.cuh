// The whole pressure solve of a small grid in one launch (included by poisson.cu).
//
// One cluster of up to 16 blocks runs the solver's loop: the FP64 true residual, the (inner) flexible CG and its
// V-cycles, with a cluster barrier where the multi-launch solver starts another kernel, and the smallest levels in
// the first block's shared memory (tail_cycle).  The arithmetic is that of the multi-launch kernels; the finest
// level's half-sweeps read the FP32 coefficients.  The scalars are formed by every block from the same partial sums
// in the same order, so all blocks take the same branches.
//
// What bounds it: 25 to 60 dependent stages an iteration.  A stage is a launch of 2 to 3 us in a graph and 1 to 2 us
// here: 0.6 us for the stores to reach L2 before the barrier, 0.1 us the barrier of 16 blocks, 0.3 us the loads after
// it.  On larger grids the 16 multiprocessors are slower than the device (measured both ways: see cluster_cells).
#pragma once
#include <cooperative_groups.h>

namespace ia {
namespace {

constexpr int CL_MAX = 16;        // blocks of a cluster
constexpr int CL_PAIRS = 2;       // pairs of cells a thread keeps on a level
enum { PRE, POST, FLAT };
constexpr int CL_LEVELS = 4;      // levels above the tail
constexpr int CL_WORDS = TAIL_WORDS + 1;   // a pair's words: tail_words', and the blocks whose windows hold its cells

// Pairs of a level are dealt to the blocks in order, equally many each.  In 2D a block keeps x of a level above the tail
// in shared memory, in a window that its neighbours write directly, so that a stage has no store that must reach L2
// before the barrier and no load from there after it: a step of 161 x 97 cells on one level 14.1 -> 11.8 ms, in FP64
// 12.2 -> 9.2.  In 3D a block's two planes are all in the neighbours' windows, and L2 is the faster way (a solve of
// 32 x 64 x 32 cells 1404 us, with windows 1531).  A block's window
// is x on the rows [lo, hi] that its own cells and their neighbours span (whole rows: a cell's copies across a wrap in x
// lie in the windows that hold the cell).
template <int D>
__host__ __device__ inline int cl_pairs(const Grid& g) {
    return (g.n[0] - 1) / 2 * (g.n[1] - 2) * (D == 3 ? g.n[2] - 2 : 1);
}
template <int D>
__host__ __device__ inline int cl_cell(const Grid& g, int t) {   // first cell of pair t
    const int hx = (g.n[0] - 1) / 2, ny = g.n[1] - 2, r = t / hx, z = r / ny;
    return 1 + 2 * (t - r * hx) + (1 + r - z * ny) * int(g.s[1]) + (D == 3 ? (1 + z) * int(g.s[2]) : 0);
}
template <int D>
__host__ __device__ inline void cl_window(const Grid& g, int C, int rank, int& lo, int& hi) {
    const int n = cl_pairs<D>(g), share = (n + C - 1) / C, far = int(g.s[D - 1]);
    const int t0 = rank * share, t1 = min((rank + 1) * share, n);
    lo = 0;
    hi = -1;   // a block without pairs
    if (t0 >= t1) return;
    const int s1 = int(g.s[1]);
    lo = (cl_cell<D>(g, t0) - far) / s1 * s1;
    hi = (cl_cell<D>(g, t1 - 1) + 1 + far) / s1 * s1 + s1 - 1;
}

struct SolveOut {
    double res;
    int total, vcycles, outer, pad;
};

template <class T>
struct SolveArgs {
    TailArgs<T> tail;
    int nd;                                           // levels above the tail (0: the tail is the hierarchy)
    int flat;                                         // one level, solved by the coarsest level's sweeps
    int win[CL_LEVELS];                               // windows: offsets in values behind the words; win[0] < 0: none
    int win_values;
    int kp[CL_LEVELS + 1], wo[CL_LEVELS + 2];         // pairs a thread keeps of each level, and where their words lie
    Grid g[CL_LEVELS + 1];
    T* x[CL_LEVELS + 1];
    T* b[CL_LEVELS + 1];                              // b[nd]: the tail's right-hand side
    const T* L[CL_LEVELS + 1];
    const T* iD[CL_LEVELS + 1];
    T* r[CL_LEVELS];                                  // residual scratch
    int nu1[CL_LEVELS], nu2[CL_LEVELS];
    T omega;
    T *p, *q, *e;                                     // directions; e: FP32 correction (mixed)
    const T* L0;                                      // the finest operator of the CG
    double* xs;                                       // solution, right-hand side, FP64 operator
    const double* z;
    const double* L64;
    const double* diag64;
    double tol, inner_rtol;
    int itmx, inner_max;
    double* partial;                                  // 4 * CL_MAX
    SolveOut* out;
};

template <class T, int D>
__global__ void __launch_bounds__(TAIL_THREADS) solve_cluster_k(const __grid_constant__ SolveArgs<T> a) {
    namespace cg = cooperative_groups;
    constexpr bool MIXED = sizeof(T) == 4;
    extern __shared__ __align__(16) unsigned char tail_raw[];
    T* sm = reinterpret_cast<T*>(tail_raw);
    unsigned* words = reinterpret_cast<unsigned*>(sm + a.tail.values) + a.tail.words;   // kp * CL_WORDS a thread and level
    T* windows = reinterpret_cast<T*>(words + a.wo[a.nd + 1]);
    __shared__ int wlo[CL_LEVELS][CL_MAX], whi[CL_LEVELS][CL_MAX];
    __shared__ int greach[CL_LEVELS][3][2];   // blocks whose windows hold this block's copies across a wrap, by direction
    __shared__ T mean_s, red[2][TAIL_THREADS];
    __shared__ unsigned long long red_max;
    __shared__ double sc[4];
    cg::cluster_group cl = cg::this_cluster();
    const int tid = threadIdx.x, rank = int(cl.block_rank()), C = int(cl.num_blocks());
    const int t0 = rank * TAIL_THREADS + tid, stride = C * TAIL_THREADS;
    const Grid& g0 = a.g[0];
    const int s1 = int(g0.s[1]), s2 = int(g0.s[2]);

    // cluster barrier: the block's writes are released by one thread's fence (a releasing arrive by each of 1024
    // threads makes every warp wait for its own stores)
    auto sync = [&]() {
        __syncthreads();
        if (tid == 0) asm volatile("fence.acq_rel.cluster;" ::: "memory");
        asm volatile("barrier.cluster.arrive.relaxed;" ::: "memory");
        asm volatile("barrier.cluster.wait.acquire;" ::: "memory");
    };
    // the same for windows alone, which other blocks write directly: nothing has to reach L2
    auto wsync = [&]() {
        asm volatile("barrier.cluster.arrive.release;" ::: "memory");
        asm volatile("barrier.cluster.wait.acquire;" ::: "memory");
    };
    const bool windowed = D == 2 && a.win[0] >= 0;
    auto cells = [&](const Grid& g, auto&& f) {
        const int nx = g.n[0] - 2, ny = g.n[1] - 2, nz = D == 3 ? g.n[2] - 2 : 1, n = nx * ny * nz;
        for (int t = t0; t < n; t += stride) {
            const int r = t / nx, x = 1 + t - r * nx, rz = r / ny, y = 1 + r - rz * ny, z = D == 3 ? 1 + rz : 0;
            f(x, y, z, x + y * int(g.s[1]) + z * int(g.s[2]));
        }
    };
    // block sums of v0 (and v1) into partial[slot (+ 1)]: the threads' sums stay as they are and are added as
    // FP32 pairs or FP64 by one warp each
    auto block_partial = [&](T v0, T v1, int slot, int n) {
        red[0][tid] = v0;
        red[1][tid] = v1;
        __syncthreads();
        const int w = tid >> 5, lane = tid & 31;
        if (w < n) {
            double s;
            if constexpr (MIXED) {
                float hi = 0.f, lo = 0.f;
#pragma unroll 8
                for (int k = 0; k < TAIL_THREADS / 32; ++k) {
                    const ff t = two_sum(hi, red[w][lane + 32 * k]);
                    hi = t.hi;
                    lo += t.lo;
                }
                s = double(hi) + double(lo);
            } else {
                s = 0.0;
#pragma unroll 8
                for (int k = 0; k < TAIL_THREADS / 32; ++k) s += red[w][lane + 32 * k];
            }
            s = warp_sum(s);
            if (lane == 0) a.partial[(slot + w) * CL_MAX + rank] = s;
        }
        __syncthreads();
    };
    // (after a cluster barrier) the cluster's sum of a slot, in lane 0 of the calling warp
    auto cluster_total = [&](int slot) {
        const int lane = tid & 31;
        return warp_sum(lane < C ? __ldcg(a.partial + slot * CL_MAX + lane) : 0.0);
    };
    // A thread's pairs of level l: pre-smoothing (from x = 0) and the residual (PRE), prolongation and post-smoothing
    // (POST), or the coarsest level's sweeps from x = 0 on the right-hand side less its mean (FLAT).
    // What a thread needs of its cells is in shared memory (tail_words); every operand of a cell lies at its byte
    // offset from a pointer that is the same for all threads, as copies of the cells across a periodic wrap are kept in
    // x's ghosts (tail_store).
    auto smooth = [&](int l, int mode) {
        const bool post = mode == POST;
        const Grid& g = a.g[l];
        T* const xg = keep(a.x[l]);
        T* const win = windows + a.win[l];                                  // (windowed)
        T* const xv = windowed ? win - wlo[l][rank] : xg;
        T* b = keep(a.b[l]);
        const T* __restrict__ L = keep(a.L[l]);
        const T* __restrict__ iD = keep(a.iD[l]);
        const T om = mode == FLAT ? T(1) : a.omega;
        const int N = keep(int(g.N)), r1 = keep(int(g.s[1])), r2 = keep(int(g.s[2])), conflicts = keep(wrap_conflicts(g));
        const Wraps wr(g);
        const unsigned* w = words + a.wo[l] + tid;
        const int kp = a.kp[l];
        PairCells pc[CL_PAIRS];
        unsigned in[CL_PAIRS];
        T bv[2 * CL_PAIRS];   // right-hand side of the red and the black cell
#pragma unroll
        for (int k = 0; k < CL_PAIRS; ++k) {
            const unsigned w0 = k < kp ? w[(k * CL_WORDS) * TAIL_THREADS] : 0u;
            if (w0) pc[k] = PairCells(w0, w[(k * CL_WORDS + 1) * TAIL_THREADS]);
            in[k] = w0 ? pc[k].order(w[(k * CL_WORDS + TAIL_WORDS) * TAIL_THREADS]) : 0u;
            bv[2 * k] = pc[k].red ? b[pc[k].red] : T(0);
            bv[2 * k + 1] = pc[k].black ? b[pc[k].black] : T(0);
            if (mode == FLAT) {
                // mean-free.  In FP64 the right-hand side in memory is the CG's residual, which the stopping test reads:
                // it keeps its mean.  The mixed mode's inner residual loses it there, too (the outer one is formed anew).
                const T mean = T(sc[2]);
                if (pc[k].red) bv[2 * k] -= mean;
                if (pc[k].black) bv[2 * k + 1] -= mean;
                if (MIXED && pc[k].red) b[pc[k].red] = bv[2 * k];
                if (MIXED && pc[k].black) b[pc[k].black] = bv[2 * k + 1];
            }
        }
        // v into cell I (flags f) and its ghost copies: in this block's window and those in mask m that hold it too
        auto store = [&](unsigned I, unsigned f, unsigned m, T v) {
            if (!windowed) {
                tail_store<T, D>(wr, xv, I, f, v);
                return;
            }
            const int gx = f & 1u ? wr.w0 : f & 2u ? -wr.w0 : 0;   // both at a single cell: the other copy below
            xv[I] = v;
            if (gx) xv[int(I) + gx] = v;
            for (; m; m &= m - 1) {
                const int r = __ffs(m) - 1;
                T* p = cl.map_shared_rank(win, r) + (int(I) - wlo[l][r]);
                *p = v;
                if (gx) p[gx] = v;
            }
            if (!(f & 12u) && (f & 3u) != 3u) return;
            auto ghost = [&](int J, int q) {
                for (int r = greach[l][q][0]; r <= greach[l][q][1]; ++r)
                    if (J >= wlo[l][r] && J <= whi[l][r]) cl.map_shared_rank(win, r)[J - wlo[l][r]] = v;
            };
            if ((f & 3u) == 3u) ghost(int(I) - wr.w0, 0);
            if (f & 4u) ghost(int(I) + wr.w1, 1);
            if (f & 8u) ghost(int(I) - wr.w1, 2);
        };
        auto stage = [&]() {
            if (windowed) wsync();
            else sync();
        };
        const T* xc = post ? keep(a.x[l + 1]) : nullptr;
        // From zero, the first red half-sweep reads no neighbour, and no black cell is read before its own half-sweep
        // unless cells of a colour touch across a wrap.
        const bool direct = !post && !conflicts;
#pragma unroll
        for (int k = 0; k < CL_PAIRS; ++k) {
            const int r = pc[k].red, c = pc[k].black;
            T vr = T(0), vc = T(0);
            if (post) {
                const unsigned par = r || c ? pc[k].order(w[(k * CL_WORDS + 2) * TAIL_THREADS]) : 0u;
                if (r) vr = xv[r] + xc[par & 0xFFFFu];
                if (c) vc = xv[c] + xc[par >> 16];
            } else if (direct && r) {
                vr = om * (bv[2 * k] * __ldg(iD + r));
            }
            if (r) store(r, pc[k].fl & 0xFFFFu, in[k] & 0xFFFFu, vr);
            if (c && (!direct || !windowed)) store(c, pc[k].fl >> 16, in[k] >> 16, vc);
            else if (c) xv[c] = T(0);
        }
        stage();
        auto ld = [](const T* p, unsigned o) { return *reinterpret_cast<const T*>(reinterpret_cast<const char*>(p) + o); };
        auto nc = [](const T* p, unsigned o) { return __ldg(reinterpret_cast<const T*>(reinterpret_cast<const char*>(p) + o)); };
        // b - Σ c x_nb of the cell at byte offset o, and Σ c when asked for
        auto gather = [&](unsigned o, T r, T* dd) {
            const T c0 = nc(L, o), c1 = nc(L + 1, o), c2 = nc(L + N, o), c3 = nc(L + N + r1, o);
            const T x0 = ld(xv - 1, o), x1 = ld(xv + 1, o), x2 = ld(xv - r1, o), x3 = ld(xv + r1, o);
            T c4 = T(0), c5 = T(0), x4 = T(0), x5 = T(0);
            if (D == 3) {
                c4 = nc(L + 2 * N, o);
                c5 = nc(L + 2 * N + r2, o);
                x4 = ld(xv - r2, o);
                x5 = ld(xv + r2, o);
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
        const int nh = mode == FLAT ? keep(a.tail.nuc) + 1 : post ? 2 * keep(a.nu2[l]) : 2 * keep(a.nu1[l]);
        for (int s = direct ? 1 : 0; s < nh; ++s) {
            const int color = (s + (post ? 1 : 0)) & 1, sh = 16 * color;
            for (int cls = 0; cls <= conflicts; ++cls) {
                if (cls & ~conflicts) continue;
                // the operands of every pair are read before the first store
                T nv[CL_PAIRS];
#pragma unroll
                for (int k = 0; k < CL_PAIRS; ++k) {
                    const unsigned I = color ? pc[k].black : pc[k].red, o = I * unsigned(sizeof(T));
                    if (!I) continue;
                    const T xo = ld(xv, o), d = nc(iD, o), r = gather(o, color ? bv[2 * k + 1] : bv[2 * k], nullptr);
                    nv[k] = om == T(1) ? r * d : fma(om, fma(r, d, -xo), xo);
                }
#pragma unroll
                for (int k = 0; k < CL_PAIRS; ++k) {
                    const int I = color ? pc[k].black : pc[k].red;
                    const unsigned f = pc[k].fl >> sh & 0xFFFFu;
                    if (I && int(f >> 6 & 7u) == cls) store(I, f, in[k] >> sh & 0xFFFFu, nv[k]);
                }
                stage();
            }
        }
        if (mode != PRE) {
            if (windowed) {   // the finer level's prolongation and the CG read x in memory
#pragma unroll
                for (int k = 0; k < CL_PAIRS; ++k) {
                    if (pc[k].red) xg[pc[k].red] = xv[pc[k].red];
                    if (pc[k].black) xg[pc[k].black] = xv[pc[k].black];
                }
                sync();
            }
            return;
        }
        T* res = keep(a.r[l]);
#pragma unroll
        for (int k = 0; k < CL_PAIRS; ++k)
#pragma unroll
            for (int c = 0; c < 2; ++c) {
                const unsigned I = c ? pc[k].black : pc[k].red, o = I * unsigned(sizeof(T));
                if (!I) continue;
                T dd;
                const T r = gather(o, bv[2 * k + c], &dd);
                res[I] = fma(dd, ld(xv, o), r);
            }
        sync();
        // the next level's right-hand side: its words are those of this slot's threads, the tail's of the first ones
        T* bc = keep(a.b[l + 1]);
        const unsigned* wc = words + a.wo[l + 1] + tid;
        const int kc = a.kp[l + 1];
#pragma unroll
        for (int k = 0; k < CL_PAIRS; ++k) {
            if (k >= kc) continue;
            const unsigned w0 = wc[(k * CL_WORDS) * TAIL_THREADS], f = wc[(k * CL_WORDS + 1) * TAIL_THREADS], I = w0 & 0x3FFFFFFFu;
            if (!w0) continue;
            const T* r = res + wc[(k * CL_WORDS + 3) * TAIL_THREADS];
            bc[I] = tail_children<T, D>(r, f & 0xFFFFu, r1, r2);
            if (w0 >> 31) bc[I + 1] = tail_children<T, D>(r + (f & 512u ? 2 : 1), f >> 16, r1, r2);
        }
        sync();
    };
    auto vcycle = [&]() {
        if (a.flat) {
            T acc = T(0);
            cells(g0, [&](int, int, int, int I) { acc += a.b[0][I]; });
            block_partial(acc, T(0), 0, 1);
            sync();
            if (tid < 32) {
                const double sum = cluster_total(0);
                if (tid == 0) sc[2] = sum / double((g0.n[0] - 2) * (g0.n[1] - 2) * (D == 3 ? g0.n[2] - 2 : 1));
            }
            __syncthreads();
            smooth(0, FLAT);
            return;
        }
        for (int l = 0; l < a.nd; ++l) smooth(l, PRE);
        if (rank == 0) tail_cycle<T, D>(a.tail, sm, mean_s);
        sync();
        for (int l = a.nd - 1; l >= 0; --l) smooth(l, POST);
    };
    // cluster maximum of the threads' |values| (bit patterns) into sc[3], with a cluster barrier
    auto cluster_max = [&](unsigned long long m) {
        if (tid == 0) red_max = 0ull;
        __syncthreads();
        m = warp_max(m);
        if ((tid & 31) == 0) atomicMax(&red_max, m);
        __syncthreads();
        if (tid == 0) reinterpret_cast<unsigned long long*>(a.partial)[3 * CL_MAX + rank] = red_max;
        sync();
        if (tid < 32) {
            unsigned long long v = tid < C ? __ldcg(reinterpret_cast<unsigned long long*>(a.partial) + 3 * CL_MAX + tid) : 0ull;
            v = warp_max(v);
            if (tid == 0) sc[3] = __longlong_as_double((long long)v);
        }
        __syncthreads();
        const double r = sc[3];
        __syncthreads();
        return (unsigned long long)__double_as_longlong(r);
    };
    // r = z - A x in FP64 (mixed: the next inner solve's right-hand side, with e = 0); its largest |value|
    auto true_residual = [&]() {
        unsigned long long m = 0ull;
        cells(g0, [&](int x, int y, int z, int I) {
            const double v = resid7<D>(g0, a.L64, fma(-__ldg(a.diag64 + I), a.xs[I], __ldg(a.z + I)), a.xs, I, nb_of<D>(g0, x, y, z));
            if constexpr (MIXED) {
                a.b[0][I] = f32_rn(v);
                a.e[I] = 0.f;
            } else {
                a.b[0][I] = v;
            }
            const unsigned long long k = abs_bits(v);
            m = k > m ? k : m;
        });
        return __longlong_as_double((long long)cluster_max(m));
    };

    // windows: their bounds, and zeros (the ghosts of walls stay so)
    const int tops = windowed ? a.nd + a.flat : 0;
    if (tid < tops * CL_MAX) {
        const int l = tid / CL_MAX, r = tid - l * CL_MAX;
        int lo = 0, hi = -1;
        if (r < C) cl_window<D>(a.g[l], C, r, lo, hi);
        wlo[l][r] = lo;
        whi[l][r] = hi;
    }
    if (tid < CL_LEVELS * 3) {
        greach[tid / 3][tid % 3][0] = CL_MAX;
        greach[tid / 3][tid % 3][1] = -1;
    }
    if (windowed)
        for (int i = tid; i < a.win_values; i += TAIL_THREADS) windows[i] = T(0);
    __syncthreads();
    // the words of this thread's pairs of every level (the last: the tail's largest, for its right-hand side)
    for (int l = 0; l <= a.nd; ++l) {
        const Grid& g = a.g[l];
        const int n = cl_pairs<D>(g), share = (n + C - 1) / C;
        for (int k = 0; k < a.kp[l]; ++k) {
            unsigned* w = words + a.wo[l] + k * CL_WORDS * TAIL_THREADS + tid;
            const int t = rank * share + k * TAIL_THREADS + tid;
            for (int q = 0; q < CL_WORDS; ++q) w[q * TAIL_THREADS] = 0u;
            if (k * TAIL_THREADS + tid >= share || t >= n) continue;
            tail_words<D>(g, l < a.nd ? &a.g[l + 1] : nullptr, l > 0 ? &a.g[l - 1] : nullptr, t, w, TAIL_THREADS);
            if (l >= tops) continue;
            const int I = int(w[0] & 0x3FFFFFFFu);
            unsigned m = 0u;
            for (int r = 0; r < C; ++r) {
                if (r == rank) continue;
                if (I >= wlo[l][r] && I <= whi[l][r]) m |= 1u << r;
                if (I + 1 >= wlo[l][r] && I + 1 <= whi[l][r]) m |= 0x10000u << r;
            }
            w[TAIL_WORDS * TAIL_THREADS] = m;
            const Wraps wr(g);
            for (int c = 0; c < 2; ++c) {
                const unsigned f = w[TAIL_THREADS] >> (16 * c) & 63u;
                for (int q = 0; q < 3; ++q) {
                    if (!(q == 0 ? (f & 3u) == 3u : (f >> (q + 1) & 1u) != 0u)) continue;
                    const int J = I + c + (q == 0 ? -wr.w0 : q == 1 ? wr.w1 : -wr.w1);
                    for (int r = 0; r < C; ++r)
                        if (J >= wlo[l][r] && J <= whi[l][r]) {
                            atomicMin(&greach[l][q][0], r);
                            atomicMax(&greach[l][q][1], r);
                        }
                }
            }
        }
    }
    sync();
    if (rank == 0 && !a.flat) tail_setup<T, D>(a.tail, sm);
    T* rv = a.b[0];
    T* sv = a.x[0];
    const int N0 = int(g0.N);
    int total = 0, outer = 0, vcycles = 0;
    double alpha_prev = 0.0, rho_prev = 0.0;   // of thread 0
    double res = true_residual();
    bool more = true;
    while (more && !(res <= a.tol) && total < a.itmx) {
        // FP64: one flexible CG, stopping on its recurrence's residual; mixed: inner solves of A e = r
        const double target = MIXED ? fmax(0.5 * a.tol / res, a.inner_rtol) * res : a.tol;
        const int most = MIXED ? a.inner_max : a.itmx;
        for (int it = 0; it < most && total < a.itmx; ++it) {
            vcycle();
            ++vcycles;
            T a1 = T(0), a2 = T(0);
            for (int i = t0; i < N0; i += stride) {
                const T s = sv[i];
                a1 = fma(s, a.q[i], a1);
                a2 = fma(s, rv[i], a2);
            }
            block_partial(a1, a2, 0, 2);
            sync();
            if (tid < 32) {
                const double sq = cluster_total(0), sr = cluster_total(1);
                if (tid == 0) {
                    sc[0] = it == 0 ? 0.0 : (-alpha_prev * sq) / rho_prev;
                    sc[1] = sr;
                }
            }
            __syncthreads();
            const double beta = sc[0], sr = sc[1];
            const T bt = T(beta);
            for (int i = t0; i < N0; i += stride) a.p[i] = bt == T(0) ? sv[i] : fma(bt, a.p[i], sv[i]);
            sync();
            T acc = T(0);
            cells(g0, [&](int x, int y, int z, int I) {
                const T d = MIXED ? diag7<D>(g0, a.L0, I) : T(__ldg(a.diag64 + I));
                const T v = -resid7<D>(g0, a.L0, -d * a.p[I], a.p, I, nb_of<D>(g0, x, y, z));
                a.q[I] = v;
                acc = fma(a.p[I], v, acc);
            });
            block_partial(acc, T(0), 2, 1);
            sync();
            if (tid < 32) {
                const double pq = cluster_total(2);
                if (tid == 0) {
                    const double alpha = sr / pq;
                    const bool stop = !(pq != 0.0) || !isfinite(pq) || !isfinite(sr) || !isfinite(beta);
                    sc[0] = stop ? 1.0 : 0.0;
                    sc[1] = alpha;
                    if (!stop) {
                        rho_prev = sr;
                        alpha_prev = alpha;
                    }
                }
            }
            __syncthreads();
            const bool stop = sc[0] != 0.0;
            const T al = T(sc[1]);
            if (stop) {   // a breakdown: no update
                if (MIXED) ++total;
                else more = false;
                __syncthreads();
                break;
            }
            unsigned long long m = 0ull;
            for (int i = t0; i < N0; i += stride) {
                if constexpr (MIXED) a.e[i] = fma(al, a.p[i], a.e[i]);
                else a.xs[i] = fma(al, a.p[i], a.xs[i]);
                const T v = fma(-al, a.q[i], rv[i]);
                rv[i] = v;
                unsigned long long k;
                if constexpr (MIXED) k = __float_as_uint(v) & 0x7FFFFFFFu;
                else k = abs_bits(v);
                m = k > m ? k : m;
            }
            m = cluster_max(m);
            ++total;
            double rinf;
            if constexpr (MIXED) rinf = double(__uint_as_float(unsigned(m)));
            else res = rinf = __longlong_as_double((long long)m);
            if (rinf <= target) break;
        }
        if constexpr (MIXED) {
            cells(g0, [&](int, int, int, int I) { a.xs[I] += widen_exact(a.e[I]); });
            sync();
            res = true_residual();
            ++outer;
        }
    }
    sync();
    for (long long t = t0; t < bc_plane_cells(g0); t += stride) perbc_cell(g0, a.xs, t);
    if (rank == 0 && tid == 0) {
        a.out->res = res;
        a.out->total = total;
        a.out->vcycles = vcycles;
        a.out->outer = outer;
    }
}

}  // namespace
}  // namespace ia
