// Learned Poisson preconditioner (see nn.cuh for the network).
//
//  * Training kernels (FP32, CUDA cores; the convolutions and their gradients in
//    nn_train.cuh): MSE and energy losses, Adam.
//  * Inference kernel (BF16 weights and activations, FP32 accumulation on the
//    5th-generation tensor cores): implicit GEMM with M = 128 output cells, a
//    patch marched through z, fed by TMA; tcgen05.mma (kind::f16, BF16 x BF16 ->
//    FP32 in TMEM) from one elected thread, tcgen05.ld for the bias / ReLU /
//    skip epilogue.  Every mbarrier wait is bounded; on timeout the kernel
//    raises an error flag, waits for its copies, releases its TMEM and returns.
#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstring>
#include <type_traits>
#include <vector>

#include "capi_internal.cuh"
#include "nn.cuh"

namespace ia {
namespace nn {

// ------------------------------------------------------------------ activation tensors
// storage [B][nz+2][ny+2][nx+2][C], interior cells (x, y, z) in 0..n-1
struct Dims {
    int B, nx, ny, nz;
    __host__ __device__ long long cells() const { return (long long)B * nx * ny * nz; }
    __host__ __device__ long long padded() const { return (long long)B * (nx + 2) * (ny + 2) * (nz + 2); }
    __host__ __device__ long long pos(int b, int x, int y, int z) const {
        return (((long long)b * (nz + 2) + z + 1) * (ny + 2) + y + 1) * (nx + 2) + x + 1;
    }
    __host__ __device__ void decode(long long q, int& b, int& x, int& y, int& z) const {
        x = int(q % nx);
        q /= nx;
        y = int(q % ny);
        q /= ny;
        z = int(q % nz);
        b = int(q / nz);
    }
    __host__ __device__ long long tap(int t) const {   // offset of tap t = (dz+1)*9 + (dy+1)*3 + (dx+1)
        const int dx = t % 3 - 1, dy = (t / 3) % 3 - 1, dz = t / 9 - 1;
        return ((long long)dz * (ny + 2) + dy) * (nx + 2) + dx;
    }
    __host__ __device__ Dims half() const { return Dims{B, nx / 2, ny / 2, nz / 2}; }
};

__device__ __forceinline__ long long child_pos(const Dims& f, int b, int X, int Y, int Z, int k) {
    return f.pos(b, 2 * X + (k & 1), 2 * Y + ((k >> 1) & 1), 2 * Z + (k >> 2));
}

#define FOR_CELLS(D)                                                                                      \
    for (long long q = blockIdx.x * (long long)blockDim.x + threadIdx.x; q < (D).cells();                \
         q += (long long)gridDim.x * blockDim.x)

}  // namespace nn
}  // namespace ia
#include "nn_train.cuh"

namespace ia {
namespace nn {

// ------------------------------------------------------------------ FP32 training kernels: loss and optimiser
// dOut = 2 (out - tgt) / n ; loss partials
__global__ void mse_k(Dims d, const float* __restrict__ out, const float* __restrict__ tgt, float* __restrict__ dout,
                      double* __restrict__ loss) {
    __shared__ double sm[256];
    const double inv = 1.0 / double(d.cells());
    double s = 0.0;
    FOR_CELLS(d) {
        int b, x, y, z;
        d.decode(q, b, x, y, z);
        const long long p = d.pos(b, x, y, z);
        const float e = out[p] - tgt[p];
        dout[p] = float(2.0 * inv) * e;
        s += double(e) * double(e);
    }
    sm[threadIdx.x] = s;
    __syncthreads();
    for (int w = 128; w > 0; w >>= 1) {
        if (threadIdx.x < w) sm[threadIdx.x] += sm[threadIdx.x + w];
        __syncthreads();
    }
    if (threadIdx.x == 0) atomicAdd(loss, sm[0] * inv);
}

// Energy norm of the error with the patch's own coefficients: δ = out - tgt,
// E = Σ_p Σ_d c[p,d] (δ[p] - δ[p-e_d])² / n with c = input channel 1+d (λρ·L on the cell's lower
// d-face; zero on walls and in the halo, where δ is zero too); dout = dE/dout.
__global__ void energy_k(Dims d, const float* __restrict__ out, const float* __restrict__ tgt,
                         const float* __restrict__ x0, float* __restrict__ dout, double* __restrict__ loss) {
    __shared__ double sm[256];
    const double inv = 1.0 / double(d.cells());
    const long long off[3] = {1, (long long)(d.nx + 2), (long long)(d.nx + 2) * (d.ny + 2)};
    double acc = 0.0;
    FOR_CELLS(d) {
        int b, x, y, z;
        d.decode(q, b, x, y, z);
        const long long p = d.pos(b, x, y, z);
        const float dp = out[p] - tgt[p];
        float g = 0.f;
        for (int k = 0; k < 3; ++k) {
            const long long lo = p - off[k], hi = p + off[k];
            const float dl = dp - (out[lo] - tgt[lo]);          // across the lower face
            const float dh = (out[hi] - tgt[hi]) - dp;          // across the upper face
            const float cl = x0[p * 4 + 1 + k], ch = x0[hi * 4 + 1 + k];
            acc += double(cl) * double(dl) * double(dl);
            g += cl * dl - ch * dh;
        }
        dout[p] = float(2.0 * inv) * g;
    }
    sm[threadIdx.x] = acc;
    __syncthreads();
    for (int w = 128; w > 0; w >>= 1) {
        if (threadIdx.x < w) sm[threadIdx.x] += sm[threadIdx.x + w];
        __syncthreads();
    }
    if (threadIdx.x == 0) atomicAdd(loss, sm[0] * inv);
}

__global__ void adam_k(long long n, float* __restrict__ w, const float* __restrict__ g, float* __restrict__ m,
                       float* __restrict__ v, float lr, float b1, float b2, float eps, float c1, float c2) {
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
        const float gi = g[i];
        const float mi = b1 * m[i] + (1.f - b1) * gi;
        const float vi = b2 * v[i] + (1.f - b2) * gi * gi;
        m[i] = mi;
        v[i] = vi;
        w[i] -= lr * (mi / c1) / (sqrtf(vi / c2) + eps);
    }
}

// ------------------------------------------------------------------ tcgen05 inference convolution
__device__ __forceinline__ uint32_t smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

// shared-memory matrix descriptor, K-major, no swizzle: core matrices of 8 rows x 16 bytes,
// LBO = byte distance of K-adjacent core matrices, SBO = of M/N-adjacent ones
__device__ __forceinline__ uint64_t smem_desc(uint32_t saddr, uint32_t lbo, uint32_t sbo) {
    uint64_t d = (uint64_t)((saddr >> 4) & 0x3FFFu);
    d |= (uint64_t)((lbo >> 4) & 0x3FFFu) << 16;
    d |= (uint64_t)((sbo >> 4) & 0x3FFFu) << 32;
    d |= (uint64_t)1 << 46;   // descriptor version of the 5th-generation tensor cores
    return d;                 // base offset 0, layout SWIZZLE_NONE
}
// instruction descriptor, kind::f16: D F32, A/B BF16, both K-major
__host__ __device__ constexpr uint32_t idesc_bf16(int M, int N) {
    return (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(N >> 3) << 17) | ((uint32_t)(M >> 4) << 24);
}

__device__ __forceinline__ uint64_t global_ns() {
    uint64_t t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}

// Poll an mbarrier phase for at most ~1 s of wall time (and a fixed number of polls), or until *fail (another
// wait of the block has given up).
__device__ __forceinline__ bool mbar_wait(uint32_t mbar, uint32_t parity, const volatile int* fail) {
    uint64_t t0 = 0;
    for (uint32_t i = 0; i < (1u << 28); ++i) {
        uint32_t ok = 0;
        asm volatile(
            "{\n\t.reg .pred P;\n\tmbarrier.try_wait.parity.shared::cta.b64 P, [%1], %2;\n\tselp.b32 %0, 1, 0, P;\n\t}\n"
            : "=r"(ok)
            : "r"(mbar), "r"(parity)
            : "memory");
        if (ok) return true;
        if ((i & 255u) == 255u) {
            if (fail && *fail) return false;
            const uint64_t t = global_ns();
            if (t0 == 0) t0 = t;
            if (t - t0 > 1000000000ull) return false;
        }
    }
    return false;
}

__device__ __forceinline__ void tmem_ld16(uint32_t taddr, float (&v)[16]) {
    uint32_t r[16];
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
          "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
        : "r"(taddr));
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
    for (int i = 0; i < 16; ++i) v[i] = __uint_as_float(r[i]);
}

// ------------------------------------------------------------------ TMA-fed tensor-core convolution
// Inference activations are stored as 8-channel planes: plane j holds channels 8j..8j+7 of every
// (padded, halo-included) cell, 16 B per cell.
// A block marches a patch of 8 x 16 cells (x, y: the MMA's M = 128 rows) through up to ZP planes of z.  One TMA box
// brings one z plane of the patch with its halo, all channels: 10 x 18 cells of 16 B for each 8 channels, the
// 160 B of a row as one run.  In
// shared memory that is a K-major no-swizzle operand: 8 cells of a row are a core matrix of 128 B, the next row is
// 160 B on (SBO), the next 8 channels one box on (LBO), and the A operand of tap (dx, dy) starts (dy+1)·10 + dx+1
// cells in.  A plane is loaded once and multiplied once for its three output planes: the B operand of a tap has
// the weights of dz = +1, 0, -1 side by side (N = 3·Cout) and the accumulators of the output planes z-1, z, z+1
// are neighbouring column blocks of TMEM.  An output's 27·Cin products are added in the order of the taps
// (dz, then dy, dx, then channels), as one tap after the other into one accumulator would.
// Warp 4 issues the loads, warp 5 the MMAs, warps 0-3 read finished planes with tcgen05.ld and clear their columns
// for the next patch; a ring of NS stages and per-plane barriers let the three run independently, also from one
// patch to the next.  The MMAs of a plane have one accumulator and one shape; the next plane's, one column block on,
// are issued when they have finished (the order of MMAs on overlapping accumulators of another base or shape is not
// specified), while the other block of the multiprocessor keeps the tensor cores busy.
// What bounds it: an MMA takes about 50 ns whatever its N (16 more of them a plane cost 110 us more over 242 planes
// a multiprocessor: the A operand's rows, not the products), so the 9·Cin/16 MMAs a plane, a third of a tap-by-tap
// N = Cout form's.  A plane is fetched from L2 1.4 times (halo) instead of 9 times.  Measured, 32 -> 16 channels on
// 128 x 256 x 128 cells: 1334 us with the tap-by-tap kernel (one 128-cell row a tile, 9 windows each), 213 us here;
// 16 -> 16 channels 389 and 103 us.
constexpr int kM = 128;                  // output cells per patch plane (the MMA M)
constexpr int kPX = 8, kPY = 16;         // patch
constexpr int kBX = kPX + 2, kBY = kPY + 2;
constexpr int BOX_BYTES = kBX * kBY * 16;   // one plane of a patch, 8 channels
constexpr int kTmemCols = 256;           // two blocks share a multiprocessor's 512
constexpr int kConvThreads = 192;

template <int CI, int COP>
struct TmaSmem {
    static constexpr int W_BYTES = 27 * COP * CI * 2;
    static constexpr int STAGE_BYTES = CI / 8 * BOX_BYTES;
    static constexpr int NS = COP > 16 ? 4 : 6;
    static constexpr int ZP = kTmemCols / COP;                       // output planes in flight
    static constexpr int A_OFF = (W_BYTES + 1023) / 1024 * 1024;
    static constexpr int BAR_OFF = A_OFF + NS * STAGE_BYTES;
    static constexpr int USED = BAR_OFF + 8 * (2 * NS + 2 * ZP + 1);
    // at least 80 KB, so that no third block waits for TMEM on a multiprocessor
    static constexpr int TOTAL = USED > 80 * 1024 ? USED : 80 * 1024;
    static_assert(STAGE_BYTES % 128 == 0, "TMA destination");
};

// box at (x, y, z) of the padded grid: the innermost dimension runs over the 8 channels of the cells of a row
__device__ __forceinline__ void tma_load_box(uint32_t dst, const CUtensorMap* map, int x, int y, int z, uint32_t bar) {
    asm volatile(
        "cp.async.bulk.tensor.4d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4, %5}], [%6];"
        ::"r"(dst), "l"(reinterpret_cast<uint64_t>(map)), "r"(8 * x), "r"(y), "r"(z), "r"(0), "r"(bar)
        : "memory");
}
__device__ __forceinline__ void mbar_arrive(uint32_t bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ void mma_commit(uint32_t bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ void mma_bf16(uint32_t d, uint64_t ad, uint64_t bd, uint32_t idesc) {   // D += A B
    asm volatile(
        "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}\n" ::"r"(d),
        "l"(ad), "l"(bd), "r"(idesc), "r"(1u));
}
__device__ __forceinline__ void tmem_zero16(uint32_t taddr) {
    asm volatile("tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1,%1,%1,%1,%1,%1,%1,%1,%1,%1,%1,%1,%1,%1,%1,%1};" ::"r"(taddr),
                 "r"(0u)
                 : "memory");
}

template <int CI, int CO, bool RELU, bool OUTF32>
__global__ void __launch_bounds__(kConvThreads) conv_tma_kernel(const __grid_constant__ CUtensorMap tmap, Dims d,
                                                                int zc, const uint8_t* __restrict__ Wg,
                                                                const float* __restrict__ bias,
                                                                const __nv_bfloat16* __restrict__ skip,
                                                                __nv_bfloat16* __restrict__ Y, float* __restrict__ Yf,
                                                                int* __restrict__ err) {
    constexpr int COP = CO < 16 ? 16 : CO;
    using S = TmaSmem<CI, COP>;
    constexpr int NS = S::NS;
    static_assert(CI % 16 == 0 && COP % 16 == 0 && COP <= 32, "tile shape");
    extern __shared__ __align__(1024) uint8_t smem[];
    __shared__ uint32_t tmem_holder;
    __shared__ int fail;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    // weights: chunk (tap of the plane q, block k) holds dz = 1 - k
    constexpr int CHUNK = COP * CI * 2 / 16;
    for (int i = tid; i < S::W_BYTES / 16; i += blockDim.x) {
        const int q = i / (3 * CHUNK), k = i / CHUNK % 3;
        reinterpret_cast<uint4*>(smem)[i] = __ldg(reinterpret_cast<const uint4*>(Wg) + ((2 - k) * 9 + q) * CHUNK + i % CHUNK);
    }
    const uint32_t full0 = smem_u32(smem + S::BAR_OFF), empty0 = full0 + 8 * NS, out0 = empty0 + 8 * NS,
                   free0 = out0 + 8 * S::ZP, drain = free0 + 8 * S::ZP;
    if (tid == 0) {
        fail = 0;
        for (int k = 0; k < 2 * NS + S::ZP; ++k) asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(full0 + 8 * k));
        for (int k = 0; k < S::ZP; ++k) asm volatile("mbarrier.init.shared::cta.b64 [%0], 4;" ::"r"(free0 + 8 * k));
        asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(drain));
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_holder)),
                     "r"(kTmemCols));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
    }
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");   // weights: generic writes, async reads
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem = tmem_holder;
    if (warp < 4) {
        for (int c0 = 0; c0 < kTmemCols; c0 += 16) tmem_zero16(tmem + c0 + ((uint32_t)(warp * 32) << 16));
        asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t wbase = smem_u32(smem), abase = smem_u32(smem + S::A_OFF);
    const int npx = (d.nx + kPX - 1) / kPX, npy = (d.ny + kPY - 1) / kPY, npz = (d.nz + zc - 1) / zc;
    const int items = npx * npy * npz * d.B;
    // item -> patch origin and output planes [z0, z1)
    auto item_of = [&](int it, int& x0, int& y0, int& z0, int& z1, int& b) {
        x0 = it % npx * kPX;
        it /= npx;
        y0 = it % npy * kPY;
        it /= npy;
        z0 = it % npz * zc;
        z1 = min(z0 + zc, d.nz);
        b = it / npz;
    };
    // a wait gives up when another role has, or after about a second; the kernel then raises err and ends
    auto wait = [&](uint32_t bar, uint32_t parity) {
        const bool ok = mbar_wait(bar, parity, &fail);
        if (!ok) atomicExch(&fail, 1);
        return ok;
    };
    if (warp == 4 && lane == 0) {   // loads
        int n = 0;   // planes issued
        bool ok = true;
        for (int it = blockIdx.x; it < items && ok; it += gridDim.x) {
            int x0, y0, z0, z1, b;
            item_of(it, x0, y0, z0, z1, b);
            for (int zi = z0 - 1; zi <= z1; ++zi, ++n) {
                const int s = n % NS;
                if (n >= NS && !(ok = wait(empty0 + 8 * s, uint32_t(n / NS - 1) & 1))) break;
                asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(full0 + 8 * s), "r"(S::STAGE_BYTES)
                             : "memory");
                // padded coordinates of the box's first cell: x0 - 1 + 1, ...
                tma_load_box(abase + s * S::STAGE_BYTES, &tmap, x0, y0, b * (d.nz + 2) + zi + 1, full0 + 8 * s);
            }
        }
        // a block must not end with copies in flight
        if (!ok)
            for (int k = n > NS ? n - NS : 0; k < n; ++k) mbar_wait(full0 + 8 * (k % NS), uint32_t(k / NS) & 1, nullptr);
    } else if (warp == 5 && lane == 0) {   // MMAs
        int n = 0;
        uint32_t used = 0, par = 0;   // per TMEM block: used before, parity of its uses
        bool ok = true;
        for (int it = blockIdx.x; it < items && ok; it += gridDim.x) {
            int x0, y0, z0, z1, b;
            item_of(it, x0, y0, z0, z1, b);
            for (int zi = z0 - 1; zi <= z1; ++zi, ++n) {
                const int s = n % NS;
                if (!(ok = wait(full0 + 8 * s, uint32_t(n / NS) & 1))) break;
                if (n > 0 && !(ok = wait(empty0 + 8 * ((n - 1) % NS), uint32_t((n - 1) / NS) & 1))) break;   // the last plane's MMAs
                // weight blocks k0..k1: output planes zi-1+k0 .. zi-1+k1 inside [z0, z1)
                const int k0 = zi - 1 < z0 ? z0 - zi + 1 : 0, k1 = zi + 1 >= z1 ? z1 - zi : 2;
                if (k1 == 2) {   // the first products of plane zi + 1: its block has to be free and cleared
                    const int slot = zi + 1 - z0;
                    if ((used >> slot) & 1)
                        if (!(ok = wait(free0 + 8 * slot, ((par >> slot) & 1) ^ 1))) break;
                    used |= 1u << slot;
                    par ^= 1u << slot;
                }
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                const uint32_t st = abase + s * S::STAGE_BYTES, dcol = tmem + (zi - 1 + k0 - z0) * COP;
                const uint32_t nb = k1 - k0 + 1, idesc = idesc_bf16(kM, 0) | (nb * COP >> 3 << 17);
                // one thread issues: descriptors by constant steps from the plane's first (addresses are below 2^18,
                // so a step never leaves the 14-bit address field), or the issue takes longer than the MMA
                const uint64_t ad = smem_desc(st, BOX_BYTES, kBX * 16);
                const uint64_t bd = smem_desc(wbase + k0 * COP * CI * 2, 128, CI * 16);
#pragma unroll
                for (int q = 0; q < 9; ++q)
#pragma unroll
                    for (int ks = 0; ks < CI / 16; ++ks)
                        mma_bf16(dcol, ad + ((2 * ks * BOX_BYTES + (q / 3 * kBX + q % 3) * 16) >> 4),
                                 bd + ((q * 3 * COP * CI * 2 + ks * 256) >> 4), idesc);
                mma_commit(empty0 + 8 * s);
                if (zi - 1 >= z0) mma_commit(out0 + 8 * (zi - 1 - z0));
            }
        }
        mma_commit(drain);
        mbar_wait(drain, 0, nullptr);
    } else if (warp < 4) {   // finished planes
        uint32_t par = 0;
        float bias_r[CO];
#pragma unroll
        for (int o = 0; o < CO; ++o) bias_r[o] = __ldg(bias + o);
        const long long plane = d.padded() * 8;   // elements per 8-channel plane
        const int px = tid & 7, py = tid >> 3;    // row of the accumulator: cell (px, py) of the patch
        bool ok = true;
        for (int it = blockIdx.x; it < items && ok; it += gridDim.x) {
            int x0, y0, z0, z1, b;
            item_of(it, x0, y0, z0, z1, b);
            const bool valid = x0 + px < d.nx && y0 + py < d.ny;
            for (int z = z0; z < z1; ++z) {
                const int slot = z - z0;
                ok = wait(out0 + 8 * slot, (par >> slot) & 1);
                if (!(ok = __all_sync(0xffffffffu, ok))) break;
                par ^= 1u << slot;
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                const long long p = d.pos(b, x0 + px, y0 + py, z);
                const uint32_t trow = tmem + slot * COP + ((uint32_t)(warp * 32) << 16);
                float v[COP];
#pragma unroll
                for (int c0 = 0; c0 < COP; c0 += 16) tmem_ld16(trow + c0, *reinterpret_cast<float(*)[16]>(v + c0));
#pragma unroll
                for (int c0 = 0; c0 < COP; c0 += 16) tmem_zero16(trow + c0);
                asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
                asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
                __syncwarp();
                if (lane == 0) mbar_arrive(free0 + 8 * slot);
                if (!valid) continue;
                if (OUTF32) {
                    Yf[p] = v[0] + bias_r[0];
                } else {
#pragma unroll
                    for (int c0 = 0; c0 < CO; c0 += 8) {
                        uint32_t packed[4];
                        uint4 sk4 = make_uint4(0u, 0u, 0u, 0u);
                        if (skip) sk4 = __ldg(reinterpret_cast<const uint4*>(skip + (long long)(c0 / 8) * plane + p * 8));
                        const uint32_t* skp = reinterpret_cast<const uint32_t*>(&sk4);
#pragma unroll
                        for (int k = 0; k < 8; k += 2) {
                            float a = v[c0 + k] + bias_r[(c0 + k) % CO], b2 = v[c0 + k + 1] + bias_r[(c0 + k + 1) % CO];
                            if (RELU) {
                                a = fmaxf(a, 0.f);
                                b2 = fmaxf(b2, 0.f);
                            }
                            if (skip) {
                                const __nv_bfloat162 sk = *reinterpret_cast<const __nv_bfloat162*>(&skp[k / 2]);
                                a += __low2float(sk);
                                b2 += __high2float(sk);
                            }
                            const __nv_bfloat162 o2 = __floats2bfloat162_rn(a, b2);
                            packed[k / 2] = *reinterpret_cast<const uint32_t*>(&o2);
                        }
                        *reinterpret_cast<uint4*>(Y + (long long)(c0 / 8) * plane + p * 8) =
                            make_uint4(packed[0], packed[1], packed[2], packed[3]);
                    }
                }
            }
        }
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (tid == 0 && fail) atomicExch(err, 1);
    if (warp == 0) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(kTmemCols));
}

// ------------------------------------------------------------------ BF16 glue kernels (inference)
// 8-channel planes: element (cell p, channel c) at (c/8)·8·padded + 8p + c%8; 16 B per cell and plane
__device__ __forceinline__ void acc8(float (&a)[8], const uint4& v) {
    const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&v);
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        a[2 * i] += __low2float(h[i]);
        a[2 * i + 1] += __high2float(h[i]);
    }
}
__device__ __forceinline__ uint4 pack8(const float (&a)[8]) {
    uint4 v;
    __nv_bfloat162* h = reinterpret_cast<__nv_bfloat162*>(&v);
#pragma unroll
    for (int i = 0; i < 4; ++i) h[i] = __floats2bfloat162_rn(a[2 * i], a[2 * i + 1]);
    return v;
}

// out (coarse dims dc) = mean of the 8 children of in (fine dims 2dc), C/8 planes
__global__ void pool_bf16(Dims dc, int C, const __nv_bfloat16* __restrict__ in, __nv_bfloat16* __restrict__ out) {
    const Dims df{dc.B, 2 * dc.nx, 2 * dc.ny, 2 * dc.nz};
    const long long pin = df.padded() * 8, pout = dc.padded() * 8;
    FOR_CELLS(dc) {
        int b, x, y, z;
        dc.decode(q, b, x, y, z);
        const long long P = dc.pos(b, x, y, z);
        for (int j = 0; j < C / 8; ++j) {
            float a[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
            for (int k = 0; k < 8; ++k)
                acc8(a, *reinterpret_cast<const uint4*>(in + j * pin + child_pos(df, b, x, y, z, k) * 8));
#pragma unroll
            for (int i = 0; i < 8; ++i) a[i] *= 0.125f;
            *reinterpret_cast<uint4*>(out + j * pout + P * 8) = pack8(a);
        }
    }
}
// out[child] = in[parent] (+ skip[child])  (fine dims df), C/8 planes
__global__ void up_bf16(Dims df, int C, const __nv_bfloat16* __restrict__ in, const __nv_bfloat16* __restrict__ skip,
                        __nv_bfloat16* __restrict__ out) {
    const Dims dc = df.half();
    const long long pf = df.padded() * 8, pc = dc.padded() * 8;
    FOR_CELLS(df) {
        int b, x, y, z;
        df.decode(q, b, x, y, z);
        const long long p = df.pos(b, x, y, z), P = dc.pos(b, x / 2, y / 2, z / 2);
        for (int j = 0; j < C / 8; ++j) {
            const uint4 v = *reinterpret_cast<const uint4*>(in + j * pc + P * 8);
            if (skip) {
                float a[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
                acc8(a, v);
                acc8(a, *reinterpret_cast<const uint4*>(skip + j * pf + p * 8));
                *reinterpret_cast<uint4*>(out + j * pf + p * 8) = pack8(a);
            } else {
                *reinterpret_cast<uint4*>(out + j * pf + p * 8) = v;
            }
        }
    }
}
// FP32 4-channel input (training layout) -> BF16 planes 0 (channels 0-3, 4-7 zero) and 1 (zero)
__global__ void in_to_bf16(Dims d, const float* __restrict__ x4, __nv_bfloat16* __restrict__ x16) {
    const long long pl = d.padded() * 8;
    FOR_CELLS(d) {
        int b, x, y, z;
        d.decode(q, b, x, y, z);
        const long long p = d.pos(b, x, y, z);
        const float4 v = *reinterpret_cast<const float4*>(x4 + p * 4);
        const float a[8] = {v.x, v.y, v.z, v.w, 0.f, 0.f, 0.f, 0.f};
        *reinterpret_cast<uint4*>(x16 + p * 8) = pack8(a);
        *reinterpret_cast<uint4*>(x16 + pl + p * 8) = make_uint4(0u, 0u, 0u, 0u);
    }
}

// ---- preconditioner input from the solver's grid arrays.  The padded activation layout of
// a batch of one equals the solver's ghost-width-1 column-major grid layout, so the solver's
// residual, coefficients and the net output share one index p.
__global__ void absmax_k(Dims d, const float* __restrict__ r, unsigned int* __restrict__ out) {
    __shared__ unsigned int sm[256];
    unsigned int m = 0u;
    FOR_CELLS(d) {
        int b, x, y, z;
        d.decode(q, b, x, y, z);
        const unsigned int v = __float_as_uint(r[d.pos(b, x, y, z)]) & 0x7FFFFFFFu;
        m = v > m ? v : m;
    }
    sm[threadIdx.x] = m;
    __syncthreads();
    for (int w = 128; w > 0; w >>= 1) {
        if (threadIdx.x < w) sm[threadIdx.x] = sm[threadIdx.x] > sm[threadIdx.x + w] ? sm[threadIdx.x] : sm[threadIdx.x + w];
        __syncthreads();
    }
    if (threadIdx.x == 0) atomicMax(out, sm[0]);
}

// channels: r / max|r|, λρ·L_x, λρ·L_y, λρ·L_z (lower-face coefficients of the cell), zeros;
// written as 8-channel planes
__global__ void prep_k(Dims d, const float* __restrict__ r, const float* __restrict__ L, long long ncomp, float lrho,
                       const unsigned int* __restrict__ scale, __nv_bfloat16* __restrict__ x16) {
    const float sc = __uint_as_float(*scale);
    const float inv = sc > 0.f ? 1.f / sc : 0.f;
    FOR_CELLS(d) {
        int b, x, y, z;
        d.decode(q, b, x, y, z);
        const long long p = d.pos(b, x, y, z);
        const __nv_bfloat162 c01 = __floats2bfloat162_rn(r[p] * inv, lrho * L[p]);
        const __nv_bfloat162 c23 = __floats2bfloat162_rn(lrho * L[p + ncomp], lrho * L[p + 2 * ncomp]);
        // plane 0; plane 1 (channels 8-15) stays zero from the allocation
        *reinterpret_cast<uint4*>(x16 + p * 8) =
            make_uint4(*reinterpret_cast<const uint32_t*>(&c01), *reinterpret_cast<const uint32_t*>(&c23), 0u, 0u);
    }
}

}  // namespace nn

// ------------------------------------------------------------------ state
struct NNState {
    float *w = nullptr, *g = nullptr, *m = nullptr, *v = nullptr;   // FP32 parameters, gradient, Adam moments
    long long step = 0;
    int loss_kind = 0;                                               // 0 MSE, 1 energy norm
    uint8_t* wtc[nn::NLAYER] = {nullptr};                            // BF16 weights, shared-memory layout
    float* bias_tc = nullptr;                                        // padded biases (16 or 32 per layer)
    bool tc_dirty = true;
    // training activations (FP32); zeroed whenever the dims change so every halo is zero
    float* buf = nullptr;
    size_t buf_bytes = 0;
    nn::Dims buf_dims{0, 0, 0, 0};
    float* part = nullptr;                                           // the blocks' weight gradients, one layer's at a time
    int sms = 152;                                                   // multiprocessors of the device
    // inference activations (BF16), same rule
    __nv_bfloat16* ibuf = nullptr;
    size_t ibuf_bytes = 0;
    nn::Dims ibuf_dims{0, 0, 0, 0};
    // preconditioner input (BF16, 16 channels, grid-shaped) and its scale
    __nv_bfloat16* x16 = nullptr;
    size_t x16_bytes = 0;
    nn::Dims x16_dims{0, 0, 0, 0};
    unsigned int* dscale = nullptr;
    double* dloss = nullptr;
    int* derr = nullptr;
};

inline bool same_dims(const nn::Dims& a, const nn::Dims& b) {
    return a.B == b.B && a.nx == b.nx && a.ny == b.ny && a.nz == b.nz;
}

namespace {

NNState* nn_state(ia_handle* h) {
    if (h->nn) return h->nn;
    NNState* s = new NNState();
    const size_t n = (size_t)nn::NPARAM;
    cudaError_t e = cudaSuccess;
    e = e ? e : cudaMalloc(&s->w, 4 * n);
    e = e ? e : cudaMalloc(&s->g, 4 * n);
    e = e ? e : cudaMalloc(&s->m, 4 * n);
    e = e ? e : cudaMalloc(&s->v, 4 * n);
    e = e ? e : cudaMalloc(&s->dloss, 8);
    e = e ? e : cudaMalloc(&s->derr, 4);
    e = e ? e : cudaMalloc(&s->dscale, 4);
    e = e ? e : cudaMalloc(&s->bias_tc, 4 * 32 * nn::NLAYER);
    for (int l = 0; l < nn::NLAYER && !e; ++l) {
        const int co = nn::COUT[l] < 16 ? 16 : nn::COUT[l], ci = nn::CIN[l] < 16 ? 16 : nn::CIN[l];
        e = cudaMalloc(&s->wtc[l], (size_t)27 * co * ci * 2);
    }
    if (e != cudaSuccess) return nullptr;
    cudaDeviceGetAttribute(&s->sms, cudaDevAttrMultiProcessorCount, h->device);
    cudaMemset(s->w, 0, 4 * n);
    cudaMemset(s->m, 0, 4 * n);
    cudaMemset(s->v, 0, 4 * n);
    cudaMemset(s->derr, 0, 4);
    h->nn = s;
    return s;
}

float* take(float*& cur, long long n) {
    float* p = cur;
    cur += (n + 63) / 64 * 64;
    return p;
}

// padded tensor sizes (floats) of the training graph for dims d (full resolution)
struct Graph {
    nn::Dims f, hf, qt;
    float *x0, *z1, *a1, *p1, *z2, *a2, *p2, *z3, *a3, *u2, *z4, *a4, *u1, *z5, *a5, *out, *tgt;
    float *dout, *da5, *dz5, *du1, *dz4, *du2, *dz3, *dp2, *dz2, *dp1, *dz1;
};

size_t graph_floats(const nn::Dims& f) {
    const nn::Dims hf = f.half(), qt = hf.half();
    const long long F = f.padded(), H = hf.padded(), Q = qt.padded();
    const long long per = F * (4 + 16 * 3 + 32 + 16 * 2 + 1 + 1) + H * (16 + 32 * 5) + Q * (32 * 3) +
                          F * (1 + 16 * 2 + 32 + 16) + H * (16 + 32 * 3) + Q * (32 * 2);
    return (size_t)per + 64 * 40;
}

Graph carve(float* base, const nn::Dims& f) {
    Graph G;
    G.f = f;
    G.hf = f.half();
    G.qt = G.hf.half();
    const long long F = f.padded(), H = G.hf.padded(), Q = G.qt.padded();
    float* c = base;
    G.x0 = take(c, F * 4);
    G.z1 = take(c, F * 16);
    G.a1 = take(c, F * 16);
    G.p1 = take(c, H * 16);
    G.z2 = take(c, H * 32);
    G.a2 = take(c, H * 32);
    G.p2 = take(c, Q * 32);
    G.z3 = take(c, Q * 32);
    G.a3 = take(c, Q * 32);
    G.u2 = take(c, H * 32);
    G.z4 = take(c, H * 32);
    G.a4 = take(c, H * 32);
    G.u1 = take(c, F * 32);
    G.z5 = take(c, F * 16);
    G.a5 = take(c, F * 16);
    G.out = take(c, F);
    G.tgt = take(c, F);
    G.dout = take(c, F);
    G.da5 = take(c, F * 16);
    G.dz5 = take(c, F * 16);
    G.du1 = take(c, F * 32);
    G.dz4 = take(c, H * 32);
    G.du2 = take(c, H * 32);
    G.dz3 = take(c, Q * 32);
    G.dp2 = take(c, Q * 32);
    G.dz2 = take(c, H * 32);
    G.dp1 = take(c, H * 16);
    G.dz1 = take(c, F * 16);
    return G;
}

int ensure_graph(ia_handle* h, NNState* s, const nn::Dims& f, Graph& G) {
    const size_t need = graph_floats(f) * 4;
    if (need > s->buf_bytes) {
        cudaFree(s->buf);
        s->buf = nullptr;
        s->buf_bytes = 0;
        s->buf_dims = nn::Dims{0, 0, 0, 0};
        if (cudaMalloc(&s->buf, need) != cudaSuccess) return IA_ERR_CUDA;
        s->buf_bytes = need;
    }
    if (!same_dims(f, s->buf_dims)) {
        if (cudaMemsetAsync(s->buf, 0, s->buf_bytes, h->stream) != cudaSuccess) return IA_ERR_CUDA;
        s->buf_dims = f;
    }
    G = carve(s->buf, f);
    return IA_OK;
}

inline int nblk(long long n) {
    long long b = (n + 255) / 256;
    return int(b < 4096 ? (b < 1 ? 1 : b) : 4096);
}

// a data gradient on the tile that fills the device: 32 x 8 x 4 cells, 2 planes where 4 leave fewer than two blocks
// for a multiprocessor, 16 cells along x on short rows
template <int CI, int CO, int TX, int TZ>
cudaError_t conv32_tile(const nn::Dims& d, const float* dY, const float* W, float* dX, cudaStream_t st) {
    using C = nn::Conv32<CI, CO, TX, TZ>;
    const long long blocks = (long long)((d.nx + TX - 1) / TX) * ((d.ny + nn::CONV_TY - 1) / nn::CONV_TY) * ((d.nz + TZ - 1) / TZ) * d.B;
    const cudaError_t e = cudaFuncSetAttribute(nn::conv32_k<CI, CO, TX, TZ>, cudaFuncAttributeMaxDynamicSharedMemorySize, C::BYTES);
    if (e != cudaSuccess) return e;
    { nn::conv32_k<CI, CO, TX, TZ><<<unsigned(blocks), C::THREADS, C::BYTES, st>>>(d, dY, W, dX); ia::note_launch(); }
    return cudaGetLastError();
}
template <int CI, int CO>
cudaError_t conv32(const NNState* s, const nn::Dims& d, const float* dY, const float* W, float* dX, cudaStream_t st) {
    if (d.nx <= 16) return conv32_tile<CI, CO, 16, 2>(d, dY, W, dX, st);
    const long long blocks = (long long)((d.nx + 31) / 32) * ((d.ny + nn::CONV_TY - 1) / nn::CONV_TY) * ((d.nz + 3) / 4) * d.B;
    if (blocks < 2 * s->sms) return conv32_tile<CI, CO, 32, 2>(d, dY, W, dX, st);
    return conv32_tile<CI, CO, 32, 4>(d, dY, W, dX, st);
}
// a layer's forward convolution: 32 x 8 x 4 cells, 2 planes where 4 leave more than half of the multiprocessors without a
// block (the layers together, 4 samples of 64^3: 1412 us, 1440 by the data gradient's rule; one sample 546 and 571)
template <int CI, int CO, int TX, int TZ>
cudaError_t fwd32_tile(const nn::Dims& d, const float* X, const float* W, const float* b, float* Z, float* A, const float* skip,
                       int relu, cudaStream_t st) {
    using C = nn::Fwd32<CI, CO, TX, TZ>;
    const long long blocks = (long long)((d.nx + TX - 1) / TX) * ((d.ny + nn::CONV_TY - 1) / nn::CONV_TY) * ((d.nz + TZ - 1) / TZ) * d.B;
    const cudaError_t e = cudaFuncSetAttribute(nn::fwd32_k<CI, CO, TX, TZ>, cudaFuncAttributeMaxDynamicSharedMemorySize, C::BYTES);
    if (e != cudaSuccess) return e;
    { nn::fwd32_k<CI, CO, TX, TZ><<<unsigned(blocks), C::THREADS, C::BYTES, st>>>(d, X, W, b, Z, A, skip, relu); ia::note_launch(); }
    return cudaGetLastError();
}
template <int CI, int CO>
cudaError_t fwd32(const NNState* s, const nn::Dims& d, const float* X, const float* W, const float* b, float* Z, float* A,
                  const float* skip, int relu, cudaStream_t st) {
    if (d.nx <= 16) return fwd32_tile<CI, CO, 16, 2>(d, X, W, b, Z, A, skip, relu, st);
    const long long blocks = (long long)((d.nx + 31) / 32) * ((d.ny + nn::CONV_TY - 1) / nn::CONV_TY) * ((d.nz + 3) / 4) * d.B;
    if (2 * blocks < s->sms) return fwd32_tile<CI, CO, 32, 2>(d, X, W, b, Z, A, skip, relu, st);
    return fwd32_tile<CI, CO, 32, 4>(d, X, W, b, Z, A, skip, relu, st);
}
// gradients of the weights and the bias of a layer into g (W[27][CO][CI], then b[CO])
template <int CI, int CO>
cudaError_t wgrad(const NNState* s, const nn::Dims& d, const float* X, const float* dY, float* g, cudaStream_t st) {
    using G = nn::Wgrad<CI, CO>;
    const long long tiles = (long long)((d.nx + nn::WG_X - 1) / nn::WG_X) * ((d.ny + nn::WG_Y - 1) / nn::WG_Y) *
                            ((d.nz + nn::WG_Z - 1) / nn::WG_Z) * d.B;
    const int blocks = int(std::min<long long>(tiles, nn::WG_BLOCKS * s->sms));
    const cudaError_t e = cudaFuncSetAttribute(nn::wgrad_k<CI, CO>, cudaFuncAttributeMaxDynamicSharedMemorySize, 4 * G::SM);
    if (e != cudaSuccess) return e;
    { nn::wgrad_k<CI, CO><<<blocks, G::THREADS, 4 * G::SM, st>>>(d, X, dY, s->part, int(tiles)); ia::note_launch(); }
    { nn::wgrad_sum_k<<<(G::N + 31) / 32, 256, 0, st>>>(s->part, blocks, G::N, g); ia::note_launch(); }
    return cudaGetLastError();
}

inline float4* v4(float* p) { return reinterpret_cast<float4*>(p); }

// forward of the training graph (inputs already in G.x0)
cudaError_t forward_f32(const NNState* s, const Graph& G, cudaStream_t st) {
    using namespace nn;
    const float* w = s->w;
    cudaError_t e = fwd32<4, 16>(s, G.f, G.x0, w + layer_w(0), w + layer_b(0), G.z1, G.a1, nullptr, 1, st);
    { pool_fwd_k<<<nblk(G.hf.cells() * 4), 256, 0, st>>>(G.hf, 4, v4(G.a1), v4(G.p1)); ia::note_launch(); }
    e = e ? e : fwd32<16, 32>(s, G.hf, G.p1, w + layer_w(1), w + layer_b(1), G.z2, G.a2, nullptr, 1, st);
    { pool_fwd_k<<<nblk(G.qt.cells() * 8), 256, 0, st>>>(G.qt, 8, v4(G.a2), v4(G.p2)); ia::note_launch(); }
    e = e ? e : fwd32<32, 32>(s, G.qt, G.p2, w + layer_w(2), w + layer_b(2), G.z3, G.a3, nullptr, 1, st);
    { up_fwd_k<<<nblk(G.hf.cells() * 8), 256, 0, st>>>(G.hf, 8, v4(G.a3), v4(G.a2), v4(G.u2)); ia::note_launch(); }
    e = e ? e : fwd32<32, 32>(s, G.hf, G.u2, w + layer_w(3), w + layer_b(3), G.z4, G.a4, nullptr, 1, st);
    { up_fwd_k<<<nblk(G.f.cells() * 8), 256, 0, st>>>(G.f, 8, v4(G.a4), nullptr, v4(G.u1)); ia::note_launch(); }
    e = e ? e : fwd32<32, 16>(s, G.f, G.u1, w + layer_w(4), w + layer_b(4), G.z5, G.a5, G.a1, 1, st);
    e = e ? e : fwd32<16, 1>(s, G.f, G.a5, w + layer_w(5), w + layer_b(5), nullptr, G.out, nullptr, 0, st);
    return e ? e : cudaGetLastError();
}

cudaError_t backward_f32(const NNState* s, const Graph& G, cudaStream_t st) {
    using namespace nn;
    const float* w = s->w;
    float* g = s->g;
    // data gradient of layer l
    auto W = [&](int l) { return w + layer_w(l); };
    cudaError_t e = wgrad<16, 1>(s, G.f, G.a5, G.dout, g + layer_w(5), st);
    e = e ? e : conv32<1, 16>(s, G.f, G.dout, W(5), G.da5, st);
    { relu_bwd_k<<<nblk(G.f.cells() * 4), 256, 0, st>>>(G.f, 4, v4(G.z5), v4(G.da5), v4(G.dz5)); ia::note_launch(); }
    e = e ? e : wgrad<32, 16>(s, G.f, G.u1, G.dz5, g + layer_w(4), st);
    e = e ? e : conv32<16, 32>(s, G.f, G.dz5, W(4), G.du1, st);
    { up_bwd_relu_k<<<nblk(G.hf.cells() * 8), 256, 0, st>>>(G.hf, 8, v4(G.du1), v4(G.z4), v4(G.dz4)); ia::note_launch(); }
    e = e ? e : wgrad<32, 32>(s, G.hf, G.u2, G.dz4, g + layer_w(3), st);
    e = e ? e : conv32<32, 32>(s, G.hf, G.dz4, W(3), G.du2, st);
    { up_bwd_relu_k<<<nblk(G.qt.cells() * 8), 256, 0, st>>>(G.qt, 8, v4(G.du2), v4(G.z3), v4(G.dz3)); ia::note_launch(); }
    e = e ? e : wgrad<32, 32>(s, G.qt, G.p2, G.dz3, g + layer_w(2), st);
    e = e ? e : conv32<32, 32>(s, G.qt, G.dz3, W(2), G.dp2, st);
    // a2 feeds the skip connection (du2) and the pooling (dp2)
    { pool_bwd_relu_k<<<nblk(G.hf.cells() * 8), 256, 0, st>>>(G.hf, 8, v4(G.du2), v4(G.dp2), v4(G.z2), v4(G.dz2)); ia::note_launch(); }
    e = e ? e : wgrad<16, 32>(s, G.hf, G.p1, G.dz2, g + layer_w(1), st);
    e = e ? e : conv32<32, 16>(s, G.hf, G.dz2, W(1), G.dp1, st);
    // a1 feeds the skip connection (da5) and the pooling (dp1)
    { pool_bwd_relu_k<<<nblk(G.f.cells() * 4), 256, 0, st>>>(G.f, 4, v4(G.da5), v4(G.dp1), v4(G.z1), v4(G.dz1)); ia::note_launch(); }
    e = e ? e : wgrad<4, 16>(s, G.f, G.x0, G.dz1, g + layer_w(0), st);
    return e ? e : cudaGetLastError();
}

int loss_grad(ia_handle* h, NNState* s, const float* x0, const float* tgt, const nn::Dims& f, double* loss_out) {
    cudaStream_t st = h->stream;
    Graph G;
    if (ensure_graph(h, s, f, G) != IA_OK) return IA_ERR_CUDA;
    cudaMemcpyAsync(G.x0, x0, sizeof(float) * f.padded() * 4, cudaMemcpyDeviceToDevice, st);
    cudaMemcpyAsync(G.tgt, tgt, sizeof(float) * f.padded(), cudaMemcpyDeviceToDevice, st);
    if (forward_f32(s, G, st) != cudaSuccess) return IA_ERR_CUDA;
    cudaMemsetAsync(s->dloss, 0, 8, st);
    const int nbl = nblk(f.cells()) < 1024 ? nblk(f.cells()) : 1024;
    if (s->loss_kind == 1) { nn::energy_k<<<nbl, 256, 0, st>>>(f, G.out, G.tgt, G.x0, G.dout, s->dloss); ia::note_launch(); }
    else { nn::mse_k<<<nbl, 256, 0, st>>>(f, G.out, G.tgt, G.dout, s->dloss); ia::note_launch(); }
    if (!s->part && cudaMalloc(&s->part, sizeof(float) * (size_t)(nn::WG_BLOCKS * s->sms) * nn::Wgrad<32, 32>::N) != cudaSuccess)
        return IA_ERR_CUDA;
    if (backward_f32(s, G, st) != cudaSuccess) return IA_ERR_CUDA;
    if (loss_out) {
        cudaMemcpyAsync(loss_out, s->dloss, 8, cudaMemcpyDeviceToHost, st);
        if (cudaStreamSynchronize(st) != cudaSuccess) return IA_ERR_CUDA;
    }
    return cudaGetLastError() == cudaSuccess ? IA_OK : IA_ERR_CUDA;
}

// FP32 parameters -> BF16 tiles in the tcgen05 shared-memory layout (host-side re-arrangement)
int build_tc_weights(ia_handle* h, NNState* s) {
    std::vector<float> w((size_t)nn::NPARAM);
    if (cudaMemcpy(w.data(), s->w, 4 * w.size(), cudaMemcpyDeviceToHost) != cudaSuccess) return IA_ERR_CUDA;
    std::vector<float> biases(32 * nn::NLAYER, 0.f);
    for (int l = 0; l < nn::NLAYER; ++l) {
        const int CI = nn::CIN[l], CO = nn::COUT[l];
        const int ci = CI < 16 ? 16 : CI, co = CO < 16 ? 16 : CO;
        const uint32_t SBO = ci * 16;
        std::vector<__nv_bfloat16> t((size_t)27 * co * ci, __float2bfloat16(0.f));
        for (int tap = 0; tap < 27; ++tap)
            for (int n = 0; n < CO; ++n)
                for (int k = 0; k < CI; ++k) {
                    const float v = w[nn::layer_w(l) + ((long long)tap * CO + n) * CI + k];
                    const size_t byte = (size_t)tap * co * ci * 2 + (n / 8) * SBO + (k / 8) * 128 + (n % 8) * 16 + (k % 8) * 2;
                    t[byte / 2] = __float2bfloat16(v);
                }
        if (cudaMemcpy(s->wtc[l], t.data(), t.size() * 2, cudaMemcpyHostToDevice) != cudaSuccess) return IA_ERR_CUDA;
        for (int n = 0; n < CO; ++n) biases[32 * l + n] = w[nn::layer_b(l) + n];
    }
    if (cudaMemcpy(s->bias_tc, biases.data(), 4 * biases.size(), cudaMemcpyHostToDevice) != cudaSuccess)
        return IA_ERR_CUDA;
    s->tc_dirty = false;
    return IA_OK;
}

// cuTensorMapEncodeTiled from the driver, without linking libcuda
using EncodeTiled = CUresult (*)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                 const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                 CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
EncodeTiled encode_tiled() {
    static EncodeTiled fn = nullptr;
    static bool tried = false;
    if (!tried) {
        tried = true;
        void* p = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &p, 12000, cudaEnableDefault, &q) ==
                cudaSuccess && q == cudaDriverEntryPointSuccess)
            fn = reinterpret_cast<EncodeTiled>(p);
    }
    return fn;
}

// tensor map of a BF16 activation stored as Cin/8 planes of 8 channels: (channel and x, y, z and batch, plane) of
// the padded cells, box = one z plane of a patch with its halo, every plane; loads past an end read zeros
bool make_act_map(CUtensorMap* m, const __nv_bfloat16* X, int CI, const nn::Dims& d) {
    EncodeTiled enc = encode_tiled();
    if (!enc) return false;
    const cuuint64_t nx = d.nx + 2, ny = d.ny + 2, nz = (cuuint64_t)(d.nz + 2) * d.B;
    const cuuint64_t dims[4] = {8 * nx, ny, nz, (cuuint64_t)(CI / 8)};
    const cuuint64_t strides[3] = {16 * nx, 16 * nx * ny, 16 * nx * ny * nz};
    const cuuint32_t box[4] = {8 * nn::kBX, (cuuint32_t)nn::kBY, 1, (cuuint32_t)(CI / 8)};
    const cuuint32_t estr[4] = {1, 1, 1, 1};
    return enc(m, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 4, const_cast<__nv_bfloat16*>(X), dims, strides, box, estr,
               CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
               CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

template <int CI, int CO, bool RELU, bool OUTF32>
cudaError_t launch_tma(const nn::Dims& d, const __nv_bfloat16* X, const uint8_t* W, const float* b,
                       const __nv_bfloat16* skip, __nv_bfloat16* Y, float* Yf, int* err, cudaStream_t st, int sms) {
    using Sm = nn::TmaSmem<CI, CO < 16 ? 16 : CO>;
    CUtensorMap map;
    if (!make_act_map(&map, X, CI, d)) return cudaErrorNotSupported;
    auto kfn = nn::conv_tma_kernel<CI, CO, RELU, OUTF32>;
    cudaError_t e = cudaFuncSetAttribute(kfn, cudaFuncAttributeMaxDynamicSharedMemorySize, Sm::TOTAL);
    if (e != cudaSuccess) return e;
    // output planes of an item: z cut evenly; shorter cuts where the patches alone would leave multiprocessors idle
    const long long patches = (long long)((d.nx + nn::kPX - 1) / nn::kPX) * ((d.ny + nn::kPY - 1) / nn::kPY) * d.B;
    long long cuts = (d.nz + Sm::ZP - 1) / Sm::ZP;
    cuts = std::min<long long>(std::max<long long>(cuts, 2ll * sms / patches), std::max(1, d.nz / 4));
    cuts = std::max<long long>(cuts, (d.nz + Sm::ZP - 1) / Sm::ZP);
    const int zc = int((d.nz + cuts - 1) / cuts);
    const long long items = patches * ((d.nz + zc - 1) / zc);
    if (items > 0x7fffffffll) return cudaErrorInvalidValue;
    const int grid = int(std::min<long long>(items, 2ll * sms));
    { kfn<<<grid, nn::kConvThreads, Sm::TOTAL, st>>>(map, d, zc, W, b, skip, Y, Yf, err); ia::note_launch(); }
    return cudaGetLastError();
}

// one convolution layer of the inference path
#define conv_layer(CI_, CO_, RELU_, F32_, dims, X_, W_, B_, SK_, Y_, YF_) \
    launch_tma<CI_, CO_, RELU_, F32_>(dims, X_, W_, B_, SK_, Y_, YF_, s->derr, st, sms)

// inference with the tensor-core kernels; x16 = BF16 16-channel input, out = FP32 channel
int forward_tc(ia_handle* h, NNState* s, const nn::Dims& f, const __nv_bfloat16* x16, float* out) {
    cudaStream_t st = h->stream;
    if (s->tc_dirty && build_tc_weights(h, s) != IA_OK) return IA_ERR_CUDA;
    const nn::Dims hf = f.half(), qt = hf.half();
    const long long F = f.padded(), H = hf.padded(), Q = qt.padded();
    const size_t need = 2 * (size_t)(F * (16 + 32 + 16) + H * (16 + 32 * 3) + Q * (32 * 2) + 64 * 16);
    if (need > s->ibuf_bytes) {
        cudaFree(s->ibuf);
        s->ibuf = nullptr;
        s->ibuf_bytes = 0;
        s->ibuf_dims = nn::Dims{0, 0, 0, 0};
        if (cudaMalloc(&s->ibuf, need) != cudaSuccess) return IA_ERR_CUDA;
        s->ibuf_bytes = need;
    }
    if (!same_dims(f, s->ibuf_dims)) {   // halos must be zero: the kernels write interior cells only
        if (cudaMemsetAsync(s->ibuf, 0, s->ibuf_bytes, st) != cudaSuccess) return IA_ERR_CUDA;
        s->ibuf_dims = f;
    }
    __nv_bfloat16* c = s->ibuf;
    auto tk = [&](long long n) { __nv_bfloat16* p = c; c += (n + 63) / 64 * 64; return p; };
    __nv_bfloat16 *a1 = tk(F * 16), *u1 = tk(F * 32), *a5 = tk(F * 16), *p1 = tk(H * 16), *a2 = tk(H * 32),
                  *u2 = tk(H * 32), *a4 = tk(H * 32), *p2 = tk(Q * 32), *a3 = tk(Q * 32);
    const int sms = s->sms;
    const float* b = s->bias_tc;
    cudaError_t e = cudaSuccess;
    e = e ? e : conv_layer(16, 16, true, false, f, x16, s->wtc[0], b + 0, nullptr, a1, nullptr);
    if (!e) { nn::pool_bf16<<<nblk(hf.cells()), 256, 0, st>>>(hf, 16, a1, p1); ia::note_launch(); }
    e = e ? e : conv_layer(16, 32, true, false, hf, p1, s->wtc[1], b + 32, nullptr, a2, nullptr);
    if (!e) { nn::pool_bf16<<<nblk(qt.cells()), 256, 0, st>>>(qt, 32, a2, p2); ia::note_launch(); }
    e = e ? e : conv_layer(32, 32, true, false, qt, p2, s->wtc[2], b + 64, nullptr, a3, nullptr);
    if (!e) { nn::up_bf16<<<nblk(hf.cells()), 256, 0, st>>>(hf, 32, a3, a2, u2); ia::note_launch(); }
    e = e ? e : conv_layer(32, 32, true, false, hf, u2, s->wtc[3], b + 96, nullptr, a4, nullptr);
    if (!e) { nn::up_bf16<<<nblk(f.cells()), 256, 0, st>>>(f, 32, a4, nullptr, u1); ia::note_launch(); }
    e = e ? e : conv_layer(32, 16, true, false, f, u1, s->wtc[4], b + 128, a1, a5, nullptr);
    e = e ? e : conv_layer(16, 1, false, true, f, a5, s->wtc[5], b + 160, nullptr, nullptr, out);
    return e == cudaSuccess ? IA_OK : IA_ERR_CUDA;
}

// the BF16 input of the inference path (16 channels), its halo and the channels that no one writes zero
int ensure_x16(NNState* s, const nn::Dims& f, cudaStream_t st) {
    const size_t need = 2 * 16 * (size_t)f.padded();
    if (need > s->x16_bytes) {
        cudaFree(s->x16);
        s->x16 = nullptr;
        s->x16_bytes = 0;
        s->x16_dims = nn::Dims{0, 0, 0, 0};
        if (cudaMalloc(&s->x16, need) != cudaSuccess) return IA_ERR_CUDA;
        s->x16_bytes = need;
    }
    if (!same_dims(f, s->x16_dims)) {
        if (cudaMemsetAsync(s->x16, 0, need, st) != cudaSuccess) return IA_ERR_CUDA;
        s->x16_dims = f;
    }
    return IA_OK;
}

int check_dims(int B, int nx, int ny, int nz) {
    if (B < 1 || nx < 4 || ny < 4 || nz < 4 || nx % 4 || ny % 4 || nz % 4) return IA_ERR_INVALID;
    return IA_OK;
}

}  // namespace

// Preconditioner application for the Poisson solver: out (FP32, grid layout, interior cells
// written) = net(r / max|r|, λρ·L) on a 3D grid with interior dims nx, ny, nz.
int nn_apply(ia_handle* h, const float* r, const float* L32, float* out, int nx, int ny, int nz, long long ncomp) {
    NNState* s = nn_state(h);
    if (!s) return IA_ERR_CUDA;
    cudaStream_t st = h->stream;
    const nn::Dims f{1, nx, ny, nz};
    if (ensure_x16(s, f, st) != IA_OK) return IA_ERR_CUDA;
    cudaMemsetAsync(s->dscale, 0, 4, st);
    const int nb = nblk(f.cells()) < 1216 ? nblk(f.cells()) : 1216;
    { nn::absmax_k<<<nb, 256, 0, st>>>(f, r, s->dscale); ia::note_launch(); }
    { nn::prep_k<<<nblk(f.cells()), 256, 0, st>>>(f, r, L32, ncomp, float(h->cfg.lrho), s->dscale, s->x16); ia::note_launch(); }
    return forward_tc(h, s, f, s->x16, out);
}
int nn_error_flag(ia_handle* h) {
    if (!h->nn) return 0;
    int v = 0;
    cudaMemcpy(&v, h->nn->derr, 4, cudaMemcpyDeviceToHost);
    return v;
}
void nn_destroy(ia_handle* h) {
    NNState* s = h->nn;
    if (!s) return;
    cudaFree(s->w); cudaFree(s->g); cudaFree(s->m); cudaFree(s->v);
    for (int l = 0; l < nn::NLAYER; ++l) cudaFree(s->wtc[l]);
    cudaFree(s->bias_tc); cudaFree(s->buf); cudaFree(s->part); cudaFree(s->ibuf); cudaFree(s->x16);
    cudaFree(s->dloss); cudaFree(s->derr); cudaFree(s->dscale);
    delete s;
    h->nn = nullptr;
}

}  // namespace ia

using namespace ia;

extern "C" {

int64_t ia_nn_param_count(void) { return nn::NPARAM; }

int ia_nn_set_params(ia_handle* h, const float* params) {
    if (!h || !params) return IA_ERR_INVALID;
    NNState* s = nn_state(h);
    if (!s) return IA_ERR_CUDA;
    if (cudaMemcpy(s->w, params, 4 * (size_t)nn::NPARAM, cudaMemcpyHostToDevice) != cudaSuccess) return IA_ERR_CUDA;
    cudaMemset(s->m, 0, 4 * (size_t)nn::NPARAM);
    cudaMemset(s->v, 0, 4 * (size_t)nn::NPARAM);
    s->step = 0;
    s->tc_dirty = true;
    return IA_OK;
}

int ia_nn_set_loss(ia_handle* h, int32_t kind) {
    if (!h || kind < 0 || kind > 1) return IA_ERR_INVALID;
    NNState* s = nn_state(h);
    if (!s) return IA_ERR_CUDA;
    s->loss_kind = kind;
    return IA_OK;
}

int ia_nn_get_params(ia_handle* h, float* params) {
    if (!h || !params) return IA_ERR_INVALID;
    NNState* s = nn_state(h);
    if (!s) return IA_ERR_CUDA;
    return cuda_fail(cudaMemcpy(params, s->w, 4 * (size_t)nn::NPARAM, cudaMemcpyDeviceToHost));
}

int ia_nn_forward(ia_handle* h, const float* x0, float* out, int32_t B, int32_t nx, int32_t ny, int32_t nz,
                  int32_t tensor_cores) {
    if (!h || !x0 || !out) return IA_ERR_INVALID;
    if (check_dims(B, nx, ny, nz) != IA_OK) return IA_ERR_INVALID;
    NNState* s = nn_state(h);
    if (!s) return IA_ERR_CUDA;
    const nn::Dims f{B, nx, ny, nz};
    cudaStream_t st = h->stream;
    if (!tensor_cores) {
        Graph G;
        if (ensure_graph(h, s, f, G) != IA_OK) return IA_ERR_CUDA;
        cudaMemcpyAsync(G.x0, x0, sizeof(float) * f.padded() * 4, cudaMemcpyDeviceToDevice, st);
        if (forward_f32(s, G, st) != cudaSuccess) return IA_ERR_CUDA;
        cudaMemcpyAsync(out, G.out, sizeof(float) * f.padded(), cudaMemcpyDeviceToDevice, st);
        return cuda_fail(cudaStreamSynchronize(st));
    }
    if (ensure_x16(s, f, st) != IA_OK) return IA_ERR_CUDA;
    { nn::in_to_bf16<<<nblk(f.cells()), 256, 0, st>>>(f, x0, s->x16); ia::note_launch(); }
    cudaMemsetAsync(s->derr, 0, 4, st);
    if (forward_tc(h, s, f, s->x16, out) != IA_OK) return IA_ERR_CUDA;
    int err = 0;
    cudaError_t e = cudaMemcpyAsync(&err, s->derr, 4, cudaMemcpyDeviceToHost, st);
    if (e == cudaSuccess) e = cudaStreamSynchronize(st);
    return e != cudaSuccess || err ? IA_ERR_CUDA : IA_OK;
}

int ia_nn_loss_grad(ia_handle* h, const float* x0, const float* target, int32_t B, int32_t nx, int32_t ny,
                    int32_t nz, float* grad, double* loss) {
    if (!h || !x0 || !target) return IA_ERR_INVALID;
    if (check_dims(B, nx, ny, nz) != IA_OK) return IA_ERR_INVALID;
    NNState* s = nn_state(h);
    if (!s) return IA_ERR_CUDA;
    int rc = loss_grad(h, s, x0, target, nn::Dims{B, nx, ny, nz}, loss);
    if (rc != IA_OK) return rc;
    if (grad) cudaMemcpyAsync(grad, s->g, 4 * (size_t)nn::NPARAM, cudaMemcpyDeviceToDevice, h->stream);
    return cuda_fail(cudaStreamSynchronize(h->stream));
}

int ia_nn_train_step(ia_handle* h, const float* x0, const float* target, int32_t B, int32_t nx, int32_t ny,
                     int32_t nz, float lr, double* loss) {
    if (!h || !x0 || !target) return IA_ERR_INVALID;
    if (check_dims(B, nx, ny, nz) != IA_OK) return IA_ERR_INVALID;
    NNState* s = nn_state(h);
    if (!s) return IA_ERR_CUDA;
    int rc = loss_grad(h, s, x0, target, nn::Dims{B, nx, ny, nz}, nullptr);
    if (rc != IA_OK) return rc;
    s->step += 1;
    const float b1 = 0.9f, b2 = 0.999f;
    const float c1 = 1.f - std::pow(b1, float(s->step)), c2 = 1.f - std::pow(b2, float(s->step));
    { nn::adam_k<<<256, 256, 0, h->stream>>>(nn::NPARAM, s->w, s->g, s->m, s->v, lr, b1, b2, 1e-8f, c1, c2); ia::note_launch(); }
    s->tc_dirty = true;
    if (loss) {
        cudaMemcpyAsync(loss, s->dloss, 8, cudaMemcpyDeviceToHost, h->stream);
    }
    return cuda_fail(cudaStreamSynchronize(h->stream));
}

}  // extern "C"
