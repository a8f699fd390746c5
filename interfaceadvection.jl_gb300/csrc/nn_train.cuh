// FP32 training kernels of the learned preconditioner's network (included by nn.cu): the 3x3x3 convolution,
// its data gradient, the weight gradient, and the pooling / upsampling / ReLU passes between them.
//
// The contractions run on the FP32 pipes: the gradients are checked against FP64 at 5e-5 and the BF16 and TF32
// tensor formats round their inputs to 8 and 11 bits.  The bound is therefore the FMA rate, and the kernels are
// built so that a multiply-add costs little else: 64 (convolution) or 48 (weight gradient) accumulators a thread,
// operands read from shared memory as vectors and used 12 to 24 times each.
// Measured on GB300, 4 samples of 64^3 (136 GFLOP in all, 1.8 ms at the measured FMA rate): 38.4 ms for one
// gradient with a thread per cell and scalar loads, 4.3 ms with these kernels.
#pragma once

namespace ia {
namespace nn {

// ------------------------------------------------------------------ data gradient
// dX[p][o] = Σ_t Σ_c W[26 - t][c][o] dY[p + off(t)][c] on a tile of TX x 8 x TZ cells (CI: channels of dY).  A thread owns
// 8 consecutive cells of a row and COT channels of dX.  The tile of dY (with its halo) is staged channel by channel,
// x fastest, CC channels at a time: for one channel and one (dy, dz) a thread reads 10 values and multiplies them
// by the 3 x COT weights of the row, which are the same for its whole warp.
constexpr int CONV_TY = 8;
template <int CI, int CO, int TX, int TZ>
struct Conv32 {
    static constexpr int CC = CI < 8 ? CI : 8;
    static constexpr int COT = 8;
    static constexpr int PX = TX + 4;                                  // row pitch: 16-byte rows, no bank conflicts at TX = 32
    static constexpr int XN = CC * (TZ + 2) * (CONV_TY + 2) * PX;      // staged inputs (floats)
    static constexpr int WN = 27 * CC * CO;                            // staged weights
    static constexpr int THREADS = TX / 8 * CONV_TY * TZ * (CO / COT);
    static constexpr int BYTES = 4 * (XN + WN);
};

template <int CI, int CO, int TX, int TZ>
__global__ void __launch_bounds__(Conv32<CI, CO, TX, TZ>::THREADS, 512 / Conv32<CI, CO, TX, TZ>::THREADS)
conv32_k(Dims d, const float* __restrict__ dY, const float* __restrict__ W, float* __restrict__ dX) {
    using C = Conv32<CI, CO, TX, TZ>;
    constexpr int CC = C::CC, COT = C::COT, PX = C::PX, RX = TX + 2, RY = CONV_TY + 2, RZ = TZ + 2;
    extern __shared__ __align__(16) float conv_sm[];
    float* xs = conv_sm;
    float* ws = conv_sm + C::XN;
    const int tid = threadIdx.x;
    const int j = tid % (TX / 8), ty = tid / (TX / 8) % CONV_TY, tz = tid / (TX / 8 * CONV_TY) % TZ;
    const int o0 = tid / (TX / 8 * CONV_TY * TZ) * COT;
    // tile origin
    const int ntx = (d.nx + TX - 1) / TX, nty = (d.ny + CONV_TY - 1) / CONV_TY, ntz = (d.nz + TZ - 1) / TZ;
    int t = blockIdx.x;
    const int x0 = t % ntx * TX;
    t /= ntx;
    const int y0 = t % nty * CONV_TY;
    t /= nty;
    const int z0 = t % ntz * TZ, b = t / ntz;
    float acc[8][COT];
#pragma unroll
    for (int o = 0; o < COT; ++o)
#pragma unroll
        for (int i = 0; i < 8; ++i) acc[i][o] = 0.f;
    for (int c0 = 0; c0 < CI; c0 += CC) {
        if (c0) __syncthreads();
        for (int e = tid; e < RX * RY * RZ; e += C::THREADS) {
            const int rx = e % RX, r = e / RX, ry = r % RY, rz = r / RY;
            const bool in = x0 + rx < d.nx + 2 && y0 + ry < d.ny + 2 && z0 + rz < d.nz + 2;   // the padded tensor
            float v[CC];
            if (in) {
                const float* src = dY + d.pos(b, x0 + rx - 1, y0 + ry - 1, z0 + rz - 1) * CI + c0;
                if (CC % 4 == 0) {
#pragma unroll
                    for (int q = 0; q < CC / 4; ++q) {
                        const float4 f = __ldg(reinterpret_cast<const float4*>(src) + q);
                        v[4 * q] = f.x; v[4 * q + 1] = f.y; v[4 * q + 2] = f.z; v[4 * q + 3] = f.w;
                    }
                } else {
#pragma unroll
                    for (int c = 0; c < CC; ++c) v[c] = __ldg(src + c);
                }
            } else {
#pragma unroll
                for (int c = 0; c < CC; ++c) v[c] = 0.f;
            }
#pragma unroll
            for (int c = 0; c < CC; ++c) xs[((c * RZ + rz) * RY + ry) * PX + rx] = v[c];
        }
        // weights as ws[(row (dz, dy) * CC + c) * 3 + dx][o]
        for (int e = tid; e < C::WN; e += C::THREADS) {
            const int o = e % CO, r = e / CO, dx = r % 3, rc = r / 3, c = rc % CC, tap = rc / CC * 3 + dx;
            ws[e] = __ldg(W + ((26 - tap) * CI + c0 + c) * CO + o);
        }
        __syncthreads();
#pragma unroll 1
        for (int row = 0; row < 9; ++row) {
            const float* xr = xs + ((tz + row / 3) * RY + ty + row % 3) * PX + 8 * j;
            const float* wr = ws + row * CC * 3 * CO + o0;
#pragma unroll 2
            for (int c = 0; c < CC; ++c) {
                float xv[10];
                *reinterpret_cast<float4*>(xv) = *reinterpret_cast<const float4*>(xr);
                *reinterpret_cast<float4*>(xv + 4) = *reinterpret_cast<const float4*>(xr + 4);
                *reinterpret_cast<float2*>(xv + 8) = *reinterpret_cast<const float2*>(xr + 8);
#pragma unroll
                for (int dx = 0; dx < 3; ++dx) {
                    float wv[COT];
                    *reinterpret_cast<float4*>(wv) = *reinterpret_cast<const float4*>(wr + dx * CO);
                    *reinterpret_cast<float4*>(wv + 4) = *reinterpret_cast<const float4*>(wr + dx * CO + 4);
#pragma unroll
                    for (int i = 0; i < 8; ++i)
#pragma unroll
                        for (int o = 0; o < COT; ++o) acc[i][o] = fmaf(wv[o], xv[i + dx], acc[i][o]);
                }
                xr += RZ * RY * PX;
                wr += 3 * CO;
            }
        }
    }
    const int y = y0 + ty, z = z0 + tz;
    if (y >= d.ny || z >= d.nz) return;
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        const int x = x0 + 8 * j + i;
        if (x >= d.nx) break;
        const long long q = d.pos(b, x, y, z) * CO + o0;
#pragma unroll
        for (int h = 0; h < 8; h += 4)
            *reinterpret_cast<float4*>(dX + q + h) = make_float4(acc[i][h], acc[i][h + 1], acc[i][h + 2], acc[i][h + 3]);
    }
}

// ------------------------------------------------------------------ forward convolution
// out[p][o] = bias[o] + Σ_t Σ_c W[t][o][c] X[p + off(t)][c], summed in that order: one chain of multiply-adds from the bias,
// tap by tap with the channels inside.  The order decides the ReLU units whose input is zero but for rounding, and a few
// such units move a gradient by 1e-6 to 1e-5 of its norm, so that it is part of the result; the data gradient, which
// decides nothing, takes the channels in chunks.
// A thread owns 8 cells and COT channels as above.  All channels are staged at once, the planes of one dz at a time: TZ
// planes in a ring (a further dz replaces one of them), and the weights of its 9 taps.  A tap reads its own 8 values of
// the row, 1.6 times the loads of the chunked order, which still issue beside the multiply-adds; with few channels the
// rows stay in registers for three taps.  The forward convolutions of 4 samples of 64^3: 1.41 ms so, 1.30 ms in chunks of
// channels; of the first, whose loads are few, 126 and 124 us, of 32 -> 16 channels at full resolution (8 warps a
// multiprocessor, as many as 32 channels leave room for) 795 and 712.
template <int CI, int CO, int TX, int TZ>
struct Fwd32 {
    static constexpr int COT = CO < 8 ? CO : 8;
    static constexpr int PX = TX + 4;
    static constexpr int PLANE = (CONV_TY + 2) * PX;                   // one channel of one plane (floats)
    static constexpr int XN = CI * TZ * PLANE;
    static constexpr int WN = 9 * CI * CO;
    static constexpr int THREADS = TX / 8 * CONV_TY * TZ * (CO / COT);
    static constexpr int BYTES = 4 * (XN + WN);
    // channels whose rows a thread holds at once: all of them where 10 values each fit beside the 8·COT sums
    static constexpr int ROWS = CI * 10 + 8 * COT <= 176 && (COT == 1 || CI == 4) ? CI : 1;
    static constexpr int UNROLL = ROWS == CI ? CI : 8;
    // blocks on a multiprocessor: 512 threads, or what shared memory leaves
    static constexpr int FIT = 220 * 1024 / BYTES, BLOCKS = 512 / THREADS < FIT ? 512 / THREADS : FIT < 1 ? 1 : FIT;
};

template <int CI, int CO, int TX, int TZ>
__global__ void __launch_bounds__(Fwd32<CI, CO, TX, TZ>::THREADS, Fwd32<CI, CO, TX, TZ>::BLOCKS)
fwd32_k(Dims d, const float* __restrict__ X, const float* __restrict__ W, const float* __restrict__ bias,
        float* __restrict__ Z, float* __restrict__ A, const float* __restrict__ skip, int relu) {
    using C = Fwd32<CI, CO, TX, TZ>;
    constexpr int COT = C::COT, PX = C::PX, RX = TX + 2, RY = CONV_TY + 2, ROWS = C::ROWS;
    extern __shared__ __align__(16) float conv_sm[];
    float* xs = conv_sm;                 // [channel][plane mod TZ][row][x]
    float* ws = conv_sm + C::XN;         // [tap of the plane][channel][output]
    const int tid = threadIdx.x;
    const int j = tid % (TX / 8), ty = tid / (TX / 8) % CONV_TY, tz = tid / (TX / 8 * CONV_TY) % TZ;
    const int o0 = tid / (TX / 8 * CONV_TY * TZ) * COT;
    const int ntx = (d.nx + TX - 1) / TX, nty = (d.ny + CONV_TY - 1) / CONV_TY, ntz = (d.nz + TZ - 1) / TZ;
    int t = blockIdx.x;
    const int x0 = t % ntx * TX;
    t /= ntx;
    const int y0 = t % nty * CONV_TY;
    t /= nty;
    const int z0 = t % ntz * TZ, b = t / ntz;
    float acc[8][COT];
#pragma unroll
    for (int o = 0; o < COT; ++o) {
        const float v = __ldg(bias + o0 + o);
#pragma unroll
        for (int i = 0; i < 8; ++i) acc[i][o] = v;
    }
    // np planes of the padded tile from plane p0 on
    auto stage = [&](auto NP, int p0) {
        constexpr int cells = decltype(NP)::value * RX * RY;
#pragma unroll 4
        for (int e = tid; e < cells * (CI / 4); e += C::THREADS) {
            const int q = e / cells, cell = e - q * cells, rx = cell % RX, r = cell / RX, ry = r % RY, p = p0 + r / RY;
            const bool in = x0 + rx < d.nx + 2 && y0 + ry < d.ny + 2 && z0 + p < d.nz + 2;   // the padded tensor
            float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
            if (in) v = __ldg(reinterpret_cast<const float4*>(X + d.pos(b, x0 + rx - 1, y0 + ry - 1, z0 + p - 1) * CI) + q);
            float* dst = xs + (4 * q * TZ + p % TZ) * C::PLANE + ry * PX + rx;
            dst[0] = v.x;
            dst[TZ * C::PLANE] = v.y;
            dst[2 * TZ * C::PLANE] = v.z;
            dst[3 * TZ * C::PLANE] = v.w;
        }
    };
    for (int dz = 0; dz < 3; ++dz) {
        // planes dz .. dz + TZ - 1; all but the last are there from the dz before
        if (dz) {
            __syncthreads();
            stage(std::integral_constant<int, 1>(), dz + TZ - 1);
        } else {
            stage(std::integral_constant<int, TZ>(), 0);
        }
        for (int e = tid; e < C::WN; e += C::THREADS) {
            const int o = e % CO, r = e / CO, c = r % CI, tap = r / CI;
            ws[e] = __ldg(W + ((9 * dz + tap) * CO + o) * CI + c);
        }
        __syncthreads();
        const float* xp = xs + (tz + dz) % TZ * C::PLANE + ty * PX + 8 * j;
        const float* wr = ws + o0;
#pragma unroll 1
        for (int dy = 0; dy < 3; ++dy) {
            // the 8 + 2 values of a channel's row; of a few channels they stay in registers for the three taps
            float xv[ROWS][10];
            auto row = [&](int k, const float* xr) {
                *reinterpret_cast<float4*>(xv[k]) = *reinterpret_cast<const float4*>(xr);
                *reinterpret_cast<float4*>(xv[k] + 4) = *reinterpret_cast<const float4*>(xr + 4);
                *reinterpret_cast<float2*>(xv[k] + 8) = *reinterpret_cast<const float2*>(xr + 8);
            };
            if (ROWS == CI) {
#pragma unroll
                for (int c = 0; c < ROWS; ++c) row(c, xp + dy * PX + c * TZ * C::PLANE);
            }
            auto tap = [&](auto DX) {
                constexpr int dx = decltype(DX)::value;
                const float* xr = xp + dy * PX;
#pragma unroll C::UNROLL
                for (int c = 0; c < CI; ++c) {
                    const int k = ROWS == CI ? c : 0;
                    if (ROWS != CI) {   // the tap's 8 alone
                        if (dx == 2) *reinterpret_cast<float2*>(xv[k] + 2) = *reinterpret_cast<const float2*>(xr + 2);
                        else *reinterpret_cast<float4*>(xv[k]) = *reinterpret_cast<const float4*>(xr);
                        *reinterpret_cast<float4*>(xv[k] + 4) = *reinterpret_cast<const float4*>(xr + 4);
                        if (dx == 1) xv[k][8] = xr[8];
                        if (dx == 2) *reinterpret_cast<float2*>(xv[k] + 8) = *reinterpret_cast<const float2*>(xr + 8);
                        xr += TZ * C::PLANE;
                    }
                    float wv[COT];
                    if (COT == 8) {
                        *reinterpret_cast<float4*>(wv) = *reinterpret_cast<const float4*>(wr + c * CO);
                        *reinterpret_cast<float4*>(wv + 4) = *reinterpret_cast<const float4*>(wr + c * CO + 4);
                    } else {
#pragma unroll
                        for (int o = 0; o < COT; ++o) wv[o] = wr[c * CO + o];
                    }
#pragma unroll
                    for (int i = 0; i < 8; ++i)
#pragma unroll
                        for (int o = 0; o < COT; ++o) acc[i][o] = fmaf(wv[o], xv[k][i + dx], acc[i][o]);
                }
                wr += CI * CO;
            };
            tap(std::integral_constant<int, 0>());
            tap(std::integral_constant<int, 1>());
            tap(std::integral_constant<int, 2>());
        }
    }
    const int y = y0 + ty, z = z0 + tz;
    if (y >= d.ny || z >= d.nz) return;
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        const int x = x0 + 8 * j + i;
        if (x >= d.nx) break;
        const long long q = d.pos(b, x, y, z) * CO + o0;
        float v[COT];
#pragma unroll
        for (int o = 0; o < COT; ++o) {
            v[o] = relu ? fmaxf(acc[i][o], 0.f) : acc[i][o];
            if (skip) v[o] += __ldg(skip + q + o);
        }
        if (COT == 8) {
#pragma unroll
            for (int h = 0; h < 8; h += 4) {
                if (Z) *reinterpret_cast<float4*>(Z + q + h) = make_float4(acc[i][h], acc[i][h + 1], acc[i][h + 2], acc[i][h + 3]);
                *reinterpret_cast<float4*>(A + q + h) = make_float4(v[h], v[h + 1], v[h + 2], v[h + 3]);
            }
        } else {
#pragma unroll
            for (int o = 0; o < COT; ++o) {
                if (Z) Z[q + o] = acc[i][o];
                A[q + o] = v[o];
            }
        }
    }
}

// ------------------------------------------------------------------ weight gradient
// dW[t][o][c] = Σ_p X[p + off(t)][c] dY[p][o], db[o] = Σ_p dY[p][o].  A thread owns 4 input x 4 output channels of
// the three taps of one (dy, dz) row and slides along x: each cell costs it one vector of X (the other two taps'
// are the previous cells') and one of dY for 48 multiply-adds.  A block keeps its sums over all its tiles and
// writes them once; the partial sums of the blocks are added in a fixed order (wgrad_sum_k).
constexpr int WG_X = 16, WG_Y = 4, WG_Z = 2;
constexpr int WG_BLOCKS = 2;   // blocks per multiprocessor that the tiles are dealt to
template <int CI, int CO>
struct Wgrad {
    static constexpr int CQ = CI / 4, OV = CO < 4 ? CO : 4, OQ = CO / OV, R = 9 * CQ * OQ;
    static constexpr int G = R >= 288 ? 1 : 288 / R;              // groups of threads, each with its rows of the tile
    static constexpr int THREADS = R * G;
    static constexpr int XC = (WG_X + 2) * (WG_Y + 2) * (WG_Z + 2), YC = WG_X * WG_Y * WG_Z;
    static constexpr int TILE = XC * CI + YC * CO;                // floats
    static constexpr int N = 27 * CI * CO + CO;                   // gradients of the layer
    static constexpr int SM = G > 1 && G * N > TILE ? G * N : TILE;
};

template <int CI, int CO>
__global__ void __launch_bounds__(Wgrad<CI, CO>::THREADS) wgrad_k(Dims d, const float* __restrict__ X,
                                                                  const float* __restrict__ dY, float* __restrict__ part,
                                                                  int ntiles) {
    using G = Wgrad<CI, CO>;
    constexpr int OV = G::OV;
    static_assert((WG_Y * WG_Z) % G::G == 0, "rows of a tile");
    extern __shared__ __align__(16) float wg_sm[];
    float* xs = wg_sm;
    float* ys = wg_sm + G::XC * CI;
    const int tid = threadIdx.x, grp = tid / G::R, role = tid % G::R;
    const int cq = role % G::CQ, oq = role / G::CQ % G::OQ, row = role / (G::CQ * G::OQ);   // row = (dz+1)*3 + dy+1
    const int ntx = (d.nx + WG_X - 1) / WG_X, nty = (d.ny + WG_Y - 1) / WG_Y, ntz = (d.nz + WG_Z - 1) / WG_Z;
    float acc[3][4][OV], bacc[OV];
#pragma unroll
    for (int k = 0; k < 3; ++k)
#pragma unroll
        for (int c = 0; c < 4; ++c)
#pragma unroll
            for (int o = 0; o < OV; ++o) acc[k][c][o] = 0.f;
#pragma unroll
    for (int o = 0; o < OV; ++o) bacc[o] = 0.f;
    const bool bias_role = row == 4 && cq == 0;
    for (int tile = blockIdx.x; tile < ntiles; tile += gridDim.x) {
        int t = tile;
        const int x0 = t % ntx * WG_X;
        t /= ntx;
        const int y0 = t % nty * WG_Y;
        t /= nty;
        const int z0 = t % ntz * WG_Z, b = t / ntz;
        __syncthreads();
        constexpr int RX = WG_X + 2, RY = WG_Y + 2;
        for (int e = tid; e < G::XC * (CI / 4); e += G::THREADS) {
            const int q = e % (CI / 4), cell = e / (CI / 4), rx = cell % RX, r = cell / RX, ry = r % RY, rz = r / RY;
            const bool in = x0 + rx < d.nx + 2 && y0 + ry < d.ny + 2 && z0 + rz < d.nz + 2;
            float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
            if (in) v = __ldg(reinterpret_cast<const float4*>(X + d.pos(b, x0 + rx - 1, y0 + ry - 1, z0 + rz - 1) * CI) + q);
            reinterpret_cast<float4*>(xs)[e] = v;
        }
        // cells past the grid have no gradient
        for (int e = tid; e < G::YC * CO; e += G::THREADS) {
            const int o = e % CO, cell = e / CO, x = x0 + cell % WG_X, r = cell / WG_X, y = y0 + r % WG_Y, z = z0 + r / WG_Y;
            ys[e] = x < d.nx && y < d.ny && z < d.nz ? __ldg(dY + d.pos(b, x, y, z) * CO + o) : 0.f;
        }
        __syncthreads();
#pragma unroll 1
        for (int rr = grp; rr < WG_Y * WG_Z; rr += G::G) {
            const int y = rr % WG_Y, z = rr / WG_Y;
            const float4* xr = reinterpret_cast<const float4*>(xs + ((z + row / 3) * RY + y + row % 3) * RX * CI) + cq;
            const float* yr = ys + rr * WG_X * CO + oq * OV;
            float4 xw[3];
            xw[0] = xr[0];
            xw[1] = xr[CI / 4];
#pragma unroll
            for (int x = 0; x < WG_X; ++x) {
                xw[(x + 2) % 3] = xr[(x + 2) * (CI / 4)];
                float g[OV];
                if (OV == 4) *reinterpret_cast<float4*>(g) = *reinterpret_cast<const float4*>(yr + x * CO);
                else g[0] = yr[x * CO];
#pragma unroll
                for (int k = 0; k < 3; ++k) {
                    const float4 f = xw[(x + k) % 3];
#pragma unroll
                    for (int o = 0; o < OV; ++o) {
                        acc[k][0][o] = fmaf(f.x, g[o], acc[k][0][o]);
                        acc[k][1][o] = fmaf(f.y, g[o], acc[k][1][o]);
                        acc[k][2][o] = fmaf(f.z, g[o], acc[k][2][o]);
                        acc[k][3][o] = fmaf(f.w, g[o], acc[k][3][o]);
                    }
                }
                if (bias_role) {
#pragma unroll
                    for (int o = 0; o < OV; ++o) bacc[o] += g[o];
                }
            }
        }
    }
    // with several groups, their sums meet in shared memory
    float* out = part + (long long)blockIdx.x * G::N;
    float* dst = G::G > 1 ? wg_sm + grp * G::N : out;
    if (G::G > 1) __syncthreads();
#pragma unroll
    for (int k = 0; k < 3; ++k)
#pragma unroll
        for (int o = 0; o < OV; ++o)
#pragma unroll
            for (int c = 0; c < 4; ++c) dst[((row * 3 + k) * CO + oq * OV + o) * CI + 4 * cq + c] = acc[k][c][o];
    if (bias_role) {
#pragma unroll
        for (int o = 0; o < OV; ++o) dst[27 * CI * CO + oq * OV + o] = bacc[o];
    }
    if (G::G > 1) {
        __syncthreads();
        for (int e = tid; e < G::N; e += G::THREADS) {
            float s = 0.f;
#pragma unroll
            for (int g = 0; g < G::G; ++g) s += wg_sm[g * G::N + e];
            out[e] = s;
        }
    }
}

// g[i] = Σ over `blocks` partial gradients of n values each: 32 values and 8 strands a block, in a fixed order
__global__ void __launch_bounds__(256) wgrad_sum_k(const float* __restrict__ part, int blocks, int n, float* __restrict__ g) {
    __shared__ double sm[8][32];
    const int i = blockIdx.x * 32 + (threadIdx.x & 31), s = threadIdx.x >> 5;
    double a = 0.0;
    if (i < n) {
#pragma unroll 4
        for (int b = s; b < blocks; b += 8) a += double(__ldg(part + (long long)b * n + i));
    }
    sm[s][threadIdx.x & 31] = a;
    __syncthreads();
    if (s == 0 && i < n) {
        for (int k = 1; k < 8; ++k) a += sm[k][threadIdx.x];
        g[i] = float(a);
    }
}

// ------------------------------------------------------------------ passes between the layers
// One thread takes four channels of a cell (C a multiple of 4, a power of two of vectors), so that a warp reads
// and writes whole 128-byte lines; a thread per cell touched 16 to 32 lines a load.  The ReLU factor is applied
// where the gradient that it masks is formed.
#define FOR_VECS(D, C4)                                                                                             \
    for (long long e_ = blockIdx.x * (long long)blockDim.x + threadIdx.x; e_ < (D).cells() * (C4);                  \
         e_ += (long long)gridDim.x * blockDim.x)
__device__ __forceinline__ void decode32(const Dims& d, unsigned q, int& b, int& x, int& y, int& z) {
    x = int(q % unsigned(d.nx));
    q /= unsigned(d.nx);
    y = int(q % unsigned(d.ny));
    q /= unsigned(d.ny);
    z = int(q % unsigned(d.nz));
    b = int(q / unsigned(d.nz));
}
__device__ __forceinline__ float4 add4(float4 a, float4 b) { return make_float4(a.x + b.x, a.y + b.y, a.z + b.z, a.w + b.w); }
__device__ __forceinline__ float4 mask4(float4 z, float4 v) {
    return make_float4(z.x > 0.f ? v.x : 0.f, z.y > 0.f ? v.y : 0.f, z.z > 0.f ? v.z : 0.f, z.w > 0.f ? v.w : 0.f);
}

// dZ = dA · [Z > 0]
__global__ void relu_bwd_k(Dims d, int C4, const float4* __restrict__ Z, const float4* __restrict__ dA, float4* __restrict__ dZ) {
    FOR_VECS(d, C4) {
        int b, x, y, z;
        decode32(d, unsigned(e_ / C4), b, x, y, z);
        const long long p = d.pos(b, x, y, z) * C4 + e_ % C4;
        dZ[p] = mask4(Z[p], dA[p]);
    }
}
// out (coarse dims dc) = mean of the 8 children of in
__global__ void pool_fwd_k(Dims dc, int C4, const float4* __restrict__ in, float4* __restrict__ out) {
    const Dims df{dc.B, 2 * dc.nx, 2 * dc.ny, 2 * dc.nz};
    FOR_VECS(dc, C4) {
        int b, x, y, z;
        decode32(dc, unsigned(e_ / C4), b, x, y, z);
        float4 s = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
        for (int k = 0; k < 8; ++k) s = add4(s, in[child_pos(df, b, x, y, z, k) * C4 + e_ % C4]);
        out[dc.pos(b, x, y, z) * C4 + e_ % C4] = make_float4(s.x * 0.125f, s.y * 0.125f, s.z * 0.125f, s.w * 0.125f);
    }
}
// dZ = [Z > 0] (dskip + dout[parent] / 8): a skip connection's gradient plus the pooling's (fine dims df)
__global__ void pool_bwd_relu_k(Dims df, int C4, const float4* __restrict__ dskip, const float4* __restrict__ dout,
                                const float4* __restrict__ Z, float4* __restrict__ dZ) {
    const Dims dc = df.half();
    FOR_VECS(df, C4) {
        int b, x, y, z;
        decode32(df, unsigned(e_ / C4), b, x, y, z);
        const long long p = df.pos(b, x, y, z) * C4 + e_ % C4;
        const float4 s = dskip[p], o = dout[dc.pos(b, x / 2, y / 2, z / 2) * C4 + e_ % C4];
        dZ[p] = mask4(Z[p], make_float4(s.x + 0.125f * o.x, s.y + 0.125f * o.y, s.z + 0.125f * o.z, s.w + 0.125f * o.w));
    }
}
// out[child] = in[parent] (+ skip[child])  (fine dims df)
__global__ void up_fwd_k(Dims df, int C4, const float4* __restrict__ in, const float4* __restrict__ skip, float4* __restrict__ out) {
    const Dims dc = df.half();
    FOR_VECS(df, C4) {
        int b, x, y, z;
        decode32(df, unsigned(e_ / C4), b, x, y, z);
        const long long p = df.pos(b, x, y, z) * C4 + e_ % C4;
        const float4 v = in[dc.pos(b, x / 2, y / 2, z / 2) * C4 + e_ % C4];
        out[p] = skip ? add4(v, skip[p]) : v;
    }
}
// dZ[parent] = [Z > 0] Σ children dout  (coarse dims dc)
__global__ void up_bwd_relu_k(Dims dc, int C4, const float4* __restrict__ dout, const float4* __restrict__ Z, float4* __restrict__ dZ) {
    const Dims df{dc.B, 2 * dc.nx, 2 * dc.ny, 2 * dc.nz};
    FOR_VECS(dc, C4) {
        int b, x, y, z;
        decode32(dc, unsigned(e_ / C4), b, x, y, z);
        float4 s = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
        for (int k = 0; k < 8; ++k) s = add4(s, dout[child_pos(df, b, x, y, z, k) * C4 + e_ % C4]);
        const long long P = dc.pos(b, x, y, z) * C4 + e_ % C4;
        dZ[P] = mask4(Z[P], s);
    }
}

}  // namespace nn
}  // namespace ia
