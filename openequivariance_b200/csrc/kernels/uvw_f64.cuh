// 'uvw' tensor product in doubles with shared weights, multiplicities that are multiples of 32, on the FP64 matrix instruction
// (mma.sync.m8n8k4.f64: IEEE fused multiply-adds, so nothing is lost against the scalar kernels).
//
//   T_p[b][u, k]  = sum_ij C_p[i, j, k] x[b][u, i] y[b][j]
//   forward   z[b, o][w, k]  = sum_{p, u} T_p[b][u, k] W_p[u, w]              M = 8 items, N = w, K = u
//   backward  G_p[b][u, k]   = sum_w g[b, o][w, k] W_p[u, w]                  M = 8 items, N = u, K = w;  dx, dy fold G_p with C_p
//             dW_p[u, w]     = sum_{b, k} T_p[b][u, k] g[b, o][w, k]          M = u, N = w, K = items
//
// The FP64 pipe bounds these contractions (2 * 32 * 32 * D3 operations per path and item, and the Clebsch-Gordan terms), so all
// else is kept small: a lane computes the T that its own fragment of A needs in registers, weights and rows come through
// the L1 (a path's 32 x 32 weight tile is 8 KB and is read by every warp of the block), and a warp owns its outputs, so there is no
// shared memory, no barrier in the main loops and no conversion.  A warp takes eight items: sixteen would halve the weight reads but
// need 160 accumulator registers for five components.
//
// 30 paths of 32 x 32, l <= 2, 5,003 items: forward 58 us (18 TFLOP/s of contractions), dx and dy 113 us, dW 118 us; the general kernels
// took 225 us and 2,080 us (one item per warp: the weights were read again for every item).
#pragma once

// Fragments (lane = 4 g + t): A[row g][col t], B[row t][col g], C[row g][cols 2 t, 2 t + 1].
OEQ_DEV void f64_mma(double (&c)[2], double a, double b) {
    asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};" : "+d"(c[0]), "+d"(c[1]) : "d"(a), "d"(b));
}

// 32-wide tiles of the blocks, and the 32 x 32 weight tiles of the instructions, numbered in order
template <int O> struct F64Out { static constexpr int BEG = F64Out<O - 1>::BEG + Blk3<O - 1>::MUL / 32; };
template <> struct F64Out<0> { static constexpr int BEG = 0; };
template <int A> struct F64In { static constexpr int BEG = F64In<A - 1>::BEG + Blk1<A - 1>::MUL / 32; };
template <> struct F64In<0> { static constexpr int BEG = 0; };
template <int N> struct F64Sub { static constexpr int BEG = F64Sub<N - 1>::BEG + Ins<N - 1>::U / 32 * (Ins<N - 1>::WN_ / 32); };
template <> struct F64Sub<0> { static constexpr int BEG = 0; };
template <class In, int UC, int WC> struct F64Tile { static constexpr int W0 = In::WOFF + UC * 32 * In::WN_ + WC * 1024; };

constexpr int F64_WARPS = 4;

struct F64FwdParams {
    const double* __restrict__ x; const double* __restrict__ y; const double* __restrict__ W; double* __restrict__ z;
    long long batch;
    int accum;
};

// grid (32 items each, output tiles); a warp owns eight items of the tile.  The later blocks of a problem tend to have more
// components: they are started first.
extern "C" __global__ void __launch_bounds__(F64_WARPS * 32) oeq_uvw_f64_forward(const F64FwdParams p) {
    const int lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
    const long long item = (blockIdx.x * (long long)F64_WARPS + (threadIdx.x >> 5)) * 8 + g;
    const bool live = item < p.batch;
    const long long row = live ? item : p.batch - 1;   // (results of rows past the end are not stored)
    const double* xrow = p.x + row * L1_DIM;
    const double* yrow = p.y + row * L2_DIM;
    const int mine = gridDim.y - 1 - blockIdx.y;
    static_for<0, NB3>([&](auto oc) {
        constexpr int O = decltype(oc)::value;
        using B3 = Blk3<O>;
        static_for<0, B3::MUL / 32>([&](auto wc) {
            constexpr int WC = decltype(wc)::value;
            if (mine != F64Out<O>::BEG + WC) return;
            double acc[B3::D][4][2];
#pragma unroll
            for (int k = 0; k < B3::D; ++k)
#pragma unroll
                for (int n = 0; n < 4; ++n) acc[k][n][0] = acc[k][n][1] = 0.0;
            static_for<0, NINS>([&](auto ic) {
                using In = Ins<decltype(ic)::value>;
                if constexpr (In::O == O) {
                    double yv[In::D2];
#pragma unroll
                    for (int j = 0; j < In::D2; ++j) yv[j] = __ldg(yrow + Blk2<In::B>::OFF + j);
                    static_for<0, In::U / 32>([&](auto uc) {
                        constexpr int UC = decltype(uc)::value;
                        const double* w = p.W + F64Tile<In, UC, WC>::W0 + t * 32 + g;
                        const double* xb = xrow + Blk1<In::A>::OFF + (UC * 32 + t) * In::D1;
#pragma unroll 2
                        for (int kk = 0; kk < 8; ++kk) {
                            double xv[In::D1], tv[In::D3], b[4];
#pragma unroll
                            for (int i = 0; i < In::D1; ++i) xv[i] = __ldg(xb + kk * 4 * In::D1 + i);
#pragma unroll
                            for (int n = 0; n < 4; ++n) b[n] = __ldg(w + kk * 128 + 8 * n);
#pragma unroll
                            for (int k = 0; k < In::D3; ++k) tv[k] = 0.0;
                            In::fwd(xv, yv, tv);
#pragma unroll
                            for (int k = 0; k < In::D3; ++k)
#pragma unroll
                                for (int n = 0; n < 4; ++n) f64_mma(acc[k][n], tv[k], b[n]);
                        }
                    });
                }
            });
            if (live) {
                double* zb = p.z + item * L3_DIM + B3::OFF + (WC * 32 + 2 * t) * B3::D;
#pragma unroll
                for (int n = 0; n < 4; ++n)
#pragma unroll
                    for (int e = 0; e < 2; ++e)
#pragma unroll
                        for (int k = 0; k < B3::D; ++k) {
                            double* out = zb + (8 * n + e) * B3::D + k;
                            *out = p.accum ? *out + acc[k][n][e] : acc[k][n][e];
                        }
            }
        });
    });
}

struct F64BwdParams {
    const double* __restrict__ x; const double* __restrict__ y; const double* __restrict__ W; const double* __restrict__ g;
    double* __restrict__ dx; double* __restrict__ dy;
    long long batch;
    int accum;
};

// dx and dy.  A block takes eight items; its warps take half tiles (16 channels) of the input blocks in turn, so that dx is
// complete in registers, and their sums of dy are added in warp order.
extern "C" __global__ void __launch_bounds__(F64_WARPS * 32, 3) oeq_uvw_f64_backward(const F64BwdParams p) {
    __shared__ double dys[F64_WARPS][8][L2_DIM];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, g = lane >> 2, t = lane & 3;
    const long long item = blockIdx.x * 8LL + g;
    const bool live = item < p.batch;
    const long long row = live ? item : p.batch - 1;
    const double* xrow = p.x + row * L1_DIM;
    const double* yrow = p.y + row * L2_DIM;
    const double* grow = p.g + row * L3_DIM;
    double dyacc[L2_DIM];
#pragma unroll
    for (int j = 0; j < L2_DIM; ++j) dyacc[j] = 0.0;
    static_for<0, NB1>([&](auto ac) {
        constexpr int A = decltype(ac)::value;
        using B1 = Blk1<A>;
        static_for<0, B1::MUL / 32>([&](auto uc) {
            constexpr int UC = decltype(uc)::value;
            for (int h = 0; h < 2; ++h) {
                if ((2 * (F64In<A>::BEG + UC) + h) % F64_WARPS != warp) continue;
                const int u0 = UC * 32 + 16 * h + 2 * t;   // this lane's channels: u0 + 8 n + e
                double dxacc[2][2][B1::D];
#pragma unroll
                for (int q = 0; q < 4; ++q)
#pragma unroll
                    for (int i = 0; i < B1::D; ++i) dxacc[q >> 1][q & 1][i] = 0.0;
                static_for<0, NINS>([&](auto ic) {
                    using In = Ins<decltype(ic)::value>;
                    if constexpr (In::A == A) {
                        double acc[In::D3][2][2];
#pragma unroll
                        for (int k = 0; k < In::D3; ++k)
#pragma unroll
                            for (int q = 0; q < 4; ++q) acc[k][q >> 1][q & 1] = 0.0;
                        static_for<0, In::WN_ / 32>([&](auto wc) {
                            constexpr int WC = decltype(wc)::value;
                            const double* w = p.W + F64Tile<In, UC, WC>::W0 + (16 * h + g) * 32 + t;
                            const double* gb = grow + Blk3<In::O>::OFF + (WC * 32 + t) * In::D3;
#pragma unroll 2
                            for (int kk = 0; kk < 8; ++kk) {
                                const double b0 = __ldg(w + kk * 4), b1 = __ldg(w + 256 + kk * 4);
                                double a[In::D3];
#pragma unroll
                                for (int k = 0; k < In::D3; ++k) a[k] = __ldg(gb + kk * 4 * In::D3 + k);
#pragma unroll
                                for (int k = 0; k < In::D3; ++k) {
                                    f64_mma(acc[k][0], a[k], b0);
                                    f64_mma(acc[k][1], a[k], b1);
                                }
                            }
                        });
                        double yv[In::D2];
#pragma unroll
                        for (int j = 0; j < In::D2; ++j) yv[j] = __ldg(yrow + Blk2<In::B>::OFF + j);
#pragma unroll
                        for (int q = 0; q < 4; ++q) {
                            double gv[In::D3], xv[In::D1];
#pragma unroll
                            for (int k = 0; k < In::D3; ++k) gv[k] = acc[k][q >> 1][q & 1];
#pragma unroll
                            for (int i = 0; i < In::D1; ++i) xv[i] = __ldg(xrow + B1::OFF + (u0 + 8 * (q >> 1) + (q & 1)) * In::D1 + i);
                            In::dx(yv, gv, dxacc[q >> 1][q & 1]);
                            In::dy(xv, gv, dyacc + Blk2<In::B>::OFF);
                        }
                    }
                });
                if (live) {
#pragma unroll
                    for (int q = 0; q < 4; ++q) {
                        double* out = p.dx + item * L1_DIM + B1::OFF + (u0 + 8 * (q >> 1) + (q & 1)) * B1::D;
#pragma unroll
                        for (int i = 0; i < B1::D; ++i) out[i] = p.accum ? out[i] + dxacc[q >> 1][q & 1][i] : dxacc[q >> 1][q & 1][i];
                    }
                }
            }
        });
    });
#pragma unroll
    for (int j = 0; j < L2_DIM; ++j) {
        double s = dyacc[j];
        s += __shfl_xor_sync(0xffffffffu, s, 1);
        s += __shfl_xor_sync(0xffffffffu, s, 2);
        if (t == 0) dys[warp][g][j] = s;
    }
    __syncthreads();
    for (int q = threadIdx.x; q < 8 * L2_DIM; q += F64_WARPS * 32) {
        const long long b = blockIdx.x * 8LL + q / L2_DIM;
        if (b >= p.batch) break;
        double s = p.accum ? p.dy[b * L2_DIM + q % L2_DIM] : 0.0;
#pragma unroll
        for (int v = 0; v < F64_WARPS; ++v) s += dys[v][q / L2_DIM][q % L2_DIM];
        p.dy[b * L2_DIM + q % L2_DIM] = s;
    }
}

struct F64DwParams {
    const double* __restrict__ x; const double* __restrict__ y; const double* __restrict__ g; double* __restrict__ part;
    long long batch;
    int chunk;   // items per row of partial sums
};

// Partial sums of dW: grid (chunks of items, weight tiles / 4); a warp owns one 32 x 32 weight tile over a chunk of items.
// oeq_generic_dw_reduce adds the chunks' rows in order: bitwise reproducible.
extern "C" __global__ void __launch_bounds__(F64_WARPS * 32) oeq_uvw_f64_backward_dw(const F64DwParams p) {
    const int lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
    const int sub = blockIdx.y * F64_WARPS + (threadIdx.x >> 5);
    const long long b0 = blockIdx.x * (long long)p.chunk, b1 = b0 + p.chunk < p.batch ? b0 + p.chunk : p.batch;
    static_for<0, NINS>([&](auto ic) {
        constexpr int N = decltype(ic)::value;
        using In = Ins<N>;
        static_for<0, In::U / 32 * (In::WN_ / 32)>([&](auto sc) {
            constexpr int UC = decltype(sc)::value / (In::WN_ / 32), WC = decltype(sc)::value % (In::WN_ / 32);
            if (sub != F64Sub<N>::BEG + decltype(sc)::value) return;
            double acc[4][4][2];
#pragma unroll
            for (int q = 0; q < 16; ++q) acc[q >> 2][q & 3][0] = acc[q >> 2][q & 3][1] = 0.0;
            for (long long b = b0; b < b1; b += 4) {
                const bool live = b + t < b1;   // items past the end count as zero
                const long long row = live ? b + t : b;
                const double* xb = p.x + row * L1_DIM + Blk1<In::A>::OFF + (UC * 32 + g) * In::D1;
                const double* gb = p.g + row * L3_DIM + Blk3<In::O>::OFF + (WC * 32 + g) * In::D3;
                double yv[In::D2], tv[4][In::D3], gv[4][In::D3];
#pragma unroll
                for (int j = 0; j < In::D2; ++j) yv[j] = live ? __ldg(p.y + row * L2_DIM + Blk2<In::B>::OFF + j) : 0.0;
#pragma unroll
                for (int n = 0; n < 4; ++n)
#pragma unroll
                    for (int k = 0; k < In::D3; ++k) gv[n][k] = live ? __ldg(gb + 8 * n * In::D3 + k) : 0.0;
#pragma unroll
                for (int m = 0; m < 4; ++m) {
                    double xv[In::D1];
#pragma unroll
                    for (int i = 0; i < In::D1; ++i) xv[i] = live ? __ldg(xb + 8 * m * In::D1 + i) : 0.0;
#pragma unroll
                    for (int k = 0; k < In::D3; ++k) tv[m][k] = 0.0;
                    In::fwd(xv, yv, tv[m]);
                }
#pragma unroll
                for (int k = 0; k < In::D3; ++k)
#pragma unroll
                    for (int q = 0; q < 16; ++q) f64_mma(acc[q >> 2][q & 3], tv[q >> 2][k], gv[q & 3][k]);
            }
            double* out = p.part + blockIdx.x * (long long)WN + F64Tile<In, UC, WC>::W0 + g * 32 + 2 * t;
#pragma unroll
            for (int q = 0; q < 16; ++q) {
                out[(q >> 2) * 256 + 8 * (q & 3)] = acc[q >> 2][q & 3][0];
                out[(q >> 2) * 256 + 8 * (q & 3) + 1] = acc[q >> 2][q & 3][1];
            }
        });
    });
}
