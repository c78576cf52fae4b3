// 'uvw' tensor product whose weights belong to the item (an edge network made them), any multiplicities, in2 multiplicity 1.
//
//   T_p[u, k]  = sum_ij C_p[i, j, k] x[u, i] y[j]           (Clebsch-Gordan stage)
//   z[w, k]   += sum_u W_p[u, w] T_p[u, k]
//   G_p[u, k]  = sum_w W_p[u, w] g[w, k]         dW_p[u, w] = sum_k T_p[u, k] g[w, k]
//   dx, dy     = C_p folded with G_p and y, x
//
// Every weight is read once (and its gradient written once) and enters 2 D3 or 4 D3 operations, so the weight rows bound
// the kernel: the rest of an item is a few hundred floats.  A block of four warps takes one item: its operands, all T_p and
// all G_p lie in shared memory, and the weight row is walked by 16-byte accesses that are contiguous over the block.  A lane
// group of PP lanes holds one row u of a 32-wide weight tile; the columns that a lane holds are the same for every row, so
// the cotangent (or the sum) of those columns stays in registers and the sum over w is log2(PP) shuffles per row of VEC * P.
// All sums run in an order fixed by the problem: bitwise reproducible.
//
// DiffDock L = 2 (multiplicities 10 and 48, 7,128 weights), 8,191 items: forward 65 us (3.8 TB/s of rows), backward 122 us (4.1 TB/s;
// 195 us with five blocks of 127 registers to an SM and no staged row, 147 us with eight of 64 registers and none; with the row, 28 KB, and the
// static arrays, 7 KB, six blocks fit an SM's shared memory); the general kernels (a warp per item, strided stores of dW, a shuffle per
// product) took 733 us for both.  Narrow products do not earn the block's barriers back: the host decides (item_forward_pays, item_backward_pays).
#pragma once

// ITEM_VEC (emitted): the largest power of two up to 16 bytes that divides the row length and every weight offset.
constexpr int ITEM_WARPS = 4;

template <int N> struct ItemOff {   // T of instruction n, and of its G per 32-wide column tile
    static constexpr int T0 = ItemOff<N - 1>::T0 + Ins<N - 1>::U * Ins<N - 1>::D3;
    static constexpr int G0 = ItemOff<N - 1>::G0 + Ins<N - 1>::U * Ins<N - 1>::D3 * ((Ins<N - 1>::WN_ + 31) / 32);
};
template <> struct ItemOff<0> { static constexpr int T0 = 0, G0 = 0; };
template <int A> struct ItemChunk { static constexpr int BEG = ItemChunk<A - 1>::BEG + (Blk1<A - 1>::MUL + 31) / 32; };
template <> struct ItemChunk<0> { static constexpr int BEG = 0; };

constexpr int item_vec(int wlen) {
    int v = ITEM_VEC;
    while (wlen % v) v >>= 1;
    return v;
}
constexpr int item_pow2(int n) {
    int p = 1;
    while (p < n) p <<= 1;
    return p;
}

// Columns [32 WC, 32 WC + WLEN) of an output block of W channels: how a warp's lanes lie on a row-major [rows][WLEN] tile.
template <int W, int WC> struct ItemCols {
    static constexpr int WLEN = (W - 32 * WC) < 32 ? (W - 32 * WC) : 32;
    static constexpr int VEC = item_vec(WLEN), P = WLEN / VEC, PP = item_pow2(P), ROWS = 32 / PP;
};

template <int VEC> struct alignas(VEC * sizeof(T)) ItemVec { T v[VEC]; };

// f(row of the instruction, offset in the item's weight row) for this thread's part of the rows of (In, WC); the sum over
// the lanes of a row needs all lanes, so rows past the end call f(-1, 0).
template <class In, int WC, class F>
OEQ_DEV void item_rows(int warp, int lane, F&& f) {
    using C = ItemCols<In::WN_, WC>;
    const int r = lane / C::PP, c = lane % C::PP;
    static_for<0, (In::U + 31) / 32>([&](auto uc) {
        constexpr int UC = decltype(uc)::value, ULEN = (In::U - 32 * UC) < 32 ? (In::U - 32 * UC) : 32;
        constexpr int BASE = In::WOFF + 32 * UC * In::WN_ + ULEN * 32 * WC;
        constexpr int STEPS = (ULEN + ITEM_WARPS * C::ROWS - 1) / (ITEM_WARPS * C::ROWS);
#pragma unroll
        for (int s = 0; s < STEPS; ++s) {
            const int ul = (s * ITEM_WARPS + warp) * C::ROWS + r;
            const bool on = c < C::P && ul < ULEN;
            f(on ? 32 * UC + ul : -1, on ? BASE + ul * C::WLEN + c * C::VEC : 0);
        }
    });
}

// The item's weight row, requested whole by asynchronous copies before anything else is read (ITEM_STAGE_W, emitted: rows up
// to 40 KB); longer rows are read from global memory where they are used.  The backward
// gained (147 -> 122 us, DiffDock L = 2, 8,191 items); the forward, whose loads are already far ahead of their use, lost (65 -> 72 us) and
// reads global memory.
OEQ_DEV void item_request(const T* src, T* dst) {
#if ITEM_STAGE_W
    constexpr int BYTES = ITEM_VEC * (int)sizeof(T);
    const unsigned to = (unsigned)__cvta_generic_to_shared(dst);
    for (int i = threadIdx.x; i < WN / ITEM_VEC; i += ITEM_WARPS * 32)
        asm volatile("cp.async.ca.shared.global [%0], [%1], %2;" ::"r"(to + i * BYTES), "l"(src + (long long)i * ITEM_VEC), "n"(BYTES) : "memory");
#endif
}
OEQ_DEV void item_arrived() {
#if ITEM_STAGE_W
    asm volatile("cp.async.wait_all;" ::: "memory");
#endif
}

OEQ_DEV void item_stage(const T* __restrict__ src, T* dst, int n) {
    for (int i = threadIdx.x; i < n; i += ITEM_WARPS * 32) dst[i] = src[i];
}

// T of every instruction, the instructions dealt to the warps
OEQ_DEV void item_cg(const T* xs, const T* ys, T* ts, int warp, int lane) {
    static_for<0, NINS>([&](auto ic) {
        constexpr int N = decltype(ic)::value;
        using In = Ins<N>;
        if (N % ITEM_WARPS == warp) {
            for (int u = lane; u < In::U; u += 32) {
                T t[In::D3];
#pragma unroll
                for (int k = 0; k < In::D3; ++k) t[k] = T(0);
                In::fwd(xs + Blk1<In::A>::OFF + u * In::D1, ys + Blk2<In::B>::OFF, t);
#pragma unroll
                for (int k = 0; k < In::D3; ++k) ts[ItemOff<N>::T0 + u * In::D3 + k] = t[k];
            }
        }
    });
}

struct ItemFwdParams {
    const T* x; const T* y; const T* W; T* z;
    long long items;
    int add;
};

extern "C" __global__ void __launch_bounds__(ITEM_WARPS * 32) oeq_uvw_item_forward(const ItemFwdParams p) {
    __shared__ T xs[L1_DIM], ys[L2_DIM], ts[ItemOff<NINS>::T0], zs[ITEM_WARPS][L3_DIM];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    for (long long b = blockIdx.x; b < p.items; b += gridDim.x) {
        item_stage(p.x + b * L1_DIM, xs, L1_DIM);
        item_stage(p.y + b * L2_DIM, ys, L2_DIM);
        __syncthreads();
        item_cg(xs, ys, ts, warp, lane);
        __syncthreads();
        const T* __restrict__ wrow = p.W + b * WN;
        static_for<0, NB3>([&](auto oc) {
            constexpr int O = decltype(oc)::value;
            using B3 = Blk3<O>;
            static_for<0, (B3::MUL + 31) / 32>([&](auto wc) {
                constexpr int WC = decltype(wc)::value;
                using C = ItemCols<B3::MUL, WC>;
                T acc[C::VEC][B3::D];
#pragma unroll
                for (int v = 0; v < C::VEC; ++v)
#pragma unroll
                    for (int k = 0; k < B3::D; ++k) acc[v][k] = T(0);
                static_for<0, NINS>([&](auto ic) {
                    constexpr int N = decltype(ic)::value;
                    using In = Ins<N>;
                    if constexpr (In::O == O) {
                        item_rows<In, WC>(warp, lane, [&](int u, int wi) {
                            if (u >= 0) {
                                const ItemVec<C::VEC> w = *reinterpret_cast<const ItemVec<C::VEC>*>(wrow + wi);
#pragma unroll
                                for (int k = 0; k < B3::D; ++k) {
                                    const T t = ts[ItemOff<N>::T0 + u * B3::D + k];
#pragma unroll
                                    for (int v = 0; v < C::VEC; ++v) acc[v][k] += w.v[v] * t;
                                }
                            }
                        });
                    }
                });
#pragma unroll
                for (int v = 0; v < C::VEC; ++v)
#pragma unroll
                    for (int k = 0; k < B3::D; ++k) {
#pragma unroll
                        for (int s = C::PP; s < 32; s <<= 1) acc[v][k] += __shfl_xor_sync(0xffffffffu, acc[v][k], s);
                        if (lane < C::P) zs[warp][B3::OFF + (32 * WC + lane * C::VEC + v) * B3::D + k] = acc[v][k];
                    }
            });
        });
        __syncthreads();
        T* zrow = p.z + b * L3_DIM;
        for (int i = threadIdx.x; i < L3_DIM; i += ITEM_WARPS * 32) {
            T s = zs[0][i];
#pragma unroll
            for (int q = 1; q < ITEM_WARPS; ++q) s += zs[q][i];
            zrow[i] = p.add ? zrow[i] + s : s;
        }
        // the next item overwrites xs, ys and ts, last read before the barrier above, and zs only after two more
    }
}

struct ItemBwdParams {
    const T* x; const T* y_dx; const T* y_dw; const T* W; const T* g;
    T* dx; T* dy; T* dW;
    long long items;
    int add;
};

extern "C" __global__ void __launch_bounds__(ITEM_WARPS * 32, sizeof(T) == 4 ? 8 : 4) oeq_uvw_item_backward(const ItemBwdParams p) {
    __shared__ T xs[L1_DIM], y1[L2_DIM], y2[L2_DIM], gs[L3_DIM], ts[ItemOff<NINS>::T0], gp[ItemOff<NINS>::G0], dys[ITEM_WARPS][L2_DIM];
    extern __shared__ __align__(16) unsigned char item_row[];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    for (long long b = blockIdx.x; b < p.items; b += gridDim.x) {
        item_request(p.W + b * WN, (T*)item_row);
        item_stage(p.x + b * L1_DIM, xs, L1_DIM);
        item_stage(p.y_dx + b * L2_DIM, y1, L2_DIM);
        item_stage(p.y_dw + b * L2_DIM, y2, L2_DIM);
        item_stage(p.g + b * L3_DIM, gs, L3_DIM);
        __syncthreads();
        item_cg(xs, y2, ts, warp, lane);
        item_arrived();
        __syncthreads();
        const T* __restrict__ wrow = ITEM_STAGE_W ? (const T*)item_row : p.W + b * WN;
        T* __restrict__ dwrow = p.dW + b * WN;
        static_for<0, NB3>([&](auto oc) {
            constexpr int O = decltype(oc)::value;
            using B3 = Blk3<O>;
            static_for<0, (B3::MUL + 31) / 32>([&](auto wc) {
                constexpr int WC = decltype(wc)::value;
                using C = ItemCols<B3::MUL, WC>;
                const int c = lane % C::PP;
                T g[C::VEC][B3::D];
#pragma unroll
                for (int v = 0; v < C::VEC; ++v)
#pragma unroll
                    for (int k = 0; k < B3::D; ++k) g[v][k] = c < C::P ? gs[B3::OFF + (32 * WC + c * C::VEC + v) * B3::D + k] : T(0);
                static_for<0, NINS>([&](auto ic) {
                    constexpr int N = decltype(ic)::value;
                    using In = Ins<N>;
                    if constexpr (In::O == O) {
                        item_rows<In, WC>(warp, lane, [&](int u, int wi) {
                            T s[B3::D];
#pragma unroll
                            for (int k = 0; k < B3::D; ++k) s[k] = T(0);
                            if (u >= 0) {
                                const ItemVec<C::VEC> w = *reinterpret_cast<const ItemVec<C::VEC>*>(wrow + wi);
                                ItemVec<C::VEC> d;
#pragma unroll
                                for (int v = 0; v < C::VEC; ++v) d.v[v] = T(0);
#pragma unroll
                                for (int k = 0; k < B3::D; ++k) {
                                    const T t = ts[ItemOff<N>::T0 + u * B3::D + k];
#pragma unroll
                                    for (int v = 0; v < C::VEC; ++v) {
                                        s[k] += w.v[v] * g[v][k];
                                        d.v[v] += t * g[v][k];
                                    }
                                }
                                ItemVec<C::VEC>* out = reinterpret_cast<ItemVec<C::VEC>*>(dwrow + wi);
                                if (p.add) {
                                    const ItemVec<C::VEC> was = *out;
#pragma unroll
                                    for (int v = 0; v < C::VEC; ++v) d.v[v] += was.v[v];
                                }
                                *out = d;
                            }
#pragma unroll
                            for (int k = 0; k < B3::D; ++k) {
#pragma unroll
                                for (int m = 1; m < C::PP; m <<= 1) s[k] += __shfl_xor_sync(0xffffffffu, s[k], m);
                                if (u >= 0 && c == 0) gp[ItemOff<N>::G0 + (WC * In::U + u) * B3::D + k] = s[k];
                            }
                        });
                    }
                });
            });
        });
        __syncthreads();
        T dyacc[L2_DIM];
#pragma unroll
        for (int j = 0; j < L2_DIM; ++j) dyacc[j] = T(0);
        static_for<0, NB1>([&](auto ac) {   // 32 channels of an input block at a time, dealt to the warps
            constexpr int A = decltype(ac)::value;
            using B1 = Blk1<A>;
            static_for<0, (B1::MUL + 31) / 32>([&](auto cc) {
                constexpr int CH = decltype(cc)::value;
                const int u = 32 * CH + lane;
                if ((ItemChunk<A>::BEG + CH) % ITEM_WARPS == warp && u < B1::MUL) {
                    T dxacc[B1::D], xv[B1::D];
#pragma unroll
                    for (int i = 0; i < B1::D; ++i) { dxacc[i] = T(0); xv[i] = xs[B1::OFF + u * B1::D + i]; }
                    static_for<0, NINS>([&](auto ic) {
                        constexpr int N = decltype(ic)::value;
                        using In = Ins<N>;
                        if constexpr (In::A == A) {
                            T gv[In::D3];
#pragma unroll
                            for (int k = 0; k < In::D3; ++k) {
                                gv[k] = T(0);
#pragma unroll
                                for (int wc = 0; wc < (In::WN_ + 31) / 32; ++wc) gv[k] += gp[ItemOff<N>::G0 + (wc * In::U + u) * In::D3 + k];
                            }
                            In::dx(y1 + Blk2<In::B>::OFF, gv, dxacc);
                            In::dy(xv, gv, dyacc + Blk2<In::B>::OFF);
                        }
                    });
                    T* dxrow = p.dx + b * L1_DIM + B1::OFF + u * B1::D;
#pragma unroll
                    for (int i = 0; i < B1::D; ++i) dxrow[i] = p.add ? dxrow[i] + dxacc[i] : dxacc[i];
                }
            });
        });
#pragma unroll
        for (int j = 0; j < L2_DIM; ++j) {
            const T s = warp_sum(dyacc[j]);
            if (lane == 0) dys[warp][j] = s;
        }
        __syncthreads();
        for (int j = threadIdx.x; j < L2_DIM; j += ITEM_WARPS * 32) {
            T s = dys[0][j];
#pragma unroll
            for (int q = 1; q < ITEM_WARPS; ++q) s += dys[q][j];
            T* out = p.dy + b * L2_DIM + j;
            *out = p.add ? *out + s : s;
        }
        // the next item overwrites the row and the operands, last read before the barrier above; dys only after three more barriers
    }
}
