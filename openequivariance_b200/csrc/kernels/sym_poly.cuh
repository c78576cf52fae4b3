// Symmetric contraction, the kernels that are specialised for one list of (component, monomial) terms (see
// csrc/sym_contraction.cuh).  The header emitted from the list defines T, ELL, NOUT, TERMS, QUADS, CHUNK (terms per chunk of
// the weight gradient), CHUNKS, and
//   sym_eval(x, c, P)            P[w]  = sum over the terms of w of c * monomial(x)
//   sym_grad(x, cot, c, dx)      dx[i] = sum over the terms of cot[w] * c * d monomial / d x_i
//   SymChunk<N>::add(x, cot, m)  m[q] += cot[w] * monomial(x) for the terms of chunk N
// as straight-line code over registers: with the index pattern in the instruction stream a term costs one or two fused
// multiply-adds; reading it from a list in shared memory cost about 36 instructions per four terms, and the two kernels took
// 80 and 212 us for 2,003 nodes, 128 channels, ell = 16 and 410 terms.
//
// forward / gradient_x: lane = node, warp = (tile of 32 nodes of one element, channel); the channel's coefficients are the same
// for the whole warp and come from shared memory, four per read.
// backward_c: lane = channel, warp = slice of an element's nodes; the sums of one chunk of terms stay in registers.  All warps of
// a block (and, by the order of the grid, of an SM) work on the same chunk: with a chunk per warp every warp ran through its
// own 2.4 KB of code and the kernel waited for instructions (113 us instead of 25).
#pragma once

struct SymParams {
    const int* group; long long n;         // (nodes of no element are listed as element G)
    int G, F, out_dim, slices;
    const T* x; const T* cot; const T* coef;
    T* out; T* dx; T* part;
    int out_col[NOUT], out_stride[NOUT];   // output component w of channel f is column out_col + f * out_stride
};

OEQ_DEV void sym_load(const T* __restrict__ src, T (&v)[ELL], bool live) {
    if (ELL % 4 == 0) {   // rows are multiples of 16 bytes of a 16-byte aligned tensor
        const T4* s4 = reinterpret_cast<const T4*>(src);
#pragma unroll
        for (int i = 0; i < ELL / 4; ++i) {
            T4 t = {T(0), T(0), T(0), T(0)};
            if (live) t = s4[i];
            v[4 * i] = t.x; v[4 * i + 1] = t.y; v[4 * i + 2] = t.z; v[4 * i + 3] = t.w;
        }
    } else {
#pragma unroll
        for (int i = 0; i < ELL; ++i) v[i] = live ? src[i] : T(0);
    }
}

// channels (warps) per block; the host launches as many
constexpr int SYM_WPB = 8 * QUADS * (int)sizeof(T4) <= 48000 ? 8 : 1;
// one piece of the element's coefficients per channel of the block: cs[warp][QUADS]
OEQ_DEV void sym_stage(T4* cs, const SymParams& p, int e, int f0) {
    constexpr int PIECES = (int)(sizeof(T4) / 16);
    const int have = (p.F - f0 < SYM_WPB ? p.F - f0 : SYM_WPB) * PIECES;
    const char* src = reinterpret_cast<const char*>(p.coef + ((long long)e * QUADS * p.F + f0) * 4);
    constexpr int per = SYM_WPB * PIECES;
    for (int i = threadIdx.x; i < QUADS * per; i += blockDim.x) {
        const int q = i / per, r = i % per;
        if (r < have) {
            const unsigned dst = (unsigned)__cvta_generic_to_shared(reinterpret_cast<char*>(cs + (r / PIECES) * QUADS + q) + (r % PIECES) * 16);
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src + (long long)q * p.F * (int)sizeof(T4) + r * 16) : "memory");
        }
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
}

extern "C" __global__ void __launch_bounds__(32 * SYM_WPB) oeq_sym_forward(const __grid_constant__ SymParams p) {
    __shared__ T4 cs[SYM_WPB * QUADS];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, f0 = blockIdx.y * SYM_WPB, f = f0 + warp;
    const int* off = p.group + p.n;
    const int* tl = off + p.G + 1;
    if ((int)blockIdx.x >= tl[0]) return;
    const int e = tl[1 + 2 * blockIdx.x], first = tl[2 + 2 * blockIdx.x];
    const bool live = first + lane < (e < p.G ? off[e + 1] : p.n) && f < p.F;
    const long long node = live ? p.group[first + lane] : 0;
    if (e == p.G) {
        if (live)
            for (int w = 0; w < NOUT; ++w) p.out[node * p.out_dim + p.out_col[w] + f * p.out_stride[w]] = T(0);
        return;
    }
    sym_stage(cs, p, e, f0);
    T x[ELL], P[NOUT];
    sym_load(p.x + (live ? (node * p.F + f) * ELL : 0), x, live);
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    __syncthreads();
    sym_eval(x, cs + warp * QUADS, P);
    if (live)
#pragma unroll
        for (int w = 0; w < NOUT; ++w) p.out[node * p.out_dim + p.out_col[w] + f * p.out_stride[w]] = P[w];
}

extern "C" __global__ void __launch_bounds__(32 * SYM_WPB) oeq_sym_backward_x(const __grid_constant__ SymParams p) {
    __shared__ T4 cs[SYM_WPB * QUADS];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, f0 = blockIdx.y * SYM_WPB, f = f0 + warp;
    const int* off = p.group + p.n;
    const int* tl = off + p.G + 1;
    if ((int)blockIdx.x >= tl[0]) return;
    const int e = tl[1 + 2 * blockIdx.x], first = tl[2 + 2 * blockIdx.x];
    const bool live = first + lane < (e < p.G ? off[e + 1] : p.n) && f < p.F;
    const long long node = live ? p.group[first + lane] : 0;
    if (e == p.G) {
        if (live)
            for (int i = 0; i < ELL; ++i) p.dx[(node * p.F + f) * ELL + i] = T(0);
        return;
    }
    sym_stage(cs, p, e, f0);
    T x[ELL], cot[NOUT], dx[ELL];
    sym_load(p.x + (live ? (node * p.F + f) * ELL : 0), x, live);
#pragma unroll
    for (int w = 0; w < NOUT; ++w) cot[w] = live ? p.cot[node * p.out_dim + p.out_col[w] + f * p.out_stride[w]] : T(0);
#pragma unroll
    for (int i = 0; i < ELL; ++i) dx[i] = T(0);
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    __syncthreads();
    sym_grad(x, cot, cs + warp * QUADS, dx);
    if (live) {
        T* row = p.dx + (node * p.F + f) * ELL;
        if (ELL % 4 == 0) {
#pragma unroll
            for (int i = 0; i < ELL / 4; ++i) reinterpret_cast<T4*>(row)[i] = T4{dx[4 * i], dx[4 * i + 1], dx[4 * i + 2], dx[4 * i + 3]};
        } else {
#pragma unroll
            for (int i = 0; i < ELL; ++i) row[i] = dx[i];
        }
    }
}

// part[slice][e][term][f]
template <int N>
OEQ_DEV void sym_chunk(const SymParams& p, int e, int f, int lo, int hi, T* dst) {
    T m[CHUNK];
#pragma unroll
    for (int q = 0; q < CHUNK; ++q) m[q] = T(0);
    const bool live = f < p.F;
    T x[ELL], cot[NOUT];
    auto id = [&](int pos) { return pos < hi ? p.group[pos] : 0; };
    auto fetch = [&](int pos, long long node) {
        const bool on = live && pos < hi;
        sym_load(p.x + (on ? (node * p.F + f) * ELL : 0), x, on);
#pragma unroll
        for (int w = 0; w < NOUT; ++w) cot[w] = on ? p.cot[node * p.out_dim + p.out_col[w] + f * p.out_stride[w]] : T(0);
    };
    fetch(lo, id(lo));
    int next = id(lo + 1);
    for (int pos = lo; pos < hi; ++pos) {
        T xc[ELL], cc[NOUT];
#pragma unroll
        for (int i = 0; i < ELL; ++i) xc[i] = x[i];
#pragma unroll
        for (int w = 0; w < NOUT; ++w) cc[w] = cot[w];
        fetch(pos + 1, next);                 // the next node's row is on its way while this one is used
        next = id(pos + 2);
        SymChunk<N>::add(xc, cc, m);
    }
    if (live)
#pragma unroll
        for (int q = 0; q < CHUNK; ++q)
            if (N * CHUNK + q < TERMS) dst[(long long)q * p.F] = m[q];
}

// grid = (units of four (element, channel block, slice) warps, chunks)
constexpr int SYM_GC_WARPS = 4;
extern "C" __global__ void __launch_bounds__(32 * SYM_GC_WARPS) oeq_sym_backward_c(const __grid_constant__ SymParams p) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int fblocks = (p.F + 31) / 32, unit = blockIdx.x * SYM_GC_WARPS + warp, chunk = blockIdx.y;
    if (unit >= p.G * fblocks * p.slices) return;
    const int e = unit / (fblocks * p.slices), slice = unit / fblocks % p.slices, f = unit % fblocks * 32 + lane;
    const int* off = p.group + p.n;
    const int lo0 = off[e], hi0 = off[e + 1];
    const int per = (hi0 - lo0 + p.slices - 1) / p.slices;
    const int lo = lo0 + slice * per < hi0 ? lo0 + slice * per : hi0, hi = lo + per < hi0 ? lo + per : hi0;
    T* dst = p.part + (((long long)slice * p.G + e) * TERMS + (long long)chunk * CHUNK) * p.F + f;
    static_for<0, CHUNKS>([&](auto nc) {
        if (chunk == decltype(nc)::value) sym_chunk<decltype(nc)::value>(p, e, f, lo, hi, dst);
    });
}
