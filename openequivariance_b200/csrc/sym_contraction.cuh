// Symmetric contraction (the node-wise product basis that follows the convolution in MACE) in one pass over the nodes: the
// parts that do not depend on the contraction's tensors.
//
// For node n of element e and feature channel f every output component w is a polynomial of degree <= 3 in the node's
// ell features x[n, f, :].  Its coefficients c[e, f, t] are the generalised Clebsch-Gordan tensors U applied to the
// element's weights; only the (component, monomial) terms that U touches are kept (410 for 0e + 1o at ell = 16 out of 4 x 968).
//
//   compare     : whether the tensors U are still the ones that the list of terms was made from
//   group_nodes : nodes by element, in node order (the order of every sum over nodes), and the list of 32-node tiles
//   coefficients: c[e, t, f] = sum_k U[t, k] W[e, k, f]
//   (kernels/sym_poly.cuh, specialised for the list of terms: the polynomials, their gradient, and for every term the sum over
//    an element's nodes of cot * monomial)
//   gradient_w  : dW[e, k, f] = sum_t U[t, k] * (the term's sums over slices of the nodes, in order)
//
// The composed form (one gather, one product and one reduction over [N, F, ell^2] tensors per order, through torch) moved
// about 10 GB for 2,000 nodes, 128 channels and ell = 16, where inputs and outputs are 42 MB.
#pragma once

#include <cuda_runtime.h>
#include <cstdint>

namespace symc {

constexpr int MAX_SETS = 48;       // (output irrep, order) pairs
constexpr int MAX_OUT = 64;        // output components over all irreps
constexpr int MAX_ELL = 25;
constexpr int MAX_TERMS = 1024;
constexpr int TILE = 32;           // nodes per warp
constexpr int STATUS_CHANGED = 42; // code stored in the status word when a captured call meets other tensors U than it was made for

struct Sets {
    int n_sets, F, terms;
    int k[MAX_SETS];               // columns of U in a set
    int t0[MAX_SETS], t1[MAX_SETS];   // rows of U that belong to a set
    int u[MAX_SETS];               // where a set's rows start in U
    int z0[MAX_SETS + 1];          // coefficients / gradient_w: first block of the set along one grid axis
    const int* place;              // row of U -> position of its term in the order in which the polynomials use them
};
struct Pointers { void* p[MAX_SETS]; };

__device__ __forceinline__ int set_of(const Sets& s, int z) {
    int i = 0;
    while (i + 1 < s.n_sets && z >= s.z0[i + 1]) ++i;
    return i;
}

// ---- comparison -----------------------------------------------------------------------------------------------
// The kernels are specialised for the terms that the tensors U touch, and U can change in ways that leave no trace on the host (a write
// through .data, through another view of the memory, to a tensor without a version).  So every call compares the contents with the
// copy that the terms were made from.  Both are read from the L2: 3 MB for 0e + 1o at ell = 16.
struct Pairs { int n; const unsigned *a[MAX_SETS], *b[MAX_SETS]; long long words[MAX_SETS]; };
constexpr int CMP_BLOCKS = 64, CMP_THREADS = 256;

__global__ void __launch_bounds__(CMP_THREADS) compare(const __grid_constant__ Pairs p, int* changed, int code) {
    const unsigned *a = p.a[blockIdx.y], *b = p.b[blockIdx.y];
    const long long words = p.words[blockIdx.y], step = (long long)CMP_BLOCKS * CMP_THREADS;
    const long long at = blockIdx.x * (long long)CMP_THREADS + threadIdx.x;
    const long long quads = ((uintptr_t)a | (uintptr_t)b) % 16 == 0 ? words / 4 : 0;   // (a buffer may start anywhere in its storage)
    unsigned differ = 0;
    for (long long i = at; i < quads; i += step) {
        const uint4 v = reinterpret_cast<const uint4*>(a)[i], w = reinterpret_cast<const uint4*>(b)[i];
        differ |= (v.x ^ w.x) | (v.y ^ w.y) | (v.z ^ w.z) | (v.w ^ w.w);
    }
    for (long long i = 4 * quads + at; i < words; i += step) differ |= a[i] ^ b[i];
    if (differ) *(volatile int*)changed = code;   // host memory
}

// ---- grouping -------------------------------------------------------------------------------------------------
// group: [0, N) node ids by element, [N, N + G + 1) element offsets, then [1 + 2 * (N / 32 + G + 1)] the number of tiles and
// (element, first position) of each.  One block, stable: warp v takes a contiguous piece of the nodes; pieces are counted,
// scanned over (element, warp) and placed in node order.  An element counts from the end if it is negative, as an index does.  Nodes of
// no element come last, as those of element G: they are reported through the status word and their rows are zero.
constexpr int GROUP_WARPS = 32;
inline long long max_tiles(long long n, int G) { return n / TILE + G + 1; }
inline long long group_ints(long long n, int G) { return n + (G + 1) + 1 + 2 * max_tiles(n, G); }

__device__ __forceinline__ int element_of(long long k, int G) { return k >= 0 && k < G ? (int)k : k < 0 && k >= -(long long)G ? (int)k + G : G; }

__global__ void __launch_bounds__(32 * GROUP_WARPS) group_nodes(const long long* __restrict__ keys, long long n, int G, int* __restrict__ group,
                                                               int* status, int code) {
    extern __shared__ int hist[];      // [G + 1][GROUP_WARPS]
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    for (int i = threadIdx.x; i < (G + 1) * GROUP_WARPS; i += blockDim.x) hist[i] = 0;
    __syncthreads();
    const long long per = ((n + GROUP_WARPS - 1) / GROUP_WARPS + 31) / 32 * 32;
    const long long lo = warp * per, hi = (lo + per < n) ? lo + per : n;
    for (long long i = lo + lane; i < hi; i += 32) atomicAdd(&hist[element_of(keys[i], G) * GROUP_WARPS + warp], 1);
    __syncthreads();
    // exclusive scan over (element, warp), one warp, 32 entries at a time: an element's entries are exactly one row
    int* off = group + n;
    if (warp == 0) {
        int carry = 0, tiles = 0;
        int* tl = off + G + 1;
        for (int g = 0; g <= G; ++g) {
            const int v = hist[g * GROUP_WARPS + lane];
            int inc = v;
#pragma unroll
            for (int d = 1; d < 32; d <<= 1) {
                const int o = __shfl_up_sync(0xffffffffu, inc, d);
                if (lane >= d) inc += o;
            }
            hist[g * GROUP_WARPS + lane] = carry + inc - v;
            const int cnt = __shfl_sync(0xffffffffu, inc, 31);
            if (lane == 0) off[g] = carry;
            for (int t = lane; t < (cnt + TILE - 1) / TILE; t += 32) {
                tl[1 + 2 * (tiles + t)] = g;
                tl[2 + 2 * (tiles + t)] = carry + t * TILE;
            }
            tiles += (cnt + TILE - 1) / TILE;
            carry += cnt;
            if (g == G && cnt > 0 && lane == 0) *(volatile int*)status = code;
        }
        if (lane == 0) tl[0] = tiles;
    }
    __syncthreads();
    for (long long i0 = lo; i0 < hi; i0 += 32) {
        const long long i = i0 + lane;
        const int k = i < hi ? element_of(keys[i], G) : -1;
        const unsigned same = __match_any_sync(0xffffffffu, k);
        if (k >= 0) group[hist[k * GROUP_WARPS + warp] + __popc(same & ((1u << lane) - 1u))] = (int)i;
        __syncwarp();
        if (k >= 0 && (same >> lane) == 1u) hist[k * GROUP_WARPS + warp] += __popc(same);   // the last lane of its element
        __syncwarp();
    }
}

// ---- coefficients ---------------------------------------------------------------------------------------------
// coef[e][term / 4][f][4]; a block takes 16 rows of one set for 128 channels: a weight is read once for 16 terms
constexpr int CO_ROWS = 16, CO_THREADS = 128, CO_K = 64;
template <typename T>
__global__ void __launch_bounds__(CO_THREADS) coefficients(const __grid_constant__ Sets s, const T* __restrict__ U,
                                                           const __grid_constant__ Pointers weights, T* __restrict__ coef) {
    __shared__ __align__(16) T us[CO_K][CO_ROWS];
    const int set = set_of(s, blockIdx.x), e = blockIdx.z, f = blockIdx.y * CO_THREADS + threadIdx.x;
    const int K = s.k[set], r0 = s.t0[set] + ((int)blockIdx.x - s.z0[set]) * CO_ROWS;
    const int nr = s.t1[set] - r0 < CO_ROWS ? s.t1[set] - r0 : CO_ROWS;
    const T* u = U + s.u[set] + (long long)(r0 - s.t0[set]) * K;
    const T* w = (const T*)weights.p[set] + (long long)e * K * s.F + f;
    T acc[CO_ROWS];
#pragma unroll
    for (int r = 0; r < CO_ROWS; ++r) acc[r] = T(0);
    for (int k0 = 0; k0 < K; k0 += CO_K) {
        const int nk = K - k0 < CO_K ? K - k0 : CO_K;
        __syncthreads();
        for (int i = threadIdx.x; i < CO_ROWS * nk; i += CO_THREADS) {
            const int r = i / nk, k = i % nk;
            us[k][r] = r < nr ? u[(long long)r * K + k0 + k] : T(0);
        }
        __syncthreads();
        if (f < s.F) {
#pragma unroll 16
            for (int k = 0; k < nk; ++k) {
                const T wk = __ldg(w + (long long)(k0 + k) * s.F);
#pragma unroll
                for (int r = 0; r < CO_ROWS; ++r) acc[r] = fma(us[k][r], wk, acc[r]);
            }
        }
    }
    if (f >= s.F) return;
    const int quads = (s.terms + 3) / 4;
#pragma unroll
    for (int r = 0; r < CO_ROWS; ++r)
        if (r < nr) {
            const int t = s.place[r0 + r];
            coef[(((long long)e * quads + t / 4) * s.F + f) * 4 + (t & 3)] = acc[r];
        }
}

// ---- gradient of the weights ----------------------------------------------------------------------------------
// part[slice][e][term][f]: sums of cot * monomial.  A block takes 64 columns of one set for 32 channels: it adds the slices of
// the set's terms in order, then every warp forms four columns (U four columns at a time from shared memory: as uniform loads
// from global memory they took 53 us for 410 terms, 86 columns, 10 elements and 128 channels).
constexpr int GW_COLS = 64, GW_THREADS = 512;
template <typename T> struct GwRows { static constexpr int value = sizeof(T) == 8 ? 32 : 64; };
template <typename T>
__global__ void __launch_bounds__(GW_THREADS) gradient_w(const __grid_constant__ Sets s, int G, const T* __restrict__ U, const T* __restrict__ part,
                                                         int slices, const __grid_constant__ Pointers dweights) {
    constexpr int GW_ROWS = GwRows<T>::value;
    __shared__ T sum[GW_ROWS][32];
    __shared__ __align__(16) T us[GW_ROWS][GW_COLS];
    const int set = set_of(s, blockIdx.x), e = blockIdx.z, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int f = blockIdx.y * 32 + lane;
    const int K = s.k[set], kb = ((int)blockIdx.x - s.z0[set]) * GW_COLS, k0 = kb + 4 * warp;
    T acc[4] = {T(0), T(0), T(0), T(0)};
    for (int r0 = s.t0[set]; r0 < s.t1[set]; r0 += GW_ROWS) {
        const int nr = s.t1[set] - r0 < GW_ROWS ? s.t1[set] - r0 : GW_ROWS;
        const T* u = U + s.u[set] + (long long)(r0 - s.t0[set]) * K + kb;
        const int nk = K - kb < GW_COLS ? K - kb : GW_COLS;
        __syncthreads();
        for (int r = warp; r < nr; r += GW_THREADS / 32)
            for (int c = lane; c < GW_COLS; c += 32) us[r][c] = c < nk ? __ldg(u + (long long)r * K + c) : T(0);
        for (int r = warp; r < nr; r += GW_THREADS / 32) {
            const T* src = part + ((long long)e * s.terms + s.place[r0 + r]) * s.F + f;
            T v = T(0);
            if (f < s.F) {
#pragma unroll 8
                for (int c = 0; c < slices; ++c) v += __ldg(src + (long long)c * G * s.terms * s.F);
            }
            sum[r][lane] = v;
        }
        __syncthreads();
        if (k0 < K) {
#pragma unroll 8
            for (int r = 0; r < nr; ++r) {
                const T m = sum[r][lane];
#pragma unroll
                for (int c = 0; c < 4; ++c) acc[c] = fma(us[r][4 * warp + c], m, acc[c]);
            }
        }
    }
    T* dst = (T*)dweights.p[set] + ((long long)e * K + k0) * s.F + f;
#pragma unroll
    for (int c = 0; c < 4; ++c)
        if (f < s.F && k0 + c < K) dst[(long long)c * s.F] = acc[c];
}

// ---- launches -------------------------------------------------------------------------------------------------
inline cudaError_t run_compare(const Pairs& p, int* changed, int code, cudaStream_t st) {
    compare<<<dim3(CMP_BLOCKS, (unsigned)p.n), CMP_THREADS, 0, st>>>(p, changed, code);
    return cudaGetLastError();
}

inline cudaError_t run_group(const long long* keys, long long n, int G, int* group, int* status, int code, cudaStream_t st) {
    group_nodes<<<1, 32 * GROUP_WARPS, sizeof(int) * (size_t)(G + 1) * GROUP_WARPS, st>>>(keys, n, G, group, status, code);
    return cudaGetLastError();
}

template <typename T>
cudaError_t run_coefficients(Sets s, int G, const T* U, const Pointers& w, T* coef, cudaStream_t st) {
    for (int i = 0; i < s.n_sets; ++i) s.z0[i + 1] = s.z0[i] + (s.t1[i] - s.t0[i] + CO_ROWS - 1) / CO_ROWS;
    if (s.z0[s.n_sets] == 0) return cudaSuccess;
    coefficients<T><<<dim3((unsigned)s.z0[s.n_sets], (unsigned)((s.F + CO_THREADS - 1) / CO_THREADS), (unsigned)G), CO_THREADS, 0, st>>>(s, U, w, coef);
    return cudaGetLastError();
}

template <typename T>
cudaError_t run_gradient_w(Sets s, int G, const T* U, const T* part, int slices, const Pointers& dw, cudaStream_t st) {
    for (int i = 0; i < s.n_sets; ++i) s.z0[i + 1] = s.z0[i] + (s.k[i] + GW_COLS - 1) / GW_COLS;
    if (s.z0[s.n_sets] == 0) return cudaSuccess;
    gradient_w<T><<<dim3((unsigned)s.z0[s.n_sets], (unsigned)((s.F + 31) / 32), (unsigned)G), GW_THREADS, 0, st>>>(s, G, U, part, slices, dw);
    return cudaGetLastError();
}

}  // namespace symc
