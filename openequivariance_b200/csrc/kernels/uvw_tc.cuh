// 'uvw' products with shared weights on the 5th-generation tensor cores (tcgen05), 32-wide multiplicities, fp32.
//
//   z[b, o][w, k] = sum over paths p: a -> o and components i of   cy_p[b][i, k] * U_p[b][w, i]
//   U_p[b][w, i]  = sum_u W_p[u, w] x[b, a][u, i]                  (tensor cores)
//   cy_p[b][i, k] = sum_j C_p[i, j, k] y[b][j]                     (CUDA cores, one coefficient per item)
//
// The weights are applied first, to the raw components of the input, and the Clebsch-Gordan sums run over the products.  The other order
// (Clebsch-Gordan sums into the A operand, one per path and output component) needs an operand of 128 x 32 per (path, k), 102 for the 30
// paths of 32x(0+1+2, both parities); this one needs one per set and input component, 36 a tile in the forward (two sets) and 68 for the
// gradients (four), and its sums in tensor memory are 32 products long (the tensor cores add with truncation, so the error of a sum grows with
// its length).
// The gradient of x is the same computation on the cotangent with the weights transposed, and the gradient of y takes its products
// from the same accumulators:
//   V_p[b][u, k] = sum_w W_p[u, w] g[b, o][w, k]      dx[b, a][u, i] = sum cy_p[b][i, k] V_p[b][u, k]
//   dy[b][j]     = sum C_p[i, j, k] sum_u x[b, a][u, i] V_p[b][u, k]
// Below "source" is the operand whose components are multiplied by weights (x, or g) and "destination" the one that is summed.
// fp32 accuracy comes from the 3xTF32 split: every operand is hi = tf32(v), lo = v - hi and each product is issued as
// lo*hi + hi*lo + hi*hi, accumulated in fp32.  Reference counterpart: the scalar-FMA warp matmul of templates/wmm.cuh:1-87.
//
// A CTA (one per SM) works on tiles of 128 items.  The destination is dealt into sets of tiles of few components, so that a thread's sums
// fit its registers (the set's visits name the source blocks that it reads, with up to TC_NSUB weight tiles each: the N of the MMA).
// For every component of a visited source block ("chunk") the warps pass on:
//   warp 13      the block's 128 rows to shared memory (tiled copies), a block ahead
//   warps 14-15  the visit's weight tiles, split and in the canonical K-major layout, to shared memory, a block ahead
//   warps 8-11   the component's 128 x 32 values, split, to tensor memory (A operand; a ring of TC_NA)
//   warp 12      12 MMAs of 128 x (TC_NSUB tiles) x 8 into one of two accumulators
//   warps 0-7    accumulators -> registers, times the coefficients, into the destination's sums; rows are stored at a set's end
// coupled through mbarriers only.  The A operand lives in tensor memory because the shared-memory pipe would otherwise carry it twice
// (store, and two reads by the MMAs) and set the pace.  Channel 8 g + c + 4 e of a block is column 8 g + 2 c + e of A and row of B
// (both agree, so the products do not change): with it the conversion's reads fall into 32 different banks.
// Registers: 512 threads start with 128; the conversion and issue warpgroups hand theirs to the two that keep the sums (setmaxnreg).
// Every mbarrier wait is bounded; on time-out the CTA leaves after its copies and MMAs have ended and its tensor memory is free.
// What bounds it: instruction latency (0.41 instructions a cycle and scheduler, long-scoreboard stalls first; tensor pipe 29 % forward, 15 %
// gradients).  50,000 items of 32x(0+1+2, both parities): forward 455 us with the Clebsch-Gordan sums first, 117 us; gradients of x and y
// 1,070 us in two kernels of that kind, 219 us.
#pragma once
#if OEQ_TC

OEQ_DEV unsigned tc_smem_u32(const void* p) { return (unsigned)__cvta_generic_to_shared(p); }
OEQ_DEV void tc_mbar_init(unsigned long long* bar, unsigned count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(tc_smem_u32(bar)), "r"(count) : "memory");
}
// A wait gives up after 3.5e9 cycles, about two seconds (the count is of 32 bits and looked at far more often than it wraps), or when another
// thread did.  A handful of instructions, because it is inlined at every step of straight-line code: who gives up reports it with tc_give_up.
OEQ_DEV bool tc_mbar_wait(unsigned long long* bar, unsigned parity, const int* abort_flag) {
    unsigned ok;
    asm volatile(
        "{ .reg .pred p; .reg .u32 t0, t, a;\n"
        "  mov.u32 t0, %%clock;\n"
        "W: mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n"
        "  @p bra D;\n"
        "  ld.volatile.shared.u32 a, [%3];\n"
        "  setp.ne.u32 p, a, 0;\n"
        "  @p bra F;\n"
        "  mov.u32 t, %%clock;\n"
        "  sub.u32 t, t, t0;\n"
        "  setp.lt.u32 p, t, 3500000000;\n"
        "  @p bra W;\n"
        "F: setp.ne.u32 p, 0, 0;\n"
        "D: selp.u32 %0, 1, 0, p; }"
        : "=r"(ok) : "r"(tc_smem_u32(bar)), "r"(parity), "r"(tc_smem_u32(abort_flag)) : "memory");
    return ok != 0;
}
// ... by a warp, which goes on or gives up as one (what follows a wait may be a warp-wide instruction)
OEQ_DEV bool tc_warp_wait(unsigned long long* bar, unsigned parity, const int* abort_flag) {
    return __all_sync(0xffffffffu, tc_mbar_wait(bar, parity, abort_flag)) != 0;
}
OEQ_DEV void tc_give_up(int* abort_flag, int* status, int code) {
    if (*(volatile int*)abort_flag == 0) *(volatile int*)status = code;   // the first to give up; the others follow the flag
    *(volatile int*)abort_flag = 1;
}
// A box of 32 floats x 128 rows (TC_MODE 3: 32 rows) by a tiled copy (TMA; rows past the end of the tensor arrive as zeros).  The map's swizzle
// (not in mode 3) puts 16-byte piece c of row r of the box at piece c ^ (r % 8) of its 128 bytes.
struct alignas(64) TcMap { unsigned long long opaque[16]; };
OEQ_DEV void tc_tile_load(void* dst_smem, const TcMap* map, int x, int row, unsigned long long* bar) {
    asm volatile("cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];"
                 ::"r"(tc_smem_u32(dst_smem)), "l"(map), "r"(x), "r"(row), "r"(tc_smem_u32(bar)) : "memory");
}
OEQ_DEV void tc_mbar_expect_tx(unsigned long long* bar, unsigned bytes) {
    asm volatile("{ .reg .b64 st; mbarrier.arrive.expect_tx.shared::cta.b64 st, [%0], %1; }" ::"r"(tc_smem_u32(bar)), "r"(bytes) : "memory");
}
OEQ_DEV float tc_tf32(float v) {   // round to tf32 (10-bit mantissa), result is a valid fp32 bit pattern
    unsigned r;
    asm("cvt.rna.tf32.f32 %0, %1;" : "=r"(r) : "f"(v));
    return __uint_as_float(r);
}

// Shared-memory matrix descriptor, K-major, no swizzle: 8-row x 16-byte core matrices; LBO = distance between core
// matrices adjacent in K, SBO = distance between 8-row groups.  Bits: [0,14) address>>4, [16,30) LBO>>4,
// [32,46) SBO>>4, [46,48) descriptor version 1, [61,64) swizzle mode 0.
OEQ_DEV unsigned long long tc_desc(const void* smem, unsigned lbo_bytes, unsigned sbo_bytes) {
    unsigned long long d = 0;
    d |= (unsigned long long)((tc_smem_u32(smem) & 0x3FFFFu) >> 4);
    d |= (unsigned long long)((lbo_bytes >> 4) & 0x3FFFu) << 16;
    d |= (unsigned long long)((sbo_bytes >> 4) & 0x3FFFu) << 32;
    d |= 1ull << 46;
    return d;
}
// Instruction descriptor for kind::tf32, fp32 accumulate, both operands K-major, M = 128:
// [4,6) D format 1 = f32, [7,10) A format 2 = tf32, [10,13) B format 2 = tf32, [17,23) N>>3, [24,29) M>>4.
OEQ_DEV constexpr unsigned tc_idesc(unsigned n) { return (1u << 4) | (2u << 7) | (2u << 10) | ((n >> 3) << 17) | ((128u >> 4) << 24); }

OEQ_DEV void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
OEQ_DEV void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
OEQ_DEV void tc_fence_async_smem() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }

// Operand geometry: 32 K-columns = 8 core matrices of 128 bytes, 16 bytes apart, per 8-row group
constexpr unsigned TC_LBO = 144, TC_SBO = 8 * TC_LBO;
OEQ_DEV void tc_mbar_arrive(unsigned long long* bar) {
    asm volatile("{ .reg .b64 st; mbarrier.arrive.shared::cta.b64 st, [%0]; }" ::"r"(tc_smem_u32(bar)) : "memory");
}

// (by a whole warp with the same operands, one elected lane issues: the operands then stay in uniform registers.  Issued inside a branch of
// one lane, every operand was moved there afresh and an MMA took 70 cycles to issue, more than it takes to run.)
OEQ_DEV void tc_mma_ts(unsigned tmem_d, unsigned tmem_a, unsigned long long bdesc, unsigned idesc, unsigned accumulate) {
    asm volatile(
        "{ .reg .pred p, q; elect.sync _|q, 0xffffffff; setp.ne.b32 p, %4, 0;\n"
        "  @q tcgen05.mma.cta_group::1.kind::tf32 [%0], [%1], %2, %3, p; }"
        ::"r"(tmem_d), "r"(tmem_a), "l"(bdesc), "r"(idesc), "r"(accumulate) : "memory");
}
OEQ_DEV void tc_commit_elected(unsigned long long* bar) {
    asm volatile("{ .reg .pred q; elect.sync _|q, 0xffffffff;\n"
                 "  @q tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0]; }" ::"r"(tc_smem_u32(bar)) : "memory");
}

#if TC_MODE != 3
// TC_MODE (with the tables): 0 forward, 1 gradients of x and y.
struct TcParams {
    TcMap src;          // of the source operand: x, or the cotangent
    const float* y;
    const float* W;     // 16-byte aligned
    float* dst;
    const float* x;     // mode 1: the first input
    float* dy;          // mode 1: the gradient of y, or (parts > 1) rows [part][item] of contributions to it
    long long batch;
    int accum;          // add to what dst (and dy, when there is one part) holds instead of overwriting it
    int* status;
    int parts;          // a tile's instances are shared by this many CTAs: part s takes cut[s] .. cut[s + 1] of the list
    int cut[TC_MAX_PARTS + 1];
};

constexpr int TC_THREADS = 512;
constexpr int TC_CH = TC_TW / 2;                        // destination channels of a thread (of TC_TW in a tile)
constexpr int TC_DW = TC_NSUB * TC_TW;                  // columns of an accumulator
constexpr int TC_NA = (512 - 2 * TC_DW) / 64 < 6 ? (512 - 2 * TC_DW) / 64 : 6;   // A operands (hi, lo: 32 columns each) in tensor memory
static_assert(TC_NA >= 2, "tensor memory");
constexpr int TC_XS_FLOATS = 128 * 32 * TC_MAXD;        // a staged block: d boxes of 128 rows x 128 bytes
constexpr int TC_B_FLOATS = TC_DW / 8 * (TC_SBO / 4);   // weight tiles of a visit, hi or lo
// setmaxnreg: two warpgroups of sums, one of conversion, one of copies and MMAs; 2 * 184 + 56 + 88 = 4 * 128
constexpr int TC_REG_SUMS = 184, TC_REG_CONV = 56, TC_REG_ISSUE = 88;

struct __align__(1024) TcShared {
    float xs[TC_NXS][TC_XS_FLOATS];
    float b[2][2][TC_B_FLOATS];                  // [buffer][hi, lo]
    float dys[TC_MODE == 1 ? 128 * (L2_DIM | 1) : 4];   // sums of dy of the warps 4 to 7
    unsigned long long xs_full[2], xs_empty[2];  // staged rows have arrived (bytes) / are converted
    unsigned long long b_full[2], b_empty[2];    // weight tiles are in place / have been multiplied
    unsigned long long a_full[TC_NA], a_empty[TC_NA];
    unsigned long long d_full[2], d_empty[2];    // accumulators are complete / are in registers
    unsigned long long dy_full, dy_empty, drain;
    unsigned tmem_base;
    int abort_flag, never;                       // (`never` stays zero: for waits that do not end with the abort flag)
};
static_assert(sizeof(TcShared) <= 232448, "the buffers exceed shared memory");
static_assert(sizeof(TcShared) <= TC_SMEM_BYTES, "the host sized the dynamic shared memory too small");

// A operand: 16 rows x 16 columns of tensor memory from a warp, row lane / 4 (+ 8) and columns 8 g + 2 (lane % 4) + {0, 1} in v[4 g + {0, 1}]
// (+ {2, 3} for row + 8)
OEQ_DEV void tc_st_a(unsigned taddr, const float (&v)[8]) {
    asm volatile("tcgen05.st.sync.aligned.16x256b.x2.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};"
                 ::"r"(taddr), "f"(v[0]), "f"(v[1]), "f"(v[2]), "f"(v[3]), "f"(v[4]), "f"(v[5]), "f"(v[6]), "f"(v[7]) : "memory");
}
// TC_CH consecutive accumulator columns of this thread's lane; tc_ld_wait makes them readable
OEQ_DEV void tc_ld(unsigned taddr, float (&r)[8]) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
                 : "=f"(r[0]), "=f"(r[1]), "=f"(r[2]), "=f"(r[3]), "=f"(r[4]), "=f"(r[5]), "=f"(r[6]), "=f"(r[7]) : "r"(taddr) : "memory");
}
OEQ_DEV void tc_ld_wait(float (&r)[8]) {
    asm volatile("tcgen05.wait::ld.sync.aligned;" : "+f"(r[0]), "+f"(r[1]), "+f"(r[2]), "+f"(r[3]), "+f"(r[4]), "+f"(r[5]), "+f"(r[6]), "+f"(r[7]) :: "memory");
}
OEQ_DEV void tc_ld(unsigned taddr, float (&r)[16]) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
                 : "=f"(r[0]), "=f"(r[1]), "=f"(r[2]), "=f"(r[3]), "=f"(r[4]), "=f"(r[5]), "=f"(r[6]), "=f"(r[7]), "=f"(r[8]), "=f"(r[9]),
                   "=f"(r[10]), "=f"(r[11]), "=f"(r[12]), "=f"(r[13]), "=f"(r[14]), "=f"(r[15]) : "r"(taddr) : "memory");
}
OEQ_DEV void tc_ld_wait(float (&r)[16]) {
    asm volatile("tcgen05.wait::ld.sync.aligned;" : "+f"(r[0]), "+f"(r[1]), "+f"(r[2]), "+f"(r[3]), "+f"(r[4]), "+f"(r[5]), "+f"(r[6]), "+f"(r[7]),
                 "+f"(r[8]), "+f"(r[9]), "+f"(r[10]), "+f"(r[11]), "+f"(r[12]), "+f"(r[13]), "+f"(r[14]), "+f"(r[15]) :: "memory");
}
// Two channels' values in one register pair: the sums run on packed multiply-adds (fma.rn.f32x2), half the instructions.  The sets' code is
// straight-line, and with twice the size the warps waited for instructions (no_instruction stalls first, 0.23 instructions a cycle).
typedef unsigned long long TcPair;
OEQ_DEV TcPair tc_pack(float a, float b) { TcPair r; asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b)); return r; }
OEQ_DEV float tc_half(TcPair v, int h) {
    float a, b;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(v));
    return h ? b : a;
}
// What the sets' code (emitted) is made of: sums += c * products, and a dot product over the thread's channels.  One statement each: the
// compiler's time goes with their number.
constexpr int TC_H = TC_CH / 2;
OEQ_DEV void tc_axpy(float c, const TcPair (&u)[TC_H], TcPair* z) {
    if constexpr (TC_H == 4)
        asm("{ .reg .b64 c; mov.b64 c, {%4, %4}; fma.rn.f32x2 %0, c, %5, %0; fma.rn.f32x2 %1, c, %6, %1; fma.rn.f32x2 %2, c, %7, %2; fma.rn.f32x2 %3, c, %8, %3; }"
            : "+&l"(z[0]), "+&l"(z[1]), "+&l"(z[2]), "+&l"(z[3]) : "f"(c), "l"(u[0]), "l"(u[1]), "l"(u[2]), "l"(u[3]));
    else
        asm("{ .reg .b64 c; mov.b64 c, {%8, %8}; fma.rn.f32x2 %0, c, %9, %0; fma.rn.f32x2 %1, c, %10, %1; fma.rn.f32x2 %2, c, %11, %2; fma.rn.f32x2 %3, c, %12, %3;\n"
            "  fma.rn.f32x2 %4, c, %13, %4; fma.rn.f32x2 %5, c, %14, %5; fma.rn.f32x2 %6, c, %15, %6; fma.rn.f32x2 %7, c, %16, %7; }"
            : "+&l"(z[0]), "+&l"(z[1]), "+&l"(z[2]), "+&l"(z[3]), "+&l"(z[4]), "+&l"(z[5]), "+&l"(z[6]), "+&l"(z[7])
            : "f"(c), "l"(u[0]), "l"(u[1]), "l"(u[2]), "l"(u[3]), "l"(u[4]), "l"(u[5]), "l"(u[6]), "l"(u[7]));
}
#if TC_MODE == 1
static_assert(TC_H == 4, "channels of a thread");
OEQ_DEV float tc_dot(const TcPair* x, const TcPair (&u)[TC_H]) {
    float s;
    asm("{ .reg .b64 a, b; .reg .f32 f, g; mul.rn.f32x2 a, %1, %5; mul.rn.f32x2 b, %2, %6; fma.rn.f32x2 a, %3, %7, a; fma.rn.f32x2 b, %4, %8, b;\n"
        "  add.rn.f32x2 a, a, b; mov.b64 {f, g}, a; add.rn.f32 %0, f, g; }"
        : "=f"(s) : "l"(x[0]), "l"(x[1]), "l"(x[2]), "l"(x[3]), "l"(u[0]), "l"(u[1]), "l"(u[2]), "l"(u[3]));
    return s;
}
#endif

// A thread's channels of a destination (or first-input) block are TC_CH * D consecutive floats of its item's row; component k of channels
// 2 q, 2 q + 1 is v[k * TC_CH / 2 + q].  Global memory is read and written 8 floats of a row (a sector) at a time by two neighbouring lanes,
// which exchange halves: a lane per row instead costs a line and half a sector per lane and access (15,000 of the 65,000 cycles of a set),
// and a transposition through shared memory four times the accesses of the exchange (12,000).
constexpr int TC_RUN = 8;
OEQ_DEV void tc_put(TcPair* v, int D, int f, float x) {   // float f of the thread's channels (in order: the even channel of a pair first)
    TcPair& p = v[f % D * (TC_CH / 2) + f / D / 2];
    p = f / D & 1 ? tc_pack(tc_half(p, 0), x) : tc_pack(x, 0.f);
}
// rows 0 .. live of the warp's 32 at `rows` (live < 1: none is stored; something is read all the same)
template <int D>
OEQ_DEV void tc_rows_load(const float* rows, int live, TcPair* v, int lane) {
    constexpr int RUNS = TC_CH * D / TC_RUN;
    asm volatile("mov.b32 %0, %0;" : "+r"(lane));   // (addresses are formed here every time: kept across the sums they would spill)
    const int even = lane & ~1, odd = lane | 1;
    const float* at0 = rows + (even < live ? (long long)even * TC_OUT_DIM : 0ll) + 4 * (lane & 1);   // half a sector of the even lane's row,
    const float* at1 = rows + (odd < live ? (long long)odd * TC_OUT_DIM : 0ll) + 4 * (lane & 1);     // and of the odd lane's
#pragma unroll
    for (int c0 = 0; c0 < RUNS; c0 += 5) {           // ten loads in flight
        float4 t[5][2];
#pragma unroll
        for (int c = c0; c < RUNS && c < c0 + 5; ++c) {
            t[c - c0][0] = __ldg(reinterpret_cast<const float4*>(at0 + c * TC_RUN));
            t[c - c0][1] = __ldg(reinterpret_cast<const float4*>(at1 + c * TC_RUN));
        }
#pragma unroll
        for (int c = c0; c < RUNS && c < c0 + 5; ++c) {
            const float a[4] = {t[c - c0][0].x, t[c - c0][0].y, t[c - c0][0].z, t[c - c0][0].w}, b[4] = {t[c - c0][1].x, t[c - c0][1].y, t[c - c0][1].z, t[c - c0][1].w};
            float run[TC_RUN];
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                const float got = __shfl_xor_sync(0xffffffffu, lane & 1 ? a[e] : b[e], 1);
                run[e] = lane & 1 ? got : a[e];
                run[4 + e] = lane & 1 ? b[e] : got;
            }
#pragma unroll
            for (int e = 0; e < TC_RUN; ++e) tc_put(v, D, c * TC_RUN + e, run[e]);
        }
    }
}
template <int D>
OEQ_DEV void tc_rows_store(float* rows, int live, const TcPair* v, int lane, bool add) {
    constexpr int RUNS = TC_CH * D / TC_RUN;
    asm volatile("mov.b32 %0, %0;" : "+r"(lane));
    const int even = lane & ~1, odd = lane | 1;
    const unsigned how0 = even < live ? (add ? 2u : 1u) : 0u, how1 = odd < live ? (add ? 2u : 1u) : 0u;   // 0 nothing, 1 store, 2 add
    float* at0 = rows + (long long)even * TC_OUT_DIM + 4 * (lane & 1);
    float* at1 = at0 + TC_OUT_DIM;
    // (nobody else adds to these elements in this launch: the result does not depend on an order)
    auto out = [](float* at, const float (&g)[4], unsigned how) {
        asm volatile("{ .reg .pred p, q; setp.eq.u32 p, %5, 1; setp.eq.u32 q, %5, 2;\n"
                     "  @p st.global.cs.v4.f32 [%0], {%1, %2, %3, %4};\n"
                     "  @q red.global.add.v4.f32 [%0], {%1, %2, %3, %4}; }" ::"l"(at), "f"(g[0]), "f"(g[1]), "f"(g[2]), "f"(g[3]), "r"(how) : "memory");
    };
#pragma unroll
    for (int c = 0; c < RUNS; ++c) {
        float a[4], b[4];   // of the even lane's row and the odd lane's
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            const int f = c * TC_RUN + e, h = f + 4;
            const float lo = tc_half(v[f % D * (TC_CH / 2) + f / D / 2], f / D & 1), hi = tc_half(v[h % D * (TC_CH / 2) + h / D / 2], h / D & 1);
            const float got = __shfl_xor_sync(0xffffffffu, lane & 1 ? lo : hi, 1);
            a[e] = lane & 1 ? got : lo;
            b[e] = lane & 1 ? hi : got;
        }
        out(at0 + c * TC_RUN, a, how0);
        out(at1 + c * TC_RUN, b, how1);
    }
}

// A step of a summing warp: wait for the products of a chunk, number nd, ...
OEQ_DEV bool tc_step(TcShared& sh, unsigned nd, float (&y)[L2_DIM]) {
    const bool ok = tc_warp_wait(&sh.d_full[nd & 1u], (nd >> 1) & 1u, &sh.abort_flag);
    // (coefficients of other steps are not kept for this one: as common subexpressions they spilled 70 registers)
#pragma unroll
    for (int j = 0; j < L2_DIM; ++j) asm volatile("" : "+f"(y[j]));
    tc_fence_after();
    return ok;
}
// ... take those of one weight tile ...
OEQ_DEV void tc_products(unsigned taddr, TcPair (&u)[TC_H]) {
    float v[TC_CH];
    tc_ld(taddr, v);
    tc_ld_wait(v);
#pragma unroll
    for (int q = 0; q < TC_H; ++q) u[q] = tc_pack(v[2 * q], v[2 * q + 1]);
}
// ... and give the accumulator back.
OEQ_DEV void tc_step_done(TcShared& sh, unsigned nd, int lane) {
    tc_fence_before();
    __syncwarp();
    if (lane == 0) tc_mbar_arrive(&sh.d_empty[nd & 1u]);
}
// One set of one tile for a summing warp: `live` items from row0 on, channels col .. col + TC_CH of every destination tile.  Sets that differ only
// in where their blocks and weights lie share their code (the two parities do).  The functions are emitted (emit_tc_sets):
//   bool tc_set_<code>(TC_SET_ARGS) for each code, bool tc_sum_set(code, TC_SET_ARGS)
#define TC_SET_ARGS const TcParams& p, TcShared& sh, const int set, const unsigned tmem, unsigned& nd, float (&y)[L2_DIM], float (&dy)[TC_MODE == 1 ? L2_DIM : 1], \
                    const long long row0, const int live, const int col, const int lane
#define TC_SET_PASS p, sh, set, tmem, nd, y, dy, row0, live, col, lane
//@ sets

// A program holds the large sets of the problem, which a CTA walks in turn, or (TC_PARTS) the large sets or those of one destination tile each, whose
// instances are dealt to p.parts CTAs.
extern "C" __global__ void __launch_bounds__(TC_THREADS, 1) TC_KERNEL_NAME(const __grid_constant__ TcParams p) {
    extern __shared__ __align__(1024) unsigned char tc_smem_raw[];
    TcShared& sh = *reinterpret_cast<TcShared*>(tc_smem_raw);
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    if (tid == 0) {
        for (int s = 0; s < 2; ++s) {
            tc_mbar_init(&sh.xs_full[s], 1); tc_mbar_init(&sh.xs_empty[s], 4);
            tc_mbar_init(&sh.b_full[s], 2); tc_mbar_init(&sh.b_empty[s], 1);
            tc_mbar_init(&sh.d_full[s], 1); tc_mbar_init(&sh.d_empty[s], 8);
        }
        for (int s = 0; s < TC_NA; ++s) { tc_mbar_init(&sh.a_full[s], 4); tc_mbar_init(&sh.a_empty[s], 1); }
        tc_mbar_init(&sh.dy_full, 4); tc_mbar_init(&sh.dy_empty, 4); tc_mbar_init(&sh.drain, 1);
        sh.abort_flag = sh.never = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], 512;" ::"r"(tc_smem_u32(&sh.tmem_base)) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const unsigned tmem = sh.tmem_base, tmem_a = tmem + 2 * TC_DW;
    const int parts = TC_PARTS ? p.parts : 1;
    const long long nunits = (p.batch + 127) / 128 * parts;
    // Every role walks the same list: units of this CTA, instances of the unit's part, visits of the instance's set, 32-channel chunks of the
    // visit's block.  f(tile, visit, chunk of the source block, tile of the destination) returns false to leave.
    auto walk = [&](auto&& f) -> bool {
#pragma unroll 1
        for (long long unit = blockIdx.x; unit < nunits; unit += gridDim.x) {
            const long long tile = unit / parts;
            const int part = (int)(unit % parts);
            const int n0 = TC_PARTS ? p.cut[part] : 0, n1 = TC_PARTS ? p.cut[part + 1] : TC_NINST;
#pragma unroll 1
            for (int n = n0; n < n1; ++n) {
                const int set = TC_INST_SET[n], wc = TC_INST_WC[n];
#pragma unroll 1
                for (int v = TC_SET_V[set]; v < TC_SET_V[set + 1]; ++v)
#pragma unroll 1
                    for (int uc = 0; uc < TC_V_NU[v]; ++uc)
                        if (!f(tile, v, uc, wc)) return false;
            }
        }
        return true;
    };

    bool ok = true;
    if (warp < 8) {
        // ---- sums
        asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(TC_REG_SUMS));
        const int quarter = warp & 3, half = warp >> 2;
        const unsigned t = tmem + ((unsigned)(quarter * 32) << 16) + (unsigned)(half * TC_CH);
        unsigned nd = 0, nunit = 0;
#pragma unroll 1
        for (long long unit = blockIdx.x; unit < nunits && ok; unit += gridDim.x, ++nunit) {
            const long long item = unit / parts * 128 + quarter * 32 + lane;
            const int part = (int)(unit % parts);
            const bool live = item < p.batch;
            const long long b = live ? item : 0, row0 = item - lane;
            const int rows = row0 < p.batch ? (int)(p.batch - row0 < 32 ? p.batch - row0 : 32) : 0;
            float y[L2_DIM], dy[TC_MODE == 1 ? L2_DIM : 1];
#pragma unroll
            for (int j = 0; j < L2_DIM; ++j) y[j] = __ldg(p.y + b * L2_DIM + j);
#pragma unroll
            for (int j = 0; j < (TC_MODE == 1 ? L2_DIM : 1); ++j) dy[j] = 0.f;
            const int n0 = TC_PARTS ? p.cut[part] : 0, n1 = TC_PARTS ? p.cut[part + 1] : TC_NINST;
#pragma unroll 1
            for (int n = n0; n < n1 && ok; ++n) {
                const int set = TC_INST_SET[n], col = TC_INST_WC[n] * TC_TW + half * TC_CH;
                ok = tc_sum_set(TC_SET_CODE[set], p, sh, set, t, nd, y, dy, rows > 0 ? row0 : 0, rows, col, lane);
            }
            if (TC_MODE == 1 && ok) {
                // both halves of the channels: warps 4 to 7 pass theirs on
                float* mine = sh.dys + (quarter * 32 + lane) * (L2_DIM | 1);
                if (half == 1) {
                    if (nunit > 0) ok = tc_warp_wait(&sh.dy_empty, (nunit - 1) & 1u, &sh.abort_flag);
                    if (ok) {
#pragma unroll
                        for (int j = 0; j < (TC_MODE == 1 ? L2_DIM : 1); ++j) mine[j] = dy[j];
                        __syncwarp();
                        if (lane == 0) tc_mbar_arrive(&sh.dy_full);
                    }
                } else {
                    ok = tc_warp_wait(&sh.dy_full, nunit & 1u, &sh.abort_flag);
                    if (ok) {
#pragma unroll
                        for (int j = 0; j < (TC_MODE == 1 ? L2_DIM : 1); ++j) dy[j] += mine[j];
                        __syncwarp();
                        if (lane == 0) tc_mbar_arrive(&sh.dy_empty);
                        if (live) {
                            float* out = p.dy + (part * p.batch + b) * L2_DIM;
                            const bool add = !TC_PARTS && p.accum;
#pragma unroll
                            for (int j = 0; j < (TC_MODE == 1 ? L2_DIM : 1); ++j) out[j] = add ? out[j] + dy[j] : dy[j];
                        }
                    }
                }
            }
        }
    } else if (warp < 12) {
        // ---- conversion: rows 32 quarter ... + 31 of the staged block, component by component, split into tensor memory
        asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(TC_REG_CONV));
        const int quarter = warp & 3;
        const unsigned ta = tmem_a + ((unsigned)(quarter * 32) << 16);
        unsigned ns = 0, ring = 0, lap = 0;   // staged blocks so far; A operand to fill next and its use
        ok = walk([&](long long, int v, int, int) -> bool {
            const int d = TC_V_D[v];
            const unsigned sbuf = ns % TC_NXS;
            if (!tc_warp_wait(&sh.xs_full[sbuf], (ns / TC_NXS) & 1u, &sh.abort_flag)) return false;
            const float* x0 = sh.xs[sbuf] + (quarter * 32 + (lane >> 2)) * 32;
#pragma unroll 1
            for (int i = 0; i < d; ++i) {
                if (lap > 0 && !tc_warp_wait(&sh.a_empty[ring], (lap - 1) & 1u, &sh.abort_flag)) return false;
                tc_fence_after();
                // component i of channel u is float u d + i of the row: box (u d + i) / 32.  Rows 8, 16 and 24 on have the same swizzle.
                const unsigned dst = ta + 64u * ring;
#pragma unroll
                for (int g = 0; g < 2; ++g) {      // columns 16 g ...
                    const float* at[4];
#pragma unroll
                    for (int q = 0; q < 4; ++q) {
                        const int f = ((lane & 3) + 16 * g + 4 * q) * d + i;
                        at[q] = x0 + (f >> 5) * 4096 + ((f >> 2 & 7) ^ (lane >> 2)) * 4 + (f & 3);
                    }
#pragma unroll
                    for (int h = 0; h < 2; ++h) {  // rows 16 h ...
                        float hi[8], lo[8];
#pragma unroll
                        for (int q = 0; q < 4; ++q) {
                            hi[(q >> 1) * 4 + (q & 1)] = at[q][512 * h];
                            hi[(q >> 1) * 4 + (q & 1) + 2] = at[q][512 * h + 256];
                        }
#pragma unroll
                        for (int q = 0; q < 8; ++q) {
                            const float r = tc_tf32(hi[q]);
                            lo[q] = hi[q] - r;   // 12 bits, of which the tensor core reads 11: what is lost is below 2^-23
                            hi[q] = r;
                        }
                        tc_st_a(dst + ((unsigned)(16 * h) << 16) + 16u * g, hi);
                        tc_st_a(dst + ((unsigned)(16 * h) << 16) + 16u * g + 32u, lo);
                    }
                }
                asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
                tc_fence_before();
                __syncwarp();
                if (lane == 0) tc_mbar_arrive(&sh.a_full[ring]);
                if (++ring == TC_NA) { ring = 0; ++lap; }
            }
            if (lane == 0) tc_mbar_arrive(&sh.xs_empty[sbuf]);   // (its reads precede the last __syncwarp)
            ++ns;
            return true;
        });
    } else {
        asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(TC_REG_ISSUE));
        if (warp == 12) {
            // ---- MMAs
            const unsigned utmem = __shfl_sync(0xffffffffu, tmem, 0);
            unsigned ns = 0, nd = 0, ring = 0, lap = 0;
            ok = walk([&](long long, int v, int, int) -> bool {
                const int d = TC_V_D[v];
                const unsigned bbuf = ns & 1u, idesc = tc_idesc((unsigned)(TC_V_NSUB[v] * TC_TW));
                const unsigned long long bh = tc_desc(sh.b[bbuf][0], TC_LBO, TC_SBO), bl = tc_desc(sh.b[bbuf][1], TC_LBO, TC_SBO);
                if (!tc_warp_wait(&sh.b_full[bbuf], (ns >> 1) & 1u, &sh.abort_flag)) return false;
#pragma unroll 1
                for (int i = 0; i < d; ++i) {
                    const unsigned dbuf = nd & 1u;
                    if (nd >= 2 && !tc_warp_wait(&sh.d_empty[dbuf], ((nd >> 1) - 1) & 1u, &sh.abort_flag)) return false;
                    if (!tc_warp_wait(&sh.a_full[ring], lap & 1u, &sh.abort_flag)) return false;
                    tc_fence_after();
                    const unsigned dcol = utmem + dbuf * TC_DW, ah = utmem + 2 * TC_DW + 64u * ring, al = ah + 32u;
                    // the small products first: less is lost to truncation in the sums
#pragma unroll
                    for (int ks = 0; ks < 4; ++ks) {
                        tc_mma_ts(dcol, al + 8u * ks, bh + TC_LBO / 8ull * ks, idesc, ks == 0 ? 0u : 1u);   // (a k-step is two core matrices)
                        tc_mma_ts(dcol, ah + 8u * ks, bl + TC_LBO / 8ull * ks, idesc, 1u);
                    }
#pragma unroll
                    for (int ks = 0; ks < 4; ++ks) tc_mma_ts(dcol, ah + 8u * ks, bh + TC_LBO / 8ull * ks, idesc, 1u);
                    tc_commit_elected(&sh.a_empty[ring]);
                    tc_commit_elected(&sh.d_full[dbuf]);
                    if (i + 1 == d) tc_commit_elected(&sh.b_empty[bbuf]);
                    __syncwarp();
                    ++nd;
                    if (++ring == TC_NA) { ring = 0; ++lap; }
                }
                ++ns;
                return true;
            });
            if (!ok) {   // given up: the MMAs in flight end before the tensor memory is freed
                if (lane == 0) tc_give_up(&sh.abort_flag, p.status, 41 + warp);
                __syncwarp();
                tc_commit_elected(&sh.drain);
                tc_mbar_wait(&sh.drain, 0u, &sh.never);
            }
        } else if (warp == 13) {
            // ---- rows: d boxes of 32 floats
            unsigned ns = 0;
            ok = walk([&](long long tile, int v, int uc, int) -> bool {
                const unsigned sbuf = ns % TC_NXS, use = ns / TC_NXS;
                if (use > 0 && !tc_warp_wait(&sh.xs_empty[sbuf], (use - 1) & 1u, &sh.abort_flag)) return false;
                const int d = TC_V_D[v];
                if (lane == 0) tc_mbar_expect_tx(&sh.xs_full[sbuf], 128u * 128u * (unsigned)d);
                __syncwarp();
                if (lane < d) tc_tile_load(sh.xs[sbuf] + lane * 4096, &p.src, TC_V_OFF[v] + uc * 32 * d + 32 * lane, (int)(tile * 128), &sh.xs_full[sbuf]);
                ++ns;
                return true;
            });
            if (!ok) {   // given up: the copies in flight end before the CTA does
                if (lane == 0) tc_give_up(&sh.abort_flag, p.status, 41 + warp);
                __syncwarp();
                for (unsigned s = ns > TC_NXS ? ns - TC_NXS : 0; s < ns; ++s) tc_mbar_wait(&sh.xs_full[s % TC_NXS], (s / TC_NXS) & 1u, &sh.never);
            }
        } else {
            // ---- weight tiles: B[n][k], n = destination channel of a tile, k = (permuted) source channel; columns 8 g + {0 .. 7} hold channels
            // 8 g + {0, 4, 1, 5, 2, 6, 3, 7}.  The two warps take the visit's 16-row pieces in turn, all requested before the buffer is waited for; a lane forms
            // four-by-four elements (forward: W is [k][n]) or two rows' eight k (gradients: W is [n][k]), so that loads and stores are of
            // 16 bytes.  TC_LBO is what keeps the forward's stores free of bank conflicts.
            constexpr int PIECES = TC_DW / 16, MINE = (PIECES + 1) / 2;
            const int w = warp - 14;
            unsigned ns = 0;
            ok = walk([&](long long, int v, int uc, int wc) -> bool {
                const int pieces = TC_V_NSUB[v] * (TC_TW / 16), wt = wc * TC_TW / 32;
                const unsigned bbuf = ns & 1u;
                float4 raw[MINE][4];
#pragma unroll
                for (int q = 0; q < MINE; ++q) {
                    const int piece = 2 * q + w;
                    if (piece < pieces) {
                        const int at = v * TC_NSUB + piece / (TC_TW / 16), n0 = wc * TC_TW % 32 + piece % (TC_TW / 16) * 16;
                        const float* tile = p.W + TC_V_W[at] + (TC_MODE == 0 ? uc : wt) * TC_V_WS[at] + (TC_MODE == 0 ? wt : uc) * 1024;
#pragma unroll
                        for (int j = 0; j < 4; ++j)
                            raw[q][j] = __ldg(reinterpret_cast<const float4*>(
                                TC_MODE == 0 ? tile + ((lane & 6) * 4 + (lane & 1) * 2 + (j >> 1) + (j & 1) * 4) * 32 + n0 + (lane >> 3) * 4
                                             : tile + (n0 + (lane & 7) + (j >> 1) * 8) * 32 + (lane >> 3) * 8 + (j & 1) * 4));
                    }
                }
                if (ns >= 2 && !tc_warp_wait(&sh.b_empty[bbuf], ((ns >> 1) - 1) & 1u, &sh.abort_flag)) return false;
#pragma unroll
                for (int q = 0; q < MINE; ++q) {
                    const int piece = 2 * q + w;
                    if (piece < pieces) {
                        const float4* f = raw[q];
                        const float e[4][4] = {{f[0].x, f[0].y, f[0].z, f[0].w}, {f[1].x, f[1].y, f[1].z, f[1].w},
                                               {f[2].x, f[2].y, f[2].z, f[2].w}, {f[3].x, f[3].y, f[3].z, f[3].w}};
#pragma unroll
                        for (int r = 0; r < 4; ++r) {
                            // forward: row 4 (lane / 8) + r, columns 4 (lane % 8) ...; gradients: row lane % 8 + 8 (r / 2), columns 8 (lane / 8) + 4 (r % 2) ...
                            const int row = 16 * piece + (TC_MODE == 0 ? (lane >> 3) * 4 + r : (lane & 7) + (r >> 1) * 8);
                            const int quad = TC_MODE == 0 ? lane & 7 : (lane >> 3) * 2 + (r & 1);
                            float hi[4], lo[4];
#pragma unroll
                            for (int c = 0; c < 4; ++c) {
                                const float x = TC_MODE == 0 ? e[c][r] : e[(r >> 1) * 2 + (c & 1)][(r & 1) * 2 + (c >> 1)];
                                hi[c] = tc_tf32(x);
                                lo[c] = x - hi[c];
                            }
                            const int at = (row >> 3) * (TC_SBO / 4) + quad * (TC_LBO / 4) + (row & 7) * 4;
                            *reinterpret_cast<float4*>(sh.b[bbuf][0] + at) = make_float4(hi[0], hi[1], hi[2], hi[3]);
                            *reinterpret_cast<float4*>(sh.b[bbuf][1] + at) = make_float4(lo[0], lo[1], lo[2], lo[3]);
                        }
                    }
                }
                tc_fence_async_smem();
                __syncwarp();
                if (lane == 0) tc_mbar_arrive(&sh.b_full[bbuf]);
                ++ns;
                return true;
            });
        }
    }
    if (!ok && lane == 0) tc_give_up(&sh.abort_flag, p.status, 41 + warp);
    tc_fence_before();
    __syncthreads();
    if (warp == 0) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, 512;" ::"r"(tmem) : "memory");
}

#if TC_MODE == 1 && TC_PARTS
// dy[e] = (accum ? dy[e] : 0) + sum of the parts' rows, in order
extern "C" __global__ void __launch_bounds__(256) oeq_uvw_tc_backward_dy_parts(const float* rows, float* dy, long long n, int parts, int accum) {
    const long long e = blockIdx.x * 256ll + threadIdx.x;
    if (e >= n) return;
    float v = accum ? dy[e] : 0.f;
    for (int s = 0; s < parts; ++s) v += __ldg(rows + s * n + e);
    dy[e] = v;
}
#endif
#endif  // TC_MODE != 3

#if TC_MODE == 3
// ---- gradient of the shared weights ---------------------------------------------------------------------------
//   dW_p[u, w] = sum_b sum_k T_p[b][u, k] * g[b, o][w, k],     T_p[b][u, k] = sum_i cy_p[b][i, k] x[b, a][u, i]
// A GEMM whose reduction runs over the batch.  Up to four weight tiles of one output tile are stacked on M (a group; they share the B operand g):
// per chunk (group, 32 items, component k)   D[(slot, u), w] += A[(slot, u), b] * B[w, b],   A = T, B = component k of the cotangent, items on K.
// The accumulators of up to TCW_MAX_GROUPS groups live in tensor memory for one tile of 64 items (a unit of work: a tile and a part of the
// groups); its sums are one row of a partials matrix that a second kernel adds in row order: bitwise reproducible, and short sums where the
// tensor cores add with truncation (a sum over 50,000 items was off by 1e-5).
//
// Warps (twenty-one), coupled through mbarriers only; a stage is (group, half of the tile):
//   warps 19-20  the stage's boxes of x and g to shared memory (tiled copies), and the coefficients cy of its 32 items, a stage ahead
//   warps 0-15   T: warp w works on slot w % 4 and items 8 (w / 4) ...; a lane is a channel, so the coefficients are the same for the warp and
//                the items' x are read once per stage; split into tensor memory (A operand, a ring of TCW_NA chunks)
//   warps 17-18  B: the cotangent's component, split, in the canonical K-major layout
//   warp 16      12 MMAs (128 x 32 x 8) a chunk
// A in tensor memory: lane = (slot, channel), column = item, which is how the T of a warp lie in its registers; through shared memory it would be
// stored twice and read three times.  50,000 items of 32x(0+1+2, both parities): 596 us with T formed from tables by all warps for
// operands in shared memory, 325 us.  What bounds it: instruction latency (0.51 instructions a cycle and scheduler, tensor pipe 12 %).
constexpr int TCW_AW = 16;                      // warps of T
constexpr int TC_THREADS = 32 * 21;
constexpr int TCW_TILE = 64;
constexpr int TCW_MAX_GROUPS = 8;
constexpr int TCW_NA = 4;                       // A operands of a chunk (32 columns hi, 32 lo)
constexpr unsigned TC_IDESC = tc_idesc(32);
constexpr int TCW_CYS = 36;                     // row of a pair's coefficients: the lanes' 16-byte stores fall into different banks
constexpr int TCW_PPL = (TCW_PAIRS + 63) / 64;  // pairs per lane of the coefficient warps
constexpr int TCW_B_FLOATS = 4 * (TC_SBO / 4);  // 32 rows of B, hi or lo
struct TcDwParams {
    TcMap x; TcMap g;
    const float* y; float* part;
    long long batch;
    int* status;
    int splits;                                 // a unit of work is a tile and a part of the groups
    int cut[TC_MAX_PARTS + 1];                  // part s: groups cut[s] .. cut[s + 1]
};
struct __align__(1024) TcDwShared {
    float xg[2][TCW_BOXES * 1024];              // boxes of 32 items x 32 floats: the slots' input blocks, the output block
    float b[2][2][TCW_B_FLOATS];                // [buffer][hi, lo]
    float cy[2][TCW_PAIRS * TCW_CYS];           // [pair][item]
    float ys[2][TCW_TILE * (L2_DIM | 1)];       // of the two coefficient warps
    unsigned long long xs_full[2], xs_empty[2];
    unsigned long long cy_full[2], cy_empty[2];
    unsigned long long a_full[TCW_NA], a_empty[TCW_NA];
    unsigned long long b_full[2], b_empty[2];
    unsigned long long d_full, d_free, drain;
    unsigned tmem_base;
    int abort_flag, never;
};
static_assert(sizeof(TcDwShared) <= 232448, "the buffers exceed shared memory");
static_assert(sizeof(TcDwShared) <= TC_SMEM_BYTES, "the host sized the dynamic shared memory too small");

typedef unsigned long long TcPair;              // two items
OEQ_DEV float tc_half(TcPair v, int h) {
    float a, b;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(v));
    return h ? b : a;
}
// what the cells (the sums of one component of T, emitted with the tables) are made of: eight items of one coefficient
struct TcwMath {
    typedef TcPair P;
    static OEQ_DEV void step(const P (&x)[4], const float* cy, P (&t)[4]) {
        const ulonglong2 c0 = *reinterpret_cast<const ulonglong2*>(cy), c1 = *reinterpret_cast<const ulonglong2*>(cy + 4);
        asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(t[0]) : "l"(c0.x), "l"(x[0]));
        asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(t[1]) : "l"(c0.y), "l"(x[1]));
        asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(t[2]) : "l"(c1.x), "l"(x[2]));
        asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(t[3]) : "l"(c1.y), "l"(x[3]));
    }
};
// eight columns of this thread's lane of tensor memory
OEQ_DEV void tcw_st(unsigned taddr, const float (&v)[8]) {
    asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};"
                 ::"r"(taddr), "f"(v[0]), "f"(v[1]), "f"(v[2]), "f"(v[3]), "f"(v[4]), "f"(v[5]), "f"(v[6]), "f"(v[7]) : "memory");
}
OEQ_DEV void tcw_ld(unsigned taddr, float (&r)[8]) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
                 : "=f"(r[0]), "=f"(r[1]), "=f"(r[2]), "=f"(r[3]), "=f"(r[4]), "=f"(r[5]), "=f"(r[6]), "=f"(r[7]) : "r"(taddr) : "memory");
    asm volatile("tcgen05.wait::ld.sync.aligned;" : "+f"(r[0]), "+f"(r[1]), "+f"(r[2]), "+f"(r[3]), "+f"(r[4]), "+f"(r[5]), "+f"(r[6]), "+f"(r[7]) :: "memory");
}

extern "C" __global__ void __launch_bounds__(TC_THREADS, 1) oeq_uvw_tc_backward_dw(const __grid_constant__ TcDwParams p) {
    extern __shared__ __align__(1024) unsigned char tc_smem_raw[];
    TcDwShared& sh = *reinterpret_cast<TcDwShared*>(tc_smem_raw);
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    if (tid == 0) {
        for (int s = 0; s < 2; ++s) {
            tc_mbar_init(&sh.xs_full[s], 1); tc_mbar_init(&sh.xs_empty[s], TCW_AW + 2);
            tc_mbar_init(&sh.cy_full[s], 2); tc_mbar_init(&sh.cy_empty[s], TCW_AW);
            tc_mbar_init(&sh.b_full[s], 2); tc_mbar_init(&sh.b_empty[s], 1);
        }
        for (int s = 0; s < TCW_NA; ++s) { tc_mbar_init(&sh.a_full[s], TCW_AW); tc_mbar_init(&sh.a_empty[s], 1); }
        tc_mbar_init(&sh.d_full, 1); tc_mbar_init(&sh.d_free, TCW_AW); tc_mbar_init(&sh.drain, 1);
        sh.abort_flag = sh.never = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], 512;" ::"r"(tc_smem_u32(&sh.tmem_base)) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const unsigned tmem = sh.tmem_base, tmem_a = tmem + 32 * TCW_MAX_GROUPS;
    const long long nunits = (p.batch + TCW_TILE - 1) / TCW_TILE * p.splits;
    // every role walks the same stages: f(unit's tile, its first group, group, half)
    auto walk = [&](auto&& f, auto&& end) -> bool {
        unsigned nunit = 0;
#pragma unroll 1
        for (long long unit = blockIdx.x; unit < nunits; unit += gridDim.x, ++nunit) {
            const long long tile = unit / p.splits;
            const int part = (int)(unit % p.splits), g0 = p.cut[part], g1 = p.cut[part + 1];
#pragma unroll 1
            for (int q = 2 * g0; q < 2 * g1; ++q)
                if (!f(tile, nunit, g0, q >> 1, q & 1)) return false;
            if (!end(tile, nunit, g0, g1)) return false;
        }
        return true;
    };
    auto nothing = [](long long, unsigned, int, int) -> bool { return true; };

    bool ok = true;
    if (warp < TCW_AW) {
        // ---- T
        const int slot = warp & 3, sub = warp >> 2;
        const unsigned ta = tmem_a + ((unsigned)(slot * 32) << 16) + 8u * (unsigned)sub;
        unsigned ns = 0, ring = 0, lap = 0;
        ok = walk(
            [&](long long, unsigned, int, int grp, int) -> bool {
                const int q = grp * 4 + slot, d = TCW_D1[q], d3 = TCW_D3[grp];   // (d = 0: no such slot)
                const unsigned buf = ns & 1u, par = (ns >> 1) & 1u;
                if (!tc_warp_wait(&sh.xs_full[buf], par, &sh.abort_flag)) return false;
                TcPair x[TCW_MAXD][4];
                const float* xb = sh.xg[buf] + TCW_BOX0[q] * 1024 + 8 * sub * 32;
#pragma unroll
                for (int i = 0; i < TCW_MAXD; ++i)
                    if (i < d) {
                        const int f = lane * d + i;
                        const float* at = xb + (f >> 5) * 1024 + (f & 31);
#pragma unroll
                        for (int e = 0; e < 4; ++e) asm("mov.b64 %0, {%1, %2};" : "=l"(x[i][e]) : "f"(at[64 * e]), "f"(at[64 * e + 32]));
                    }
                __syncwarp();
                if (lane == 0) tc_mbar_arrive(&sh.xs_empty[buf]);
                if (!tc_warp_wait(&sh.cy_full[buf], par, &sh.abort_flag)) return false;
#pragma unroll 1
                for (int k = 0; k < d3; ++k) {
                    if (lap > 0 && !tc_warp_wait(&sh.a_empty[ring], (lap - 1) & 1u, &sh.abort_flag)) return false;
                    if (d > 0) {
                        tc_fence_after();
                        TcPair t[4] = {0, 0, 0, 0};
                        tcw_cell<TcwMath>(TCW_CELL[q * 8 + k], x, sh.cy[buf] + TCW_PAIR0[q * 8 + k] * TCW_CYS + 8 * sub, t);
                        float hi[8], lo[8];
#pragma unroll
                        for (int e = 0; e < 8; ++e) {
                            const float v = tc_half(t[e >> 1], e & 1);
                            hi[e] = tc_tf32(v);
                            lo[e] = v - hi[e];   // (12 bits, of which the tensor core reads 11)
                        }
                        tcw_st(ta + 64u * ring, hi);
                        tcw_st(ta + 64u * ring + 32u, lo);
                        asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
                        tc_fence_before();
                    }
                    __syncwarp();
                    if (lane == 0) tc_mbar_arrive(&sh.a_full[ring]);
                    if (++ring == TCW_NA) { ring = 0; ++lap; }
                }
                if (lane == 0) tc_mbar_arrive(&sh.cy_empty[buf]);
                ++ns;
                return true;
            },
            [&](long long tile, unsigned nunit, int g0, int g1) -> bool {
                // the tile's sums: row `tile` of the partials matrix (lane = (slot, u), column = 32 * group + w)
                if (!tc_warp_wait(&sh.d_full, nunit & 1u, &sh.abort_flag)) return false;
                tc_fence_after();
                float* prow = p.part + tile * WN;
#pragma unroll 1
                for (int grp = g0; grp < g1; ++grp) {
                    if (TCW_D1[grp * 4 + slot] == 0) continue;
                    float r[8];
                    tcw_ld(tmem + ((unsigned)(slot * 32) << 16) + 32u * (unsigned)(grp - g0) + 8u * (unsigned)sub, r);
                    float4* dst = reinterpret_cast<float4*>(prow + TCW_WOFF[grp * 4 + slot] + lane * 32 + 8 * sub);
                    dst[0] = make_float4(r[0], r[1], r[2], r[3]);
                    dst[1] = make_float4(r[4], r[5], r[6], r[7]);
                }
                tc_fence_before();
                __syncwarp();
                if (lane == 0) tc_mbar_arrive(&sh.d_free);
                return true;
            });
    } else if (warp == TCW_AW) {
        // ---- MMAs
        const unsigned ud = __shfl_sync(0xffffffffu, tmem, 0), ua = ud + 32 * TCW_MAX_GROUPS;
        unsigned nc = 0, ring = 0, lap = 0;
        bool fresh = true;
        ok = walk(
            [&](long long, unsigned nunit, int g0, int grp, int half) -> bool {
                if (fresh && nunit > 0 && !tc_warp_wait(&sh.d_free, (nunit - 1) & 1u, &sh.abort_flag)) return false;
                fresh = false;
                const int d3 = TCW_D3[grp];
                const unsigned dcol = ud + 32u * (unsigned)(grp - g0);
#pragma unroll 1
                for (int k = 0; k < d3; ++k, ++nc) {
                    const unsigned bbuf = nc & 1u;
                    if (!tc_warp_wait(&sh.b_full[bbuf], (nc >> 1) & 1u, &sh.abort_flag)) return false;
                    if (!tc_warp_wait(&sh.a_full[ring], lap & 1u, &sh.abort_flag)) return false;
                    tc_fence_after();
                    const unsigned long long bh = tc_desc(sh.b[bbuf][0], TC_LBO, TC_SBO), bl = tc_desc(sh.b[bbuf][1], TC_LBO, TC_SBO);
                    const unsigned ah = ua + 64u * ring, al = ah + 32u, go_on = (half | k) != 0;   // every tile starts its sums afresh
#pragma unroll
                    for (int ks = 0; ks < 4; ++ks) {
                        tc_mma_ts(dcol, al + 8u * ks, bh + TC_LBO / 8ull * ks, TC_IDESC, ks == 0 ? go_on : 1u);
                        tc_mma_ts(dcol, ah + 8u * ks, bl + TC_LBO / 8ull * ks, TC_IDESC, 1u);
                    }
#pragma unroll
                    for (int ks = 0; ks < 4; ++ks) tc_mma_ts(dcol, ah + 8u * ks, bh + TC_LBO / 8ull * ks, TC_IDESC, 1u);
                    tc_commit_elected(&sh.a_empty[ring]);
                    tc_commit_elected(&sh.b_empty[bbuf]);
                    __syncwarp();
                    if (++ring == TCW_NA) { ring = 0; ++lap; }
                }
                return true;
            },
            [&](long long, unsigned, int, int) -> bool {
                tc_commit_elected(&sh.d_full);
                fresh = true;
                return true;
            });
        if (!ok) {   // given up: the MMAs in flight end before the tensor memory is freed
            if (lane == 0) tc_give_up(&sh.abort_flag, p.status, 61 + warp);
            __syncwarp();
            tc_commit_elected(&sh.drain);
            tc_mbar_wait(&sh.drain, 0u, &sh.never);
        }
    } else if (warp < TCW_AW + 3) {
        // ---- B: a lane is a channel of the output tile; a warp takes four of the stage's eight item quads
        const int w2 = warp - TCW_AW - 1;
        unsigned ns = 0, nc = 0;
        ok = walk(
            [&](long long, unsigned, int, int grp, int) -> bool {
                const int d3 = TCW_D3[grp];
                const unsigned buf = ns & 1u;
                if (!tc_warp_wait(&sh.xs_full[buf], (ns >> 1) & 1u, &sh.abort_flag)) return false;
                const float* gb = sh.xg[buf] + TCW_GBOX0[grp] * 1024 + 16 * w2 * 32;
#pragma unroll 1
                for (int k = 0; k < d3; ++k, ++nc) {
                    const unsigned bbuf = nc & 1u;
                    const int f = lane * d3 + k;
                    const float* at = gb + (f >> 5) * 1024 + (f & 31);
                    float v[16];
#pragma unroll
                    for (int e = 0; e < 16; ++e) v[e] = at[32 * e];
                    if (nc >= 2 && !tc_warp_wait(&sh.b_empty[bbuf], ((nc >> 1) - 1) & 1u, &sh.abort_flag)) return false;
#pragma unroll
                    for (int t = 0; t < 4; ++t) {
                        float hi[4], lo[4];
#pragma unroll
                        for (int e = 0; e < 4; ++e) { hi[e] = tc_tf32(v[4 * t + e]); lo[e] = v[4 * t + e] - hi[e]; }
                        const int to = (lane >> 3) * (TC_SBO / 4) + (4 * w2 + t) * (TC_LBO / 4) + (lane & 7) * 4;
                        *reinterpret_cast<float4*>(sh.b[bbuf][0] + to) = make_float4(hi[0], hi[1], hi[2], hi[3]);
                        *reinterpret_cast<float4*>(sh.b[bbuf][1] + to) = make_float4(lo[0], lo[1], lo[2], lo[3]);
                    }
                    tc_fence_async_smem();
                    __syncwarp();
                    if (lane == 0) tc_mbar_arrive(&sh.b_full[bbuf]);
                }
                if (lane == 0) tc_mbar_arrive(&sh.xs_empty[buf]);   // (its reads precede the last __syncwarp)
                ++ns;
                return true;
            },
            nothing);
    } else {
        // ---- boxes (the first of the two warps) and coefficients: a lane is a pair (i, k), whose terms it keeps for both halves, four items at a
        // time.  (With an item per lane the terms came one after the other from constant memory, 200 cycles a pair, and set the pace.)
        const int w2 = warp - TCW_AW - 3;
        constexpr int LD = L2_DIM | 1;
        float* ys = sh.ys[w2];
        unsigned ns = 0, nload = 0;   // stages, and those whose boxes are requested
        float tc[TCW_PPL][TCW_TERMS];
        int tj[TCW_PPL][TCW_TERMS];
        ok = walk(
            [&](long long tile, unsigned, int g0, int grp, int half) -> bool {
                const unsigned buf = ns & 1u;
                if (w2 == 0) {
                    if (ns >= 2 && !tc_warp_wait(&sh.xs_empty[buf], ((ns >> 1) - 1) & 1u, &sh.abort_flag)) return false;
                    const int nbox = TCW_NBOX[grp], gbox = TCW_GBOX0[grp];
                    if (lane == 0) tc_mbar_expect_tx(&sh.xs_full[buf], 4096u * (unsigned)nbox);
                    __syncwarp();
                    if (lane < nbox) tc_tile_load(sh.xg[buf] + lane * 1024, lane < gbox ? &p.x : &p.g, TCW_BOX[grp * 32 + lane], (int)(tile * TCW_TILE + 32 * half), &sh.xs_full[buf]);
                    ++nload;
                }
                if (grp == g0 && half == 0) {      // the tile's harmonics (no item: zeros, and T = 0)
                    __syncwarp();
#pragma unroll
                    for (int h = 0; h < 2; ++h) {
                        const long long b = tile * TCW_TILE + 32 * h + lane;
                        const bool live = b < p.batch;
#pragma unroll
                        for (int j = 0; j < L2_DIM; ++j) ys[(32 * h + lane) * LD + j] = live ? __ldg(p.y + b * L2_DIM + j) : 0.f;
                    }
                    __syncwarp();
                }
                const int p0 = TCW_CY0[grp], np = TCW_CY0[grp + 1] - p0;
                if (half == 0)
#pragma unroll
                    for (int r = 0; r < TCW_PPL; ++r) {
                        const int c = (2 * r + w2) * 32 + lane;
#pragma unroll
                        for (int t = 0; t < TCW_TERMS; ++t) {
                            tc[r][t] = c < np ? __ldg(TCW_PC + (p0 + c) * TCW_TERMS + t) : 0.f;
                            tj[r][t] = c < np ? __ldg(TCW_PJ + (p0 + c) * TCW_TERMS + t) : 0;
                        }
                    }
                if (ns >= 2 && !tc_warp_wait(&sh.cy_empty[buf], ((ns >> 1) - 1) & 1u, &sh.abort_flag)) return false;
#pragma unroll
                for (int r = 0; r < TCW_PPL; ++r) {
                    const int c = (2 * r + w2) * 32 + lane;
                    if (c < np) {
                        const float* yh = ys + 32 * half * LD;
                        float* to = sh.cy[buf] + c * TCW_CYS;
#pragma unroll 4
                        for (int e = 0; e < 32; e += 4) {
                            float v[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
                            for (int t = 0; t < TCW_TERMS; ++t)
#pragma unroll
                                for (int m = 0; m < 4; ++m) v[m] = fmaf(tc[r][t], yh[(e + m) * LD + tj[r][t]], v[m]);
                            *reinterpret_cast<float4*>(to + e) = make_float4(v[0], v[1], v[2], v[3]);
                        }
                    }
                }
                __syncwarp();
                if (lane == 0) tc_mbar_arrive(&sh.cy_full[buf]);
                ++ns;
                return true;
            },
            nothing);
        if (!ok && w2 == 0) {   // given up: the copies in flight end before the CTA does
            if (lane == 0) tc_give_up(&sh.abort_flag, p.status, 61 + warp);
            __syncwarp();
            for (unsigned s = nload > 2 ? nload - 2 : 0; s < nload; ++s) tc_mbar_wait(&sh.xs_full[s & 1u], (s >> 1) & 1u, &sh.never);
        }
    }
    if (!ok && lane == 0) tc_give_up(&sh.abort_flag, p.status, 61 + warp);
    tc_fence_before();
    __syncthreads();
    if (warp == 0) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, 512;" ::"r"(tmem) : "memory");
}
#endif  // TC_MODE == 3

#endif  // OEQ_TC
