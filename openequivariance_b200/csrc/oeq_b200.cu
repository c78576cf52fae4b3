// Host side of the oeq_b200 C ABI (declared in include/oeq_b200.h):
//   descriptor parser -> problem header emitter -> NVRTC (sm_100a) -> cubin cache -> launches.
//
// The device code lives in kernels/*.cuh (hand-written templates).  The only generated text is the short
// "problem header": constexpr tables for the irreps / instructions and one straight-line function per
// instruction holding its sparse Clebsch-Gordan contraction with the coefficients as literals.
//
// Counterparts in the reference: extension/backend/backend_cuda.hpp:154-361 (CUJITKernel: NVRTC, module
// load, launch), extension/tensorproducts.hpp:10-113 and extension/convolution.hpp:15-179 (kernel lists and
// launch sequences), extension/torch_core.hpp:180-270 (hash-keyed caches under a mutex).

#include <cuda.h>
#include <cuda_runtime.h>
#include <nvrtc.h>
#include <dlfcn.h>
#include <sys/stat.h>
#include <unistd.h>

#include <algorithm>
#include <atomic>
#include <cstdarg>
#include <cstdint>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <map>
#include <memory>
#include <mutex>
#include <set>
#include <tuple>
#include <sstream>
#include <string>
#include <vector>

#include "../../include/oeq_b200.h"
#include "dealing.h"
#include "kernels_embed.inc"  // generated at build time: K_COMMON, K_GENERIC, ... as raw strings
#include "graph_prep.cuh"         // problem-independent kernels: grouping / sorting of edge lists
#include "partition_plan.cuh"     // ... and the plans of the partitioned / streamed drivers
#include "group_mm.cuh"       // problem-independent kernels: ragged grouped products of the symmetric contraction
#include "sym_contraction.cuh"    // ... and the whole contraction in one pass

namespace {

// ------------------------------------------------------------------------------------------------ errors
thread_local std::string g_err;
std::atomic<long long> g_launches{0};
bool g_log = false;
bool g_force_generic = false;
bool g_no_tc = false;          // tuning aid: keep 'uvw' forward on the general kernel
int g_tc_backward = 7;         // 'uvw' backward outputs taken from the tensor-core kernels: 1 dx, 2 dy, 4 dW (bit mask)
bool g_single_group = false;   // tuning aid: one thread group per edge on the channel-parallel path
bool g_single_producer = false;   // tuning aid: one producer warp per CTA in the forward kernels too
int g_validate = 1;            // index checks of convolution calls: 0 never, 1 first call per edge list, 2 every call
bool g_streams_fwd = false;    // the forward kernels take part in `streams` too (the backward kernels always do)
int g_streams = 1;             // edge streams per CTA on the channel-parallel path (1: two CTAs per SM; 2-4: one CTA with
                               // that many consumer sets and a register hand-over; measured slower on the benchmark graph)
bool g_record = false;         // keep the names of the kernels that are launched (oeqb_launched_kernels)
std::string g_cache_dir;
std::mutex g_mutex;

int fail(int code, const char* fmt, ...) {
    char buf[4096];
    va_list ap;
    va_start(ap, fmt);
    vsnprintf(buf, sizeof buf, fmt, ap);
    va_end(ap);
    g_err = buf;
    if (g_log) fprintf(stderr, "[oeq_b200] error %d: %s\n", code, buf);
    return code;
}

#define CUDA_TRY(expr)                                                                              \
    do {                                                                                            \
        cudaError_t _e = (expr);                                                                    \
        if (_e != cudaSuccess) return fail(OEQB_ECUDA, "%s failed: %s", #expr, cudaGetErrorString(_e)); \
    } while (0)

// -------------------------------------------------------------------------------------------- descriptor
struct Block { int mul, l, p, off; int d() const { return 2 * l + 1; } };
struct Nz { int i, j, k; double c; };
struct Instr { int a, b, o; long long woff; std::vector<Nz> nz; };
// Distinct (i, k) index pairs of an instruction's Clebsch-Gordan nonzeros, sorted, each with the nonzeros (one per j)
// that share it.  The channel-parallel kernels fold the edge's y into one coefficient per pair.
struct IkPair { int i, k; std::vector<Nz> terms; };
std::vector<IkPair> ik_pairs(const Instr& I) {
    std::vector<Nz> v = I.nz;
    std::stable_sort(v.begin(), v.end(), [](const Nz& a, const Nz& b) { return a.i != b.i ? a.i < b.i : a.k < b.k; });
    std::vector<IkPair> out;
    for (const Nz& q : v) {
        if (out.empty() || out.back().i != q.i || out.back().k != q.k) out.push_back(IkPair{q.i, q.k, {}});
        out.back().terms.push_back(q);
    }
    return out;
}
struct TcPlan;
struct Desc {
    int dtype = 1, layout = 0, shared = 0, uvw = 0, conv = 0, det = 0, kahan = 0, idx = 4;
    std::vector<Block> L[3];
    long long dim[3] = {0, 0, 0};
    long long wn = 0;
    std::vector<Instr> ins;
    bool fast = false;   // channel-parallel pipelined kernels applicable
    int fast_U = 0;      // common multiplicity on the fast path
    int fast_S = 0;      // shared-memory stages per CTA
    int fast_ctas = 0;   // resident CTAs per SM the stages are sized for
    int fast_ncy = 0;    // folded-coefficient slots per edge (each instruction padded to a multiple of 4)
    int fast_ng = 1;     // thread groups sharing an edge
    int fast_ch = 1;     // channels carried by one consumer thread
    int fast_bwd_ng = 1; // thread groups of the backward kernels (2 in the fp64 configuration)
    int fastb_S = 0, fastb_ctas = 0;   // stages / resident CTAs of the first-order backward kernels (differ from the forward's
    size_t fastb_smem = 0;            // only for compensated summation, whose forward alone needs the wide configuration)
    size_t fast_smem = 0;
    bool tc = false;         // tensor-core 'uvw' forward applicable (shared weights, 32-wide multiplicities, fp32)
    bool tc_bwd = false;     // ... and the tensor-core backward kernels
    bool tc_zero_z = false, tc_zero_dx = false;   // some output / input block has no path: zero the result first
    int tc_ngrp = 0;         // groups of the tensor-core weight-gradient kernel (16 per launch)
    std::shared_ptr<const TcPlan> tc_plan[2];   // how the tensor-core kernels walk the problem: forward, gradients of x and y
    size_t tc_dw_smem = 0;   // dynamic shared memory of the tensor-core weight-gradient kernel
    int fast_S3 = 0;         // stages of the atomic forward kernel (it also holds one output row for the bulk reduce)
    size_t fast_smem3 = 0;
    int fast_S4 = 0;         // stages of the second-order kernels (their stage carries a second coefficient table)
    size_t fast_smem4 = 0;
    int fast_V = 1;          // edge streams per CTA of the first-order kernels (see kernels/fast_uvu.cuh); 1 = none
    int fast_SV = 0;         // stages per stream when fast_V > 1
    size_t fast_smemV = 0;
    bool item = false;       // 'uvw' with a weight row per item: one block per item (kernels/uvw_item.cuh)
    int f64mm = 0;           // 'uvw' in doubles on the FP64 matrix instruction: number of 32 x 32 weight tiles (0: not applicable)
    size_t elt() const { return dtype == 2 ? 8 : 4; }
};

std::vector<std::vector<int>> tc_dw_groups(const Desc& d);
size_t tc_dw_smem_bytes(const Desc& d);

// The tensor-core kernels of mode 0 (forward) and 1 (gradients of x and y): see kernels/uvw_tc.cuh for the words.
constexpr int kTcMaxParts = kMaxParts;
struct TcPlan {
    struct Visit { int src; std::vector<int> ins; };   // source block, instructions from it into the set (one weight tile each)
    struct Set {
        std::vector<int> dest, at;      // destination blocks and their first component's place
        int sumd = 0, code = 0;         // sets of the same code differ in where their blocks and weights lie
        std::vector<Visit> visits;
    };
    int tw = 32, nsub = 3, maxd = 1, nxs = 2;
    std::vector<Set> sets;                       // sets of several tiles first (ncset), then one per destination block
    int ncset = 0;
    std::vector<std::string> codes;              // ncode_coarse of the former sets, then of the latter
    int ncode_coarse = 0;
    std::vector<std::pair<int, int>> inst;       // (set, tile of its destination blocks' channels): ncoarse of the former, then of the latter
    int ncoarse = 0;
    size_t smem = 0;
    long long pairs = 0;                         // coefficients in the code of the former sets
    bool ok = false;
};
std::shared_ptr<const TcPlan> make_tc_plan(const Desc& d, int mode);

bool parse_desc(const char* text, size_t len, Desc& d, std::string& why) {
    std::istringstream in(std::string(text, len));
    std::string tok;
    auto bad = [&](const char* m) { why = m; return false; };
    int version = 0;
    if (!(in >> tok >> version) || tok != "OEQB" || version != 1) return bad("missing 'OEQB 1' header");
    std::string mode;
    if (!(in >> tok >> d.dtype) || tok != "dtype" || (d.dtype != 1 && d.dtype != 2)) return bad("bad dtype");
    if (!(in >> tok >> d.layout) || tok != "layout") return bad("bad layout");
    if (!(in >> tok >> d.shared) || tok != "shared") return bad("bad shared");
    if (!(in >> tok >> mode) || tok != "mode" || (mode != "uvu" && mode != "uvw")) return bad("bad mode");
    d.uvw = mode == "uvw";
    if (!(in >> tok >> d.conv >> d.det >> d.kahan >> d.idx) || tok != "conv" || (d.idx != 3 && d.idx != 4))
        return bad("bad conv line");
    const char* tags[3] = {"L1", "L2", "L3"};
    for (int r = 0; r < 3; ++r) {
        int n = 0;
        if (!(in >> tok >> n >> d.dim[r]) || tok != tags[r] || n < 0 || n > 4096) return bad("bad irreps header");
        long long off = 0;
        for (int b = 0; b < n; ++b) {
            Block blk{};
            if (!(in >> blk.mul >> blk.l >> blk.p >> blk.off) || blk.mul < 0 || blk.l < 0 || blk.l > 32)
                return bad("bad irreps block");
            if (blk.off != off) return bad("irreps offsets are not contiguous");
            off += (long long)blk.mul * blk.d();
            d.L[r].push_back(blk);
        }
        if (off != d.dim[r]) return bad("irreps dim mismatch");
    }
    if (!(in >> tok >> d.wn) || tok != "wn" || d.wn < 0) return bad("bad wn");
    int nins = 0;
    if (!(in >> tok >> nins) || tok != "ins" || nins <= 0 || nins > 65536) return bad("bad ins count");
    long long wsum = 0;
    for (int n = 0; n < nins; ++n) {
        Instr I{};
        int nnz = 0;
        if (!(in >> tok >> I.a >> I.b >> I.o >> I.woff >> nnz) || tok != "I") return bad("bad instruction line");
        if (I.a < 0 || I.a >= (int)d.L[0].size() || I.b < 0 || I.b >= (int)d.L[1].size() || I.o < 0 ||
            I.o >= (int)d.L[2].size() || nnz < 0)
            return bad("instruction index out of range");
        const Block &A = d.L[0][I.a], &B = d.L[1][I.b], &O = d.L[2][I.o];
        if (!d.uvw && A.mul != O.mul) return bad("uvu needs mul(in1) == mul(out)");
        if (I.woff != wsum) return bad("weight offsets are not contiguous");
        wsum += (long long)A.mul * B.mul * (d.uvw ? O.mul : 1);
        for (int z = 0; z < nnz; ++z) {
            Nz q{};
            std::string hex;
            if (!(in >> q.i >> q.j >> q.k >> hex)) return bad("bad CG entry");
            if (q.i < 0 || q.i >= A.d() || q.j < 0 || q.j >= B.d() || q.k < 0 || q.k >= O.d()) return bad("CG index out of range");
            q.c = strtod(hex.c_str(), nullptr);
            I.nz.push_back(q);
        }
        d.ins.push_back(std::move(I));
    }
    if (wsum != d.wn) return bad("weight_numel mismatch");
    if (!(in >> tok) || tok != "end") return bad("missing 'end'");
    if (d.layout == 1 && d.uvw) return bad("ir_mul layout with uvw");
    if (d.dim[0] * 1LL > (1LL << 24) || d.dim[2] > (1LL << 24) || d.wn > (1LL << 30)) return bad("problem too large");

    // Fast path: fp32 or fp64, either layout, uvu, per-item weights, every in2 multiplicity 1, one common in1 multiplicity
    // that is a multiple of 32, l <= 4 everywhere, rows small enough to live in registers; Kahan summation for the
    // deterministic convolution only (the only place the reference offers it).
    // fp64 takes the "wide" configuration: one channel per thread in two block-owning thread groups (forward and
    // backward), so that half a gradient row of doubles fits a thread's registers, and one CTA per SM for the doubled stages.
    d.fast = false;
    if ((d.dtype == 1 || d.dtype == 2) && !d.uvw && !d.shared && (!d.kahan || (d.conv && d.det && d.dtype == 1)) && !d.L[0].empty()) {
        // compensated summation also takes the wide configuration: sum and compensation of half a row per thread
        const bool wide = d.dtype == 2 || d.kahan;
        bool ok = true;
        int U = d.L[0][0].mul;
        for (auto& b : d.L[0]) ok = ok && b.mul == U && b.l <= 4;
        for (auto& b : d.L[1]) ok = ok && b.mul == 1 && b.l <= 4;
        for (auto& b : d.L[2]) ok = ok && b.mul == U && b.l <= 4;
        ok = ok && U >= 32 && U % 32 == 0 && U <= (wide ? 128 : 256) && d.dim[1] <= 32;
        ok = ok && d.dim[0] / U <= 32 && d.dim[2] / U <= 112;
        if (ok) {
            const size_t elt = d.elt();
            int ncy = 0;
            for (auto& I : d.ins) ncy += ((int)ik_pairs(I).size() + 3) & ~3;
            const int nyp = d.dim[1] <= 1 ? 1 : d.dim[1] <= 2 ? 2 : d.dim[1] <= 4 ? 4 : d.dim[1] <= 8 ? 8 : d.dim[1] <= 16 ? 16 : 32;
            // Two channels per thread halve the shared-memory traffic of the coefficient loads; the row registers
            // that doubles are won back by dealing the blocks to two thread groups.
            const int ch = (!wide && !g_single_group && U % 64 == 0 && d.ins.size() >= 2) ? 2 : 1;
            const int ng = (ch == 2 || (wide && d.ins.size() >= 2 && d.L[0].size() >= 2 && d.L[2].size() >= 2)) ? 2 : 1;
            const int bwd_ng = wide ? ng : 1;
            const int nthreads = std::max(ng * U / ch, bwd_ng * U);
            const size_t stage = ((elt * (size_t)(d.dim[0] + d.wn + ncy + ((d.dim[1] + 3) & ~3) + 8 + (nthreads / 32) * nyp) + 40) + 15) & ~(size_t)15;
            // Wide configuration: one CTA per SM where half a row of doubles (or of sums and compensations) fills the registers; rows of up to 32
            // components per channel leave room for several (96 registers, nothing spilled), which cover one another's latencies: 128x(0+1) in doubles,
            // 40,000 edges, forward 146 -> 109 us, backward 207 -> 177 us with two.
            const bool narrow = wide && d.dim[2] / U <= 32;
            int ctas = wide && !narrow ? 1 : 256 / U;
            ctas = ctas < 1 ? 1 : (ctas > 4 ? 4 : ctas);
            while (ctas > 1 && (narrow ? ctas * (nthreads + 64) * 96 : ctas * (nthreads + 32) * (ch == 2 ? 168 : 128)) > 65536) --ctas;   // registers per thread
            int S = 0;
            for (; ctas >= 1; ctas /= 2) {
                const size_t budget = 232448 / ctas - 1024 - 256;
                S = (int)(budget / (stage + 32));
                if (S > 6) S = 6;
                if (S >= 3) break;
            }
            if (S >= 3 && ctas >= 1 && nthreads + 64 <= 1024) {
                d.fast = true;
                d.fast_U = U; d.fast_S = S; d.fast_ctas = ctas; d.fast_ncy = ncy; d.fast_ng = ng; d.fast_ch = ch;
                d.fast_bwd_ng = bwd_ng;
                d.fast_smem = (size_t)S * (stage + 32) + 160;
                d.fastb_S = S; d.fastb_ctas = ctas; d.fastb_smem = d.fast_smem;
                if (d.kahan && d.dtype == 1) {
                    // Only the forward accumulates over edges; the backward kernel of the compensated variant is the plain one
                    // (one channel per thread, one group) in its own, denser configuration.
                    const int nthreads_b = U;
                    const size_t stage_b = ((elt * (size_t)(d.dim[0] + d.wn + ncy + ((d.dim[1] + 3) & ~3) + 8 + (nthreads_b / 32) * nyp) + 40) + 15) & ~(size_t)15;
                    int ctas_b = 256 / U;
                    ctas_b = ctas_b < 1 ? 1 : (ctas_b > 4 ? 4 : ctas_b);
                    while (ctas_b > 1 && ctas_b * (nthreads_b + 64) * 168 > 65536) --ctas_b;
                    int S_b = 0;
                    for (; ctas_b >= 1; ctas_b /= 2) {
                        S_b = (int)((232448 / ctas_b - 1024 - 256) / (stage_b + 32));
                        if (S_b > 6) S_b = 6;
                        if (S_b >= 3) break;
                    }
                    if (S_b >= 3 && ctas_b >= 1) {
                        d.fast_bwd_ng = 1; d.fastb_S = S_b; d.fastb_ctas = ctas_b; d.fastb_smem = (size_t)S_b * (stage_b + 32) + 160;
                    }
                }
                const size_t stage4 = stage + elt * (size_t)(ncy + ((d.dim[1] + 3) & ~3));
                int S4 = wide ? 0 : (int)((232448 / ctas - 1024 - 256) / (stage4 + 32));
                if (S4 > 6) S4 = 6;
                d.fast_S4 = S4;    // < 3: second-order passes run on the general kernels
                d.fast_smem4 = (size_t)S4 * (stage4 + 32) + 160;
                // Several edge streams in one CTA per SM: consumer sets of exactly one warpgroup, three stages each
                if (!wide && g_streams > 1 && g_streams <= 4 && nthreads == 128 && U == 128) {
                    const int V = g_streams;
                    int cyt = 1;
                    for (auto& I : d.ins)
                        for (auto& pr : ik_pairs(I)) cyt = std::max(cyt, (int)pr.terms.size());
                    const size_t table = (size_t)ncy * cyt * 8;   // consumer-side folding: (coefficient, index) pairs
                    int SV = (int)((((232448 - 1024 - table) / V) - 256) / (stage + 32));
                    if (SV > 4) SV = 4;
                    if (SV >= 3) { d.fast_V = V; d.fast_SV = SV; d.fast_smemV = (size_t)V * ((size_t)SV * (stage + 32) + 128 + 64) + table + 64; }
                }
                int S3 = wide ? 0 : (int)((232448 / ctas - 1024 - 256 - elt * (size_t)d.dim[2]) / (stage + 32));
                if (S3 > 6) S3 = 6;
                d.fast_S3 = S3;    // < 2: atomic forward falls back to the general kernel
                d.fast_smem3 = (size_t)(S3 > 0 ? S3 : 0) * (stage + 32) + elt * (size_t)d.dim[2] + 192;
            }
        }
    }
    // Tensor-core path for 'uvw': shared fp32 weights, every in1 / out multiplicity a multiple of 32 (up to 128: the weight
    // blocks are walked in 32 x 32 tiles), in2 multiplicity 1, l <= 3.
    d.tc = false;
    d.tc_bwd = false;
    if (d.dtype == 1 && d.layout == 0 && d.uvw && d.shared && !d.L[0].empty()) {
        bool ok = d.dim[1] <= 16;
        for (auto& b : d.L[0]) ok = ok && b.mul % 32 == 0 && b.mul <= 128 && b.l <= 3;
        for (auto& b : d.L[1]) ok = ok && b.mul == 1 && b.l <= 3;
        for (auto& b : d.L[2]) ok = ok && b.mul % 32 == 0 && b.mul <= 128 && b.l <= 3;
        // the kernels store only the blocks they accumulate: an output block without a path (or, for the gradient, an input
        // block that no path reads) is zeroed by the host first
        std::vector<int> hit(d.L[2].size(), 0), read(d.L[0].size(), 0);
        for (auto& I : d.ins) { hit[I.o] = 1; read[I.a] = 1; }
        d.tc_zero_z = d.tc_zero_dx = false;
        for (int h : hit) d.tc_zero_z = d.tc_zero_z || !h;
        for (int h : read) d.tc_zero_dx = d.tc_zero_dx || !h;
        long long npath = 0;   // 32 x 32 weight tiles: what the index tables and the weight gradient's partial rows grow with
        if (ok) for (auto& I : d.ins) npath += (long long)(d.L[0][I.a].mul / 32) * (d.L[2][I.o].mul / 32);
        ok = ok && npath <= 1024 && !d.ins.empty();
        // At most 1,280 products per output channel (and per input channel, for the gradients).  Accuracy does not ask for it: the tensor cores,
        // which add with truncation, sum 32 of them at a time.  It is how far the kernels are tested and how much code a program may
        // become (straight-line sums: 4 to 9 s to compile near the limit); wider problems run on the general kernels.
        if (ok) {
            std::vector<long long> into(d.L[2].size(), 0), from(d.L[0].size(), 0);
            for (auto& I : d.ins) { into[I.o] += d.L[0][I.a].mul; from[I.a] += d.L[2][I.o].mul; }
            for (long long v : into) ok = ok && v <= 1280;
            for (long long v : from) ok = ok && v <= 1280;
        }
        d.tc = ok;
        d.tc_bwd = ok;
        if (ok) for (int m = 0; m < 2; ++m) d.tc_plan[m] = make_tc_plan(d, m);
        d.tc = ok && d.tc_plan[0]->ok;
        d.tc_bwd = d.tc && d.tc_plan[1]->ok;
        if (d.tc_bwd) { d.tc_ngrp = (int)tc_dw_groups(d).size(); d.tc_dw_smem = tc_dw_smem_bytes(d); d.tc_bwd = d.tc_dw_smem <= 232448; }
    }
    // 'uvw' in doubles, shared weights: multiplicities that are multiples of 32 and in2 multiplicity 1, as on the tensor-core
    // path; l <= 3 for the accumulators' registers, and no more weight tiles than compile to a few hundred KB of code.
    d.f64mm = 0;
    if (d.dtype == 2 && d.layout == 0 && d.uvw && d.shared && !d.conv) {
        bool ok = d.dim[1] > 0 && d.dim[1] <= 16;
        for (auto& b : d.L[0]) ok = ok && b.mul > 0 && b.mul % 32 == 0 && b.l <= 3;
        for (auto& b : d.L[1]) ok = ok && b.mul == 1 && b.l <= 3;
        for (auto& b : d.L[2]) ok = ok && b.mul > 0 && b.mul % 32 == 0 && b.l <= 3;
        long long tiles = 0;
        if (ok) for (auto& I : d.ins) tiles += (long long)(d.L[0][I.a].mul / 32) * (d.L[2][I.o].mul / 32);
        if (ok && tiles <= 128) d.f64mm = (int)tiles;
    }
    // 'uvw' with per-item weights: a block per item with all intermediates in (static) shared memory, in2 multiplicity 1.
    d.item = false;
    if (d.uvw && !d.shared && !d.conv && d.layout == 0) {
        bool ok = d.dim[1] > 0 && d.dim[1] <= 32;
        for (auto& b : d.L[0]) ok = ok && b.mul > 0;
        for (auto& b : d.L[1]) ok = ok && b.mul == 1;
        for (auto& b : d.L[2]) ok = ok && b.mul > 0;
        size_t t = 0, g = 0;
        for (auto& I : d.ins) {
            const size_t n = (size_t)d.L[0][I.a].mul * d.L[2][I.o].d();
            t += n;
            g += n * ((d.L[2][I.o].mul + 31) / 32);
        }
        const size_t fwd = (size_t)d.dim[0] + d.dim[1] + t + 4 * (size_t)d.dim[2];
        const size_t bwd = (size_t)d.dim[0] + 6 * (size_t)d.dim[1] + d.dim[2] + t + g;
        d.item = ok && std::max(fwd, bwd) * d.elt() <= 48 * 1024 - 256;
    }
    return true;
}

// ------------------------------------------------------------------------------------------ header emit
std::string hexf(double v) {
    char b[64];
    snprintf(b, sizeof b, "%a", v);
    return b;
}

// Straight-line contraction  out[oidx] += c * (p[pidx] * q[qidx])  grouped so each product is formed once.
void emit_contraction(std::ostringstream& s, const char* name, const char* pn, const char* qn, const char* on,
                      const std::vector<Nz>& nz, int which /*0 fwd, 1 dx, 2 dy*/) {
    s << "  template <class R> static OEQ_DEV void " << name << "(const R* " << pn << ", const R* " << qn << ", R* "
      << on << ") {\n";
    struct E { int p, q, o; double c; };
    std::vector<E> es;
    for (auto& z : nz) {
        if (which == 0) es.push_back({z.i, z.j, z.k, z.c});        // t[k] += c x[i] y[j]
        else if (which == 1) es.push_back({z.j, z.k, z.i, z.c});   // dx[i] += c y[j] g[k]
        else es.push_back({z.i, z.k, z.j, z.c});                   // dy[j] += c x[i] g[k]
    }
    std::stable_sort(es.begin(), es.end(), [](const E& a, const E& b) { return a.p != b.p ? a.p < b.p : a.q < b.q; });
    for (size_t n = 0; n < es.size();) {
        size_t m = n;
        s << "    { const R pr = " << pn << "[" << es[n].p << "] * " << qn << "[" << es[n].q << "];";
        while (m < es.size() && es[m].p == es[n].p && es[m].q == es[n].q) {
            s << " " << on << "[" << es[m].o << "] += R(" << hexf(es[m].c) << ") * pr;";
            ++m;
        }
        s << " }\n";
        n = m;
    }
    s << "  }\n";
}

std::string emit_header(const Desc& d) {
    std::ostringstream s;
    s << "// problem header (generated from the descriptor)\n";
    s << "typedef " << (d.dtype == 2 ? "double" : "float") << " T;\n";
    s << "typedef " << (d.idx == 3 ? "int" : "long long") << " IDX;\n";
    s << "#define OEQ_SHARED_W " << d.shared << "\n#define OEQ_UVW " << d.uvw << "\n#define OEQ_IR_MUL " << d.layout
      << "\n#define OEQ_KAHAN " << d.kahan << "\n";
    s << "#define OEQ_DEV __device__ __forceinline__\n";
    s << "constexpr int L1_DIM = " << d.dim[0] << ", L2_DIM = " << d.dim[1] << ", L3_DIM = " << d.dim[2]
      << ", WN = " << d.wn << ", NINS = " << d.ins.size() << ", NB1 = " << d.L[0].size() << ", NB2 = " << d.L[1].size()
      << ", NB3 = " << d.L[2].size() << ";\n";
    for (int r = 0; r < 3; ++r) {
        s << "template <int B> struct Blk" << (r + 1) << ";\n";
        for (size_t b = 0; b < d.L[r].size(); ++b) {
            const Block& k = d.L[r][b];
            s << "template <> struct Blk" << (r + 1) << "<" << b << "> { static constexpr int MUL = " << k.mul
              << ", D = " << k.d() << ", OFF = " << k.off << "; };\n";
        }
    }
    s << "template <int I> struct Ins;\n";
    for (size_t n = 0; n < d.ins.size(); ++n) {
        const Instr& I = d.ins[n];
        const Block &A = d.L[0][I.a], &B = d.L[1][I.b], &O = d.L[2][I.o];
        s << "template <> struct Ins<" << n << "> {\n";
        s << "  static constexpr int A = " << I.a << ", B = " << I.b << ", O = " << I.o << ", WOFF = " << I.woff
          << ", U = " << A.mul << ", V = " << B.mul << ", WN_ = " << O.mul << ", D1 = " << A.d() << ", D2 = " << B.d()
          << ", D3 = " << O.d() << ", NNZ = " << I.nz.size() << ";\n";
        emit_contraction(s, "fwd", "x", "y", "t", I.nz, 0);
        emit_contraction(s, "dx", "y", "g", "dx", I.nz, 1);
        emit_contraction(s, "dy", "x", "g", "dy", I.nz, 2);
        s << "};\n";
    }
    return s.str();
}

// Tables and per-instruction register kernels for the channel-parallel family (kernels/fast_uvu.cuh).
// cy[i,k] = sum_j C[i,j,k] y[j] is formed once per edge by the producer warp; the consumer code below reads it as float4.
// Producer warps of a kernel with `stages` stages: two from four stages on (its look-ahead is then a multiple of two).
int fast_producers(int stages) { return (stages >= 4 && !g_single_producer) ? 2 : 1; }

std::string emit_fast(const Desc& d, int ch, int ng, bool dbl, int stages, size_t smem_bytes, int streams, int ctas) {
    std::ostringstream s;
    if (!d.fast) { s << "#define OEQ_FAST 0\n"; return s.str(); }
    s << "#define OEQ_FAST 1\n";
    // element type T comes from the problem header; T4 = four of them (16 or 32 bytes), oeq_fma = fused multiply-add on T
    s << "template <class R> struct OeqVec4;\ntemplate <> struct OeqVec4<float> { typedef float4 type; };\n"
         "template <> struct OeqVec4<double> { typedef double4 type; };\ntypedef OeqVec4<T>::type T4;\n"
         "OEQ_DEV T oeq_fma(T a, T b, T c) { return fma(a, b, c); }\n";
    s << "#define FAST_DBL " << (dbl ? 1 : 0) << "\n";
    s << "constexpr int FAST_V = " << streams << ";\n";
    s << "constexpr int FAST_NP = " << (streams > 1 ? 1 : fast_producers(stages)) << ";\n";
    s << "constexpr size_t FAST_SMEM_BYTES = " << smem_bytes << ";\n";
    s << "constexpr int FU = " << d.fast_U << ", NCY = " << d.fast_ncy << ", FAST_S = " << stages
      << ", FAST_CTAS = " << (streams > 1 ? 1 : ctas) << ", FAST_CH = " << ch << ", FAST_XPC = " << d.dim[0] / d.fast_U
      << ", FAST_GPC = " << d.dim[2] / d.fast_U << ";\n";
    // Folded-coefficient table: slot q of an edge holds sum_t FAST_CYC[q][t] * y[FAST_CYJ[q][t]], one slot per (i, k) pair
    std::ostringstream cyc, cyj;
    std::vector<int> cyoff;
    std::vector<std::vector<IkPair>> pairs;
    int off = 0, cyt = 1;
    for (auto& I : d.ins) {
        pairs.push_back(ik_pairs(I));
        for (auto& pr : pairs.back()) cyt = std::max(cyt, (int)pr.terms.size());
    }
    for (size_t n = 0; n < d.ins.size(); ++n) {
        cyoff.push_back(off);
        const int np = (int)pairs[n].size(), pad = (np + 3) & ~3;
        for (int q = 0; q < pad; ++q)
            for (int t = 0; t < cyt; ++t) {
                const bool real = q < np && t < (int)pairs[n][q].terms.size();
                cyc << "T(" << (real ? hexf(pairs[n][q].terms[t].c) : std::string("0.0")) << "), ";
                cyj << (real ? d.L[1][d.ins[n].b].off + pairs[n][q].terms[t].j : 0) << ", ";
            }
        off += pad;
    }
    s << "constexpr int FAST_CYT = " << cyt << ";\n";
    s << "__device__ const T FAST_CYC[NCY * FAST_CYT] = {" << cyc.str() << "};\n";
    s << "__device__ const int FAST_CYJ[NCY * FAST_CYT] = {" << cyj.str() << "};\n";
    s << "template <int I> struct FIns;\n";
    const char comp[4] = {'x', 'y', 'z', 'w'};
    for (size_t n = 0; n < d.ins.size(); ++n) {
        const Instr& I = d.ins[n];
        const Block &A = d.L[0][I.a], &B = d.L[1][I.b], &O = d.L[2][I.o];
        const std::vector<IkPair>& P = pairs[n];
        const int D1 = A.d(), D3 = O.d(), np = (int)P.size(), nq = (np + 3) / 4;
        auto C = [&](int z) { std::ostringstream t; t << "c" << (z / 4) << "." << comp[z % 4]; return t.str(); };
        s << "template <> struct FIns<" << n << "> {\n";
        s << "  static constexpr int A = " << I.a << ", OB = " << I.o << ", XO = " << A.off / d.fast_U << ", GO = " << O.off / d.fast_U << ", Y0 = " << B.off
          << ", CY4 = " << cyoff[n] / 4 << ", WOFF = " << I.woff << ", D1 = " << D1 << ", D3 = " << D3 << ";\n";
        // ---- forward: FAST_CH channels per thread share the coefficient loads
        s << "  static OEQ_DEV void fwd(const T* x, const T4* cy, const T* w, T* acc) {\n";
        for (int q = 0; q < nq; ++q) s << "    const T4 c" << q << " = cy[CY4 + " << q << "];\n";
        s << "#pragma unroll\n    for (int ch = 0; ch < FAST_CH; ++ch) {\n";
        s << "      const T* xc = x + ch * D1; T* ac = acc + ch * FAST_GPC; const T wc = w[ch];\n";
        if (D1 <= D3) {
            for (int i = 0; i < D1; ++i) s << "      const T xs" << i << " = wc * xc[" << i << "];\n";
            for (int z = 0; z < np; ++z)
                s << "      ac[" << P[z].k << "] = oeq_fma(" << C(z) << ", xs" << P[z].i << ", ac[" << P[z].k << "]);\n";
        } else {
            for (int k = 0; k < D3; ++k) s << "      T t" << k << " = T(0);\n";
            for (int z = 0; z < np; ++z)
                s << "      t" << P[z].k << " = oeq_fma(" << C(z) << ", xc[" << P[z].i << "], t" << P[z].k << ");\n";
            for (int k = 0; k < D3; ++k) s << "      ac[" << k << "] = oeq_fma(wc, t" << k << ", ac[" << k << "]);\n";
        }
        s << "    }\n  }\n";
        // ---- fused second-order forward: acc += cy(y) . (w x2 + w2 x) + cy(y2) . (w x)
        if (dbl) {
            s << "  static OEQ_DEV void fwd3(const T* x, const T* x2, const T4* cy, const T4* cyb, const T* w, const T* w2, T* acc) {\n";
            for (int q = 0; q < nq; ++q) s << "    const T4 c" << q << " = cy[CY4 + " << q << "]; const T4 b" << q << " = cyb[CY4 + " << q << "];\n";
            s << "#pragma unroll\n    for (int ch = 0; ch < FAST_CH; ++ch) {\n";
            s << "      const T* xc = x + ch * D1; const T* yc = x2 + ch * D1; T* ac = acc + ch * FAST_GPC; const T wc = w[ch]; const T vc = w2[ch];\n";
            for (int i = 0; i < D1; ++i)
                s << "      const T xa" << i << " = oeq_fma(vc, xc[" << i << "], wc * yc[" << i << "]); const T xb" << i << " = wc * xc[" << i << "];\n";
            auto Bc = [&](int z) { std::ostringstream t; t << "b" << (z / 4) << "." << comp[z % 4]; return t.str(); };
            for (int z = 0; z < np; ++z)
                s << "      ac[" << P[z].k << "] = oeq_fma(" << C(z) << ", xa" << P[z].i << ", oeq_fma(" << Bc(z) << ", xb" << P[z].i << ", ac[" << P[z].k << "]));\n";
            s << "    }\n  }\n";
        }
        // ---- backward
        const bool scale_g = D3 <= D1;
        const int nqv = scale_g ? D3 : D1;
        s << "  static OEQ_DEV void bwd(const T* x, const T* g, const T4* cy, const T* w, const T* wdx, T* dx, T* dy, T* dw) {\n";
        for (int q = 0; q < nq; ++q) s << "    const T4 c" << q << " = cy[CY4 + " << q << "];\n";
        s << "    T qv[FAST_CH][" << nqv << "];\n";
        s << "#pragma unroll\n    for (int ch = 0; ch < FAST_CH; ++ch) {\n";
        s << "      const T* xc = x + ch * D1; const T* gc = g + ch * FAST_GPC; T* dxc = dx + ch * D1; const T wc = w[ch]; const T wx = wdx[ch];\n";
        for (int i = 0; i < D1; ++i) s << "      T s" << i << " = T(0);\n";
        for (int z = 0; z < np; ++z)
            s << "      s" << P[z].i << " = oeq_fma(" << C(z) << ", gc[" << P[z].k << "], s" << P[z].i << ");\n";
        s << "      T dwv = T(0);\n";
        for (int i = 0; i < D1; ++i) {
            s << "      dwv = oeq_fma(xc[" << i << "], s" << i << ", dwv);\n";
            s << "      dxc[" << i << "] = oeq_fma(wx, s" << i << ", dxc[" << i << "]);\n";
        }
        s << "      dw[ch] = dwv;\n";
        for (int t = 0; t < nqv; ++t) s << "      qv[ch][" << t << "] = wc * " << (scale_g ? "gc" : "xc") << "[" << t << "];\n";
        s << "    }\n";
        // dY: products are summed over the thread's channels before the fixed coefficients are applied
        std::vector<Nz> byik = I.nz;
        std::stable_sort(byik.begin(), byik.end(), [](const Nz& a, const Nz& b) { return a.i != b.i ? a.i < b.i : a.k < b.k; });
        for (size_t z = 0; z < byik.size();) {
            size_t m = z;
            s << "    { T pr = T(0);\n#pragma unroll\n      for (int ch = 0; ch < FAST_CH; ++ch) pr = oeq_fma(";
            if (scale_g) s << "x[ch * D1 + " << byik[z].i << "], qv[ch][" << byik[z].k << "]";
            else s << "qv[ch][" << byik[z].i << "], g[ch * FAST_GPC + " << byik[z].k << "]";
            s << ", pr);\n     ";
            while (m < byik.size() && byik[m].i == byik[z].i && byik[m].k == byik[z].k) {
                s << " dy[" << byik[m].j << "] = oeq_fma(T(" << hexf(byik[m].c) << "), pr, dy[" << byik[m].j << "]);";
                ++m;
            }
            s << " }\n";
            z = m;
        }
        s << "  }\n";
        // ---- fused second-order backward: s = cy(y).g and t = cy(y2).g;  dx += w2 s + w t;  dW = x2.s + x.t;
        //      dy[j] += C (w x2 + w2 x)[i] g[k]
        if (dbl) {
            s << "  static OEQ_DEV void bwd3(const T* x, const T* x2, const T* g, const T4* cy, const T4* cyb, const T* w, const T* w2, T* dx, T* dy, T* dw) {\n";
            for (int q = 0; q < nq; ++q) s << "    const T4 c" << q << " = cy[CY4 + " << q << "]; const T4 b" << q << " = cyb[CY4 + " << q << "];\n";
            auto Bc = [&](int z) { std::ostringstream t; t << "b" << (z / 4) << "." << comp[z % 4]; return t.str(); };
            s << "    T qv[FAST_CH][" << D1 << "];\n";
            s << "#pragma unroll\n    for (int ch = 0; ch < FAST_CH; ++ch) {\n";
            s << "      const T* xc = x + ch * D1; const T* yc = x2 + ch * D1; const T* gc = g + ch * FAST_GPC; T* dxc = dx + ch * D1; const T wc = w[ch]; const T vc = w2[ch];\n";
            for (int i = 0; i < D1; ++i) s << "      T s" << i << " = T(0), t" << i << " = T(0);\n";
            for (int z = 0; z < np; ++z)
                s << "      s" << P[z].i << " = oeq_fma(" << C(z) << ", gc[" << P[z].k << "], s" << P[z].i << "); t" << P[z].i << " = oeq_fma("
                  << Bc(z) << ", gc[" << P[z].k << "], t" << P[z].i << ");\n";
            s << "      T dwv = T(0);\n";
            for (int i = 0; i < D1; ++i) {
                s << "      dwv = oeq_fma(yc[" << i << "], s" << i << ", oeq_fma(xc[" << i << "], t" << i << ", dwv));\n";
                s << "      dxc[" << i << "] = oeq_fma(vc, s" << i << ", oeq_fma(wc, t" << i << ", dxc[" << i << "]));\n";
                s << "      qv[ch][" << i << "] = oeq_fma(vc, xc[" << i << "], wc * yc[" << i << "]);\n";
            }
            s << "      dw[ch] = dwv;\n    }\n";
            for (size_t z = 0; z < byik.size();) {
                size_t m = z;
                s << "    { T pr = T(0);\n#pragma unroll\n      for (int ch = 0; ch < FAST_CH; ++ch) pr = oeq_fma(qv[ch][" << byik[z].i
                  << "], g[ch * FAST_GPC + " << byik[z].k << "], pr);\n     ";
                while (m < byik.size() && byik[m].i == byik[z].i && byik[m].k == byik[z].k) {
                    s << " dy[" << byik[m].j << "] = oeq_fma(T(" << hexf(byik[m].c) << "), pr, dy[" << byik[m].j << "]);";
                    ++m;
                }
                s << " }\n";
                z = m;
            }
            s << "  }\n";
        }
        s << "};\n";
    }
    // Thread groups: with FAST_NG = 2 two sets of FU threads share an edge.  Backward: input blocks are dealt to the
    // groups (longest-processing-time first on CG nonzeros) so every dX block has one writer; forward: output blocks.
    {
        const int nb1 = (int)d.L[0].size(), nb3 = (int)d.L[2].size();
        std::vector<long> cost1(nb1, 0), cost3(nb3, 0);
        for (auto& I : d.ins) { cost1[I.a] += (long)I.nz.size() + 4; cost3[I.o] += (long)I.nz.size() + 4; }
        auto deal = [ng](const std::vector<long>& cost) {
            std::vector<int> order(cost.size()), grp(cost.size(), 0);
            for (size_t i = 0; i < order.size(); ++i) order[i] = (int)i;
            std::stable_sort(order.begin(), order.end(), [&](int a, int b) { return cost[a] > cost[b]; });
            long load[2] = {0, 0};
            for (int b : order) { const int g = (ng < 2 || load[0] <= load[1]) ? 0 : 1; grp[b] = g; load[g] += cost[b]; }
            return grp;
        };
        const std::vector<int> g1 = deal(cost1), g3 = deal(cost3);
        auto list = [&](const char* name, const std::vector<int>& v) {
            s << "constexpr int " << name << "[" << (v.empty() ? 1 : v.size()) << "] = {";
            for (size_t i = 0; i < v.size(); ++i) s << v[i] << (i + 1 < v.size() ? ", " : "");
            if (v.empty()) s << "0";
            s << "};\n";
        };
        s << "constexpr int FAST_NG = " << ng << ";\n";
        list("FP_X_OWNER", g1);   // backward: group that owns (reads X of, writes dX of) each input block
        list("FP_Z_OWNER", g3);   // forward: group that owns (accumulates, writes) each output block
        std::vector<int> needx0(nb1, 0), needx1(nb1, 0), needg0(nb3, 0), needg1(nb3, 0), gf, gb;
        for (auto& I : d.ins) {
            (g3[I.o] == 0 ? needx0 : needx1)[I.a] = 1;   // the instruction's forward group reads input block a
            (g1[I.a] == 0 ? needg0 : needg1)[I.o] = 1;   // the instruction's backward group reads gradient block o
            gf.push_back(g3[I.o]);
            gb.push_back(g1[I.a]);
        }
        list("FP_FWD_NEEDS_X0", needx0); list("FP_FWD_NEEDS_X1", needx1);
        list("FP_BWD_NEEDS_G0", needg0); list("FP_BWD_NEEDS_G1", needg1);
        list("FP_INS_GF", gf); list("FP_INS_GB", gb);
    }
    return s.str();
}

// A path of the tensor-core kernels: one 32 x 32 tile of an instruction's weight block (multiplicities are multiples of
// 32; the kernel weight order keeps such a tile contiguous: kernels/common.cuh::widx_uvw).
struct TcSub { int ins, uc, wc; };
std::vector<TcSub> tc_subpaths(const Desc& d) {
    std::vector<TcSub> subs;
    for (size_t n = 0; n < d.ins.size(); ++n)
        for (int uc = 0; uc < d.L[0][d.ins[n].a].mul / 32; ++uc)
            for (int wc = 0; wc < d.L[2][d.ins[n].o].mul / 32; ++wc) subs.push_back({(int)n, uc, wc});
    return subs;
}
int tc_sub_woff(const Desc& d, const TcSub& t) { return d.ins[t.ins].woff + t.uc * 32 * d.L[2][d.ins[t.ins].o].mul + t.wc * 1024; }

std::string emit_tc_dw(const Desc& d);

// Source and destination of an instruction: blocks of (x, z), or of (g, dx) for the gradients.
int tc_src(const Instr& I, int mode) { return mode == 0 ? I.a : I.o; }
int tc_dst(const Instr& I, int mode) { return mode == 0 ? I.o : I.a; }

// The sums of one instruction's products, component c of its source, into a set: a statement for every (i, k) pair that it is part of.
std::string tc_fold_code(const Desc& d, const TcPlan::Set& t, int n, int mode, int c) {
    std::ostringstream s;
    const Instr& I = d.ins[n];
    const size_t slot = std::find(t.dest.begin(), t.dest.end(), tc_dst(I, mode)) - t.dest.begin();
    const int yoff = d.L[1][I.b].off;
    for (auto& pr : ik_pairs(I)) {
        if ((mode == 0 ? pr.i : pr.k) != c) continue;
        const int at = t.at[slot] + (mode == 0 ? pr.k : pr.i);
        s << "      { float c = float(" << hexf(pr.terms[0].c) << ") * y[" << yoff + pr.terms[0].j << "];";
        for (size_t e = 1; e < pr.terms.size(); ++e) s << " c = fmaf(float(" << hexf(pr.terms[e].c) << "), y[" << yoff + pr.terms[e].j << "], c);";
        s << " tc_axpy(c, u, z + " << at << " * TC_H);";
        if (mode == 1) {
            s << " const float t = tc_dot(x + " << at << " * TC_H, u);";
            for (auto& e : pr.terms) s << " dy[" << yoff + e.j << "] = fmaf(float(" << hexf(e.c) << "), t, dy[" << yoff + e.j << "]);";
        }
        s << " }\n";
    }
    return s.str();
}

// Deals the destination blocks to sets.  A thread keeps a set's sums (and in mode 1 the first input's values beside them) in registers: nine
// components of 16 channels in the forward, of 8 channels in the gradients.  Blocks go, the largest first, to the set in which they add
// the fewest chunks (components of source blocks to convert and multiply).
std::shared_ptr<const TcPlan> make_tc_plan(const Desc& d, int mode) {
    auto plan = std::make_shared<TcPlan>();
    TcPlan& p = *plan;
    const std::vector<Block>&S = d.L[mode == 0 ? 0 : 2], &D = d.L[mode == 0 ? 2 : 0];
    std::vector<int> used;
    for (size_t b = 0; b < D.size(); ++b)
        for (auto& I : d.ins)
            if (tc_dst(I, mode) == (int)b) { used.push_back((int)b); break; }
    for (auto& I : d.ins) p.maxd = std::max(p.maxd, S[tc_src(I, mode)].d());
    p.tw = mode == 1 ? 16 : 32;
    p.nsub = 96 / p.tw;
    const int cap = 9;
    auto fill = [&](TcPlan::Set& s) {
        s.at.clear(); s.sumd = 0; s.visits.clear();
        for (int b : s.dest) { s.at.push_back(s.sumd); s.sumd += D[b].d(); }
        for (size_t a = 0; a < S.size(); ++a) {
            std::vector<int> ins;
            for (size_t n = 0; n < d.ins.size(); ++n)
                if (tc_src(d.ins[n], mode) == (int)a && std::count(s.dest.begin(), s.dest.end(), tc_dst(d.ins[n], mode))) ins.push_back((int)n);
            for (size_t q = 0; q < ins.size(); q += p.nsub)
                s.visits.push_back({(int)a, std::vector<int>(ins.begin() + q, ins.begin() + std::min(ins.size(), q + p.nsub))});
        }
    };
    auto chunks = [&](const TcPlan::Set& s) {
        int n = 0;
        for (auto& v : s.visits) n += S[v.src].d() * (S[v.src].mul / 32);
        return n;
    };
    // A set's code: its blocks, visits and sums as text without offsets; blocks and visits are put into an order that does not depend on
    // where they lie, so that like sets have like codes.
    auto add_set = [&](std::vector<int> dest, int first_code) {
        TcPlan::Set s;
        std::stable_sort(dest.begin(), dest.end(), [&](int a, int b) { return D[a].d() < D[b].d(); });
        s.dest = dest;
        fill(s);
        std::vector<std::pair<std::string, TcPlan::Visit>> coded;
        for (auto& v : s.visits) {
            std::vector<std::pair<std::string, int>> subs;
            for (int n : v.ins) {
                subs.push_back({"", n});
                for (int c = 0; c < S[v.src].d(); ++c) subs.back().first += std::to_string(c) + "\n" + tc_fold_code(d, s, n, mode, c);
            }
            std::sort(subs.begin(), subs.end());
            std::ostringstream text;
            text << "D = " << S[v.src].d() << ", NU = " << S[v.src].mul / 32 << ", NSUB = " << subs.size() << "\n";
            v.ins.clear();
            for (auto& q : subs) { v.ins.push_back(q.second); text << q.first; }
            coded.push_back({text.str(), v});
        }
        std::stable_sort(coded.begin(), coded.end(), [](auto& a, auto& b) { return a.first < b.first; });
        std::string code;
        for (int b : s.dest) code += std::to_string(D[b].d()) + " ";
        s.visits.clear();
        for (auto& v : coded) { code += v.first; s.visits.push_back(v.second); }
        const auto known = std::find(p.codes.begin() + first_code, p.codes.end(), code);
        s.code = (int)(known - p.codes.begin());
        if (known == p.codes.end()) p.codes.push_back(code);
        p.sets.push_back(s);
        return (int)p.sets.size() - 1;
    };
    // tiles of the destination's channels that the same blocks have are walked by the same sets
    std::map<std::vector<int>, std::vector<int>> known;
    for (int wc = 0;; ++wc) {
        std::vector<int> blocks;
        for (int b : used) if (D[b].mul > wc * p.tw) blocks.push_back(b);
        if (blocks.empty()) break;
        std::vector<int>& ids = known[blocks];
        if (ids.empty()) {
            std::vector<int> order = blocks;
            std::stable_sort(order.begin(), order.end(), [&](int a, int b) { return D[a].d() > D[b].d(); });
            std::vector<TcPlan::Set> open;
            for (int b : order) {
                int best = -1, cost = 0;
                for (size_t k = 0; k < open.size(); ++k) {
                    if (open[k].sumd + D[b].d() > cap) continue;
                    TcPlan::Set t = open[k];
                    t.dest.push_back(b);
                    fill(t);
                    const int more = chunks(t) - chunks(open[k]);
                    if (best < 0 || more < cost || (more == cost && open[k].sumd < open[best].sumd)) { best = (int)k; cost = more; }
                }
                if (best < 0) { open.emplace_back(); best = (int)open.size() - 1; }
                open[best].dest.push_back(b);
                fill(open[best]);
            }
            for (auto& s : open) ids.push_back(add_set(s.dest, 0));
        }
        for (int id : ids) p.inst.push_back({id, wc});
    }
    p.ncset = (int)p.sets.size();
    p.ncoarse = (int)p.inst.size();
    p.ncode_coarse = (int)p.codes.size();
    for (int b : used) {
        const int id = add_set({b}, p.ncode_coarse);
        for (int wc = 0; wc * p.tw < D[b].mul; ++wc) p.inst.push_back({id, wc});
    }
    for (int k = 0, code = 0; k < p.ncset; ++k) {
        if (p.sets[k].code != code) continue;
        ++code;
        for (auto& v : p.sets[k].visits)
            for (int n : v.ins) p.pairs += (long long)ik_pairs(d.ins[n]).size();
    }
    // sizeof(TcShared), rounded up
    const size_t xs = 4 * (size_t)128 * 32 * p.maxd, fixed = 4 * (size_t)(4 * 96 * 36 + (mode == 1 ? 128 * (d.dim[1] | 1) : 4)) + 512;
    p.nxs = fixed + 2 * xs <= 232448 ? 2 : 1;
    // never less than half of an SM's shared memory: a CTA allocates all of the tensor memory, so only one may be resident
    p.smem = std::max<size_t>((fixed + p.nxs * xs + 1023) & ~(size_t)1023, 120 * 1024);
    // (straight-line code of ten or twenty instructions per coefficient, twice)
    p.ok = p.smem <= 232448 && p.pairs <= 4096;
    return plan;
}

// Index tables of a tensor-core program: in constant memory where they fit it (64 KB a program; a weight gradient with 512 weight tiles of 128
// channels passes that), else in global memory.
std::string emit_tables(const std::vector<std::pair<const char*, std::vector<long long>>>& tables) {
    size_t words = 0;
    for (auto& t : tables) words += std::max<size_t>(t.second.size(), 1);
    std::ostringstream s;
    for (auto& t : tables) {
        s << (words <= 15000 ? "__constant__ int " : "__device__ const int ") << t.first << "[" << std::max<size_t>(t.second.size(), 1) << "] = {";
        for (long long v : t.second) s << v << ", ";
        s << "};\n";
    }
    return s.str();
}

// Tables of the tensor-core kernels of mode 0 and 1 (kernels/uvw_tc.cuh), for the large sets or for the small ones; parts: for tiles that are dealt to
// several CTAs.
std::string emit_tc(const Desc& d, int mode, bool small, bool parts) {
    std::ostringstream s;
    if (!d.tc || (mode != 0 && !d.tc_bwd)) { s << "#define OEQ_TC 0\n"; return s.str(); }
    if (mode == 3) return emit_tc_dw(d);
    const TcPlan& p = *d.tc_plan[mode];
    const std::vector<Block>&S = d.L[mode == 0 ? 0 : 2], &D = d.L[mode == 0 ? 2 : 0];
    s << "#define OEQ_TC 1\n#define TC_MODE " << mode << "\n#define TC_PARTS " << (parts ? 1 : 0) << "\n#define TC_KERNEL_NAME "
      << (mode == 0 ? "oeq_uvw_tc_forward" : "oeq_uvw_tc_backward_dx") << (parts ? "_parts\n" : "\n");
    std::vector<long long> iset, iwc, sv, scode, soff, vd, voff, vnu, vnsub, vw, vws;
    size_t maxnb = 1;
    const size_t s0 = small ? p.ncset : 0, s1 = small ? p.sets.size() : p.ncset;
    for (size_t n = small ? p.ncoarse : 0; n < (small ? p.inst.size() : p.ncoarse); ++n) { iset.push_back(p.inst[n].first - s0); iwc.push_back(p.inst[n].second); }
    for (size_t k = s0; k < s1; ++k) maxnb = std::max(maxnb, p.sets[k].dest.size());
    s << "constexpr int TC_OUT_DIM = " << d.dim[mode == 0 ? 2 : 0] << ", TC_TW = " << p.tw << ", TC_NSUB = " << p.nsub << ", TC_MAXD = " << p.maxd
      << ", TC_NXS = " << p.nxs << ", TC_MAX_PARTS = " << kTcMaxParts << ", TC_MAXNB = " << maxnb << ", TC_NINST = " << iset.size() << ";\nconstexpr size_t TC_SMEM_BYTES = " << p.smem << ";\n";
    for (size_t k = s0; k < s1; ++k) {
        const TcPlan::Set& t = p.sets[k];
        sv.push_back((long long)vd.size());
        scode.push_back(t.code);
        for (size_t b = 0; b < maxnb; ++b) soff.push_back(b < t.dest.size() ? D[t.dest[b]].off : 0);
        for (auto& v : t.visits) {
            const Block& A = S[v.src];
            const int nsub = (int)v.ins.size();
            vd.push_back(A.d()); voff.push_back(A.off); vnu.push_back(A.mul / 32); vnsub.push_back(nsub);
            for (int q = 0; q < p.nsub; ++q) {
                const Instr& I = d.ins[v.ins[q < nsub ? q : 0]];
                vw.push_back(I.woff);
                vws.push_back(32LL * d.L[2][I.o].mul);   // a weight tile row (32 channels of the first input) further on
            }
        }
    }
    sv.push_back((long long)vd.size());
    s << emit_tables({{"TC_SET_CODE", scode}, {"TC_SET_OFF", soff}, {"TC_INST_SET", iset}, {"TC_INST_WC", iwc}, {"TC_SET_V", sv}, {"TC_V_D", vd},
                      {"TC_V_OFF", voff}, {"TC_V_NU", vnu}, {"TC_V_NSUB", vnsub}, {"TC_V_W", vw}, {"TC_V_WS", vws}});
    return s.str();
}

// The sets' sums: a function for each code, as text, because a compiler takes straight-line statements several times faster than the same
// unrolled from templates (52 paths of 32 x 32 with l <= 3: 21 s, and 6 s).
std::string emit_tc_sets(const Desc& d, int mode, bool small) {
    std::ostringstream s;
    const TcPlan& p = *d.tc_plan[mode];
    const std::vector<Block>&S = d.L[mode == 0 ? 0 : 2], &D = d.L[mode == 0 ? 2 : 0];
    std::vector<int> codes;
    for (size_t k = small ? p.ncset : 0; k < (small ? p.sets.size() : p.ncset); ++k) {
        const TcPlan::Set& t = p.sets[k];
        if (std::count(codes.begin(), codes.end(), t.code)) continue;
        codes.push_back(t.code);
        s << "OEQ_DEV bool tc_set_" << t.code << "(TC_SET_ARGS) {\n  TcPair z[" << t.sumd << " * TC_H], x[TC_MODE == 1 ? " << t.sumd << " * TC_H : 1];\n";
        auto rows = [&](const char* call, size_t b, const char* at, const char* v, const char* more) {
            s << "  " << call << "<" << D[t.dest[b]].d() << ">(" << at << " + row0 * TC_OUT_DIM + TC_SET_OFF[set * TC_MAXNB + " << b << "] + col * " << D[t.dest[b]].d()
              << ", live, " << v << " + " << t.at[b] << " * TC_H, lane" << more << ");\n";
        };
        if (mode == 1) for (size_t b = 0; b < t.dest.size(); ++b) rows("tc_rows_load", b, "p.x", "x", "");
        s << "#pragma unroll\n  for (int k = 0; k < " << t.sumd << " * TC_H; ++k) z[k] = 0;\n  bool ok = true;\n  TcPair u[TC_H];\n";
        for (auto& v : t.visits) {
            s << "#pragma unroll 1\n  for (int uc = 0; uc < " << S[v.src].mul / 32 << "; ++uc) {\n";
            for (int c = 0; c < S[v.src].d(); ++c) {
                s << "    if (ok) ok = tc_step(sh, nd, y);\n    if (ok) {\n";
                for (size_t q = 0; q < v.ins.size(); ++q) {
                    s << "      tc_products(tmem + (nd & 1u) * TC_DW + " << q << " * TC_TW, u);\n";
                    if (q + 1 == v.ins.size()) s << "      tc_step_done(sh, nd, lane);\n";
                    s << tc_fold_code(d, t, v.ins[q], mode, c);
                }
                s << "      ++nd;\n    }\n";
            }
            s << "  }\n";
        }
        s << "  if (!ok) return false;\n";
        for (size_t b = 0; b < t.dest.size(); ++b) rows("tc_rows_store", b, "p.dst", "z", ", p.accum != 0");
        s << "  return true;\n}\n";
    }
    s << "OEQ_DEV bool tc_sum_set(const int code, TC_SET_ARGS) {\n  bool ok = true;\n";
    for (int c : codes) s << "  if (code == " << c << ") ok = tc_set_" << c << "(TC_SET_PASS);\n";
    s << "  return ok;\n}\n";
    return s.str();
}

// Groups of the tensor-core weight-gradient kernel: weight tiles into one tile of an output block, at most four, and so many that their input
// blocks (boxes of 32 floats for each component) and the output block's are at most `cap` boxes; the largest first.  Indexes tc_subpaths(d).
std::vector<std::vector<int>> tc_dw_groups_of(const Desc& d, int cap) {
    const std::vector<TcSub> subs = tc_subpaths(d);
    std::vector<std::vector<int>> groups;
    for (size_t o = 0; o < d.L[2].size(); ++o)
        for (int wc = 0; wc < d.L[2][o].mul / 32; ++wc) {
            std::vector<int> mine;
            for (size_t q = 0; q < subs.size(); ++q)
                if (d.ins[subs[q].ins].o == (int)o && subs[q].wc == wc) mine.push_back((int)q);
            auto boxes = [&](int q) { return d.L[0][d.ins[subs[q].ins].a].d(); };
            std::stable_sort(mine.begin(), mine.end(), [&](int a, int b) { return boxes(a) > boxes(b); });
            std::vector<std::vector<int>> open;
            std::vector<int> used;
            for (int q : mine) {
                size_t k = 0;
                while (k < open.size() && (open[k].size() == 4 || used[k] + boxes(q) + d.L[2][o].d() > cap)) ++k;
                if (k == open.size()) { open.emplace_back(); used.push_back(0); }
                open[k].push_back(q);
                used[k] += boxes(q);
            }
            groups.insert(groups.end(), open.begin(), open.end());
        }
    return groups;
}
size_t tc_dw_smem_of(const Desc& d, const std::vector<std::vector<int>>& groups, int* boxes, int* pairs) {
    const std::vector<TcSub> subs = tc_subpaths(d);
    *boxes = 1; *pairs = 1;
    for (auto& grp : groups) {
        int nb = d.L[2][d.ins[subs[grp[0]].ins].o].d(), np = 0;
        for (int q : grp) { nb += d.L[0][d.ins[subs[q].ins].a].d(); np += (int)ik_pairs(d.ins[subs[q].ins]).size(); }
        *boxes = std::max(*boxes, nb); *pairs = std::max(*pairs, np);
    }
    // sizeof(TcDwShared), rounded up; more than half of an SM's shared memory (a CTA allocates all of the tensor memory)
    const size_t bytes = 4 * (size_t)(2 * *boxes * 1024 + 2 * 2 * 4 * 288 + 2 * *pairs * 36 + 2 * 64 * (d.dim[1] | 1)) + 512;
    return std::max<size_t>((bytes + 1023) & ~(size_t)1023, 120 * 1024);
}
std::vector<std::vector<int>> tc_dw_groups(const Desc& d) {
    int boxes, pairs;
    for (int cap = 23; cap > 14; --cap) {
        auto groups = tc_dw_groups_of(d, cap);
        if (tc_dw_smem_of(d, groups, &boxes, &pairs) <= 232448) return groups;
    }
    return tc_dw_groups_of(d, 14);   // (one block of seven components, four of one)
}
size_t tc_dw_smem_bytes(const Desc& d) {
    int boxes, pairs;
    return tc_dw_smem_of(d, tc_dw_groups(d), &boxes, &pairs);
}

// Tables of the tensor-core weight-gradient kernel, and the sums that make one component of T ("cells": which components of the input, in the
// order of the coefficients).
std::string emit_tc_dw(const Desc& d) {
    std::ostringstream s;
    s << "#define OEQ_TC 1\n#define TC_MODE 3\n";
    const std::vector<std::vector<int>> groups = tc_dw_groups(d);
    const std::vector<TcSub> subs = tc_subpaths(d);
    int boxes, pairs, maxd = 1;
    const size_t smem = tc_dw_smem_of(d, groups, &boxes, &pairs);
    std::vector<long long> d3s, d1s, box0, gbox0, nbox, box, woff, cell, pair0, cy0, pj;
    std::vector<double> pc;
    int terms = 1, npairs = 0;
    for (auto& I : d.ins) for (auto& pr : ik_pairs(I)) terms = std::max(terms, (int)pr.terms.size());
    std::vector<std::vector<int>> cells;
    for (auto& grp : groups) {
        const TcSub& first = subs[grp[0]];
        const Block& O = d.L[2][d.ins[first.ins].o];
        d3s.push_back(O.d());
        cy0.push_back(npairs);
        int nb = 0, np = 0;
        std::vector<long long> mine;
        for (int slot = 0; slot < 4; ++slot) {
            const bool used = slot < (int)grp.size();
            const TcSub* t = used ? &subs[grp[slot]] : nullptr;
            const Instr* I = used ? &d.ins[t->ins] : nullptr;
            const Block* A = used ? &d.L[0][I->a] : nullptr;
            d1s.push_back(used ? A->d() : 0); box0.push_back(nb); woff.push_back(used ? tc_sub_woff(d, *t) : 0);
            if (used) {
                for (int j = 0; j < A->d(); ++j) mine.push_back(A->off + t->uc * 32 * A->d() + 32 * j);
                nb += A->d();
                maxd = std::max(maxd, A->d());
            }
            for (int k = 0; k < 8; ++k) {
                std::vector<int> c;
                pair0.push_back(np);
                if (used)
                    for (auto& pr : ik_pairs(*I))
                        if (pr.k == k) {
                            c.push_back(pr.i);
                            for (int e = 0; e < terms; ++e) {
                                const bool real = e < (int)pr.terms.size();
                                // (padded with a harmonic that the pair has: one that is not finite stays in the pairs that it is part of)
                                pj.push_back(d.L[1][I->b].off + pr.terms[real ? e : 0].j);
                                pc.push_back(real ? pr.terms[e].c : 0.0);
                            }
                            ++np;
                            ++npairs;
                        }
                const auto known = std::find(cells.begin(), cells.end(), c);
                cell.push_back((long long)(known - cells.begin()));
                if (known == cells.end()) cells.push_back(c);
            }
        }
        gbox0.push_back(nb);
        for (int j = 0; j < O.d(); ++j) mine.push_back(O.off + first.wc * 32 * O.d() + 32 * j);
        nb += O.d();
        nbox.push_back(nb);
        mine.resize(32, 0);
        box.insert(box.end(), mine.begin(), mine.end());
    }
    cy0.push_back(npairs);
    s << "constexpr int TCW_BOXES = " << boxes << ", TCW_PAIRS = " << pairs << ", TCW_MAXD = " << maxd << ", TCW_TERMS = " << terms << ", TC_MAX_PARTS = " << kTcMaxParts
      << ";\nconstexpr size_t TC_SMEM_BYTES = " << smem << ";\n";
    s << emit_tables({{"TCW_D3", d3s}, {"TCW_D1", d1s}, {"TCW_BOX0", box0}, {"TCW_GBOX0", gbox0}, {"TCW_NBOX", nbox}, {"TCW_BOX", box}, {"TCW_WOFF", woff},
                      {"TCW_CELL", cell}, {"TCW_PAIR0", pair0}, {"TCW_CY0", cy0}});
    s << "__device__ const int TCW_PJ[" << std::max<size_t>(pj.size(), 1) << "] = {";
    for (size_t i = 0; i < pj.size(); ++i) s << pj[i] << ", ";
    s << "};\n__device__ const float TCW_PC[" << std::max<size_t>(pc.size(), 1) << "] = {";
    for (double c : pc) s << "float(" << hexf(c) << "), ";
    s << "};\ntemplate <class M> OEQ_DEV void tcw_cell(int cell, const typename M::P (&x)[TCW_MAXD][4], const float* cy, typename M::P (&t)[4]) {\n  switch (cell) {\n";
    for (size_t c = 0; c < cells.size(); ++c) {
        s << "    case " << c << ":";
        for (size_t n = 0; n < cells[c].size(); ++n) s << " M::step(x[" << cells[c][n] << "], cy + " << 36 * n << ", t);";
        s << " break;\n";
    }
    s << "  }\n}\n";
    return s.str();
}

// --------------------------------------------------------------------------------------- kernel families
enum Family {
    FAM_GENERIC = 0,
    FAM_FAST_FWD_TP, FAM_FAST_FWD_DET, FAM_FAST_FWD_ATOMIC, FAM_FAST_BWD_TP, FAM_FAST_BWD_DET, FAM_FAST_BWD_ATOMIC,
    FAM_FAST_SCATTER,
    FAM_FAST_BWD2_TP, FAM_FAST_BWD2_DET, FAM_FAST_BWD2_ATOMIC,   // second-order variants of the backward kernels
    FAM_UVW_TC,                                                  // tcgen05 'uvw' forward
    FAM_FAST_FWD3_TP, FAM_FAST_FWD3_DET,                         // fused second-order forward (three terms in one pass)
    FAM_UVW_TC_DX, FAM_UVW_TC_DW,                                // tcgen05 'uvw' backward: gradients of x and y, of the weights
    FAM_UVW_TC_PARTS, FAM_UVW_TC_DX_PARTS,                       // forward and gradients of x and y with a tile's large sets dealt to several CTAs
    FAM_UVW_TC_SMALL, FAM_UVW_TC_DX_SMALL,                       // ... its small sets
    FAM_UVW_ITEM,                                                // 'uvw' with a weight row per item
    FAM_UVW_F64,                                                 // 'uvw' in doubles on the FP64 matrix instruction
    FAM_DW_REDUCE,                                               // rows of partial sums -> gradient of shared weights
    FAM_COUNT
};
const char* const kFamilyNames[FAM_COUNT] = {"generic", "fast_fwd_tp", "fast_fwd_det", "fast_fwd_atomic", "fast_bwd_tp",
                                             "fast_bwd_det", "fast_bwd_atomic", "fast_scatter", "fast_bwd2_tp",
                                             "fast_bwd2_det", "fast_bwd2_atomic", "uvw_tc", "fast_fwd3_tp", "fast_fwd3_det",
                                             "uvw_tc_dx", "uvw_tc_dw", "uvw_tc_parts", "uvw_tc_dx_parts", "uvw_tc_small", "uvw_tc_dx_small", "uvw_item", "uvw_f64", "dw_reduce"};
const char* family_name(int f) { return (f >= 0 && f < FAM_COUNT) ? kFamilyNames[f] : "?"; }
int family_from_name(const std::string& n) {
    for (int f = 0; f < FAM_COUNT; ++f)
        if (n == kFamilyNames[f]) return f;
    if (n == "generic_forward" || n == "generic_backward") return FAM_GENERIC;
    return -1;
}

// Edge streams per CTA for a kernel family: the first-order kernels except the atomic forward (whose staged output
// row leaves no room for three rings); 1 when the problem or the caller rules them out.
int family_streams(const Desc& d, int fam, bool allow) {
    const bool eligible = ((fam == FAM_FAST_FWD_TP || fam == FAM_FAST_FWD_DET) && g_streams_fwd) || fam == FAM_FAST_BWD_TP ||
                          fam == FAM_FAST_BWD_DET || fam == FAM_FAST_BWD_ATOMIC;
    return (allow && eligible && d.fast && d.fast_V > 1) ? d.fast_V : 1;
}

// Elements per access to a weight row: the largest power of two up to 16 bytes that divides the row and every offset in it.
int item_vec(const Desc& d) {
    int v = (int)(16 / d.elt());
    auto divides = [&](int v) {
        for (auto& I : d.ins) if (I.woff % v) return false;
        return d.wn % v == 0;
    };
    while (v > 1 && !divides(v)) v /= 2;
    return v;
}

// Shared memory for an item's weight row, 0: not staged.  Beside a row of 40 KB, the largest, two blocks fit an SM where the static arrays
// are near their limit (48 KB), five where they are small.
size_t item_row_bytes(const Desc& d) {
    const size_t b = (size_t)d.wn * d.elt();
    return b <= 40 * 1024 ? b : 0;
}

std::string family_source(const Desc& d, const std::string& header, int fam, bool allow_streams = true) {
    if (fam == FAM_DW_REDUCE) return std::string("typedef ") + (d.dtype == 2 ? "double" : "float") + " T;\nconstexpr int WN = " + std::to_string(d.wn) + ";\n" + K_DW_REDUCE;
    std::string src = header;
    if (fam == FAM_GENERIC) {
        src += K_COMMON;
        src += K_GENERIC;
    } else if (fam == FAM_UVW_ITEM) {
        src += "constexpr int ITEM_VEC = " + std::to_string(item_vec(d)) + ";\n#define ITEM_STAGE_W " + (item_row_bytes(d) ? "1\n" : "0\n");
        src += K_COMMON;
        src += K_UVW_ITEM;
    } else if (fam == FAM_UVW_F64) {
        src += K_COMMON;
        src += K_UVW_F64;
    } else if (fam == FAM_UVW_TC || (fam >= FAM_UVW_TC_DX && fam <= FAM_UVW_TC_DX_SMALL)) {
        const int mode = fam == FAM_UVW_TC_DW ? 3 : fam == FAM_UVW_TC_DX || fam == FAM_UVW_TC_DX_PARTS || fam == FAM_UVW_TC_DX_SMALL ? 1 : 0;
        const bool small = fam == FAM_UVW_TC_SMALL || fam == FAM_UVW_TC_DX_SMALL;
        src += emit_tc(d, mode, small, fam >= FAM_UVW_TC_PARTS);
        src += K_COMMON;
        static const std::string kernel = K_UVW_TC, here = "//@ sets\n";   // (where the emitted functions go: behind what they call)
        const size_t at = kernel.find(here);
        src += kernel.substr(0, at);
        if (mode == 0 ? d.tc : mode == 1 && d.tc_bwd) src += emit_tc_sets(d, mode, small);
        src += kernel.substr(at + here.size());
    } else {
        // Forward kernels carry two channels per thread in two block-owning groups (their code is small enough to stay
        // in the instruction cache); the backward kernels, three times larger, keep one channel per thread and one
        // code stream, which measured faster than the split variants (those stalled on instruction fetch).
        const bool fwd3 = fam == FAM_FAST_FWD3_TP || fam == FAM_FAST_FWD3_DET;
        const bool fwd = fwd3 || (fam >= FAM_FAST_FWD_TP && fam <= FAM_FAST_FWD_ATOMIC);
        const bool dbl = fwd3 || (fam >= FAM_FAST_BWD2_TP && fam <= FAM_FAST_BWD2_ATOMIC);
        const int V = family_streams(d, fam, allow_streams);
        const bool bwd1 = !fwd && !dbl;   // first-order backward: its own stage count and residency
        const int stages = V > 1 ? d.fast_SV : dbl ? d.fast_S4 : (fam == FAM_FAST_FWD_ATOMIC ? d.fast_S3 : bwd1 ? d.fastb_S : d.fast_S);
        const size_t smem = V > 1 ? d.fast_smemV : dbl ? d.fast_smem4 : (fam == FAM_FAST_FWD_ATOMIC ? d.fast_smem3 : bwd1 ? d.fastb_smem : d.fast_smem);
        src += emit_fast(d, fwd ? d.fast_ch : 1, fwd ? d.fast_ng : d.fast_bwd_ng, dbl, stages, smem, V, bwd1 ? d.fastb_ctas : d.fast_ctas);
        // the second-order variants reuse the backward entry points (kernel ids 3..5)
        src += "#define FAST_KERNEL " + std::to_string(fwd3 ? fam - FAM_FAST_FWD3_TP : dbl ? fam - FAM_FAST_BWD2_TP + 3 : fam - FAM_FAST_FWD_TP) + "\n";
        src += K_COMMON;   // (FAST_KERNEL is defined before the kernel file: it sizes the shared-memory layout)
        src += K_FAST_UVU;
    }
    return src;
}

// -------------------------------------------------------------------------------------- NVRTC + caching
uint64_t fnv1a(const std::string& s) {
    uint64_t h = 1469598103934665603ull;
    for (unsigned char c : s) { h ^= c; h *= 1099511628211ull; }
    return h;
}

std::string default_cache_dir() {
    if (const char* e = getenv("OEQB_CACHE_DIR")) return e;
    Dl_info info;
    if (dladdr((void*)&default_cache_dir, &info) && info.dli_fname) {
        std::string p = info.dli_fname;
        size_t slash = p.find_last_of('/');
        if (slash != std::string::npos) return p.substr(0, slash) + "/_cubin_cache";
    }
    return "/tmp/oeq_b200_cubin_cache";
}

std::mutex g_cache_mutex;   // of the name: not every compilation holds g_mutex
std::string cache_dir() {
    std::lock_guard<std::mutex> lock(g_cache_mutex);
    if (g_cache_dir.empty()) g_cache_dir = default_cache_dir();
    return g_cache_dir;
}
void set_cache_dir(const char* dir) {
    std::lock_guard<std::mutex> lock(g_cache_mutex);
    g_cache_dir = dir;
}

bool read_file(const std::string& path, std::string& out) {
    FILE* f = fopen(path.c_str(), "rb");
    if (!f) return false;
    fseek(f, 0, SEEK_END);
    long n = ftell(f);
    fseek(f, 0, SEEK_SET);
    out.resize(n > 0 ? n : 0);
    size_t got = n > 0 ? fread(&out[0], 1, n, f) : 0;
    fclose(f);
    return got == (size_t)(n > 0 ? n : 0) && n > 0;
}

void write_file_atomic(const std::string& path, const std::string& data) {
    mkdir(cache_dir().c_str(), 0755);
    std::string tmp = path + ".tmp" + std::to_string((long long)getpid());
    FILE* f = fopen(tmp.c_str(), "wb");
    if (!f) return;
    size_t put = fwrite(data.data(), 1, data.size(), f);
    fclose(f);
    if (put == data.size()) rename(tmp.c_str(), path.c_str()); else remove(tmp.c_str());
}

// Compiles `src` for sm_100a; returns the cubin (from the disk cache when present).
// *from_cache (optional) receives the cache file's path when the cubin was read from it, "" when it was compiled now.
int compile_cubin(const std::string& src, const char* label, std::string& cubin, std::string* from_cache = nullptr) {
    if (from_cache) from_cache->clear();
    static const char* opts[] = {"--gpu-architecture=sm_100a", "--std=c++17", "-lineinfo", "-default-device",
                                 "--extra-device-vectorization"};
    const int nopts = sizeof(opts) / sizeof(opts[0]);
    int major = 0, minor = 0;
    nvrtcVersion(&major, &minor);
    std::string keytext = src;
    for (int i = 0; i < nopts; ++i) keytext += opts[i];
    keytext += std::to_string(major * 100 + minor);
    char name[64];
    snprintf(name, sizeof name, "/%016llx.cubin", (unsigned long long)fnv1a(keytext));
    const std::string path = cache_dir() + name;
    if (read_file(path, cubin)) {
        if (g_log) fprintf(stderr, "[oeq_b200] %s: cubin cache hit %s\n", label, path.c_str());
        if (from_cache) *from_cache = path;
        return OEQB_OK;
    }
    nvrtcProgram prog;
    nvrtcResult r = nvrtcCreateProgram(&prog, src.c_str(), label, 0, nullptr, nullptr);
    if (r != NVRTC_SUCCESS) return fail(OEQB_ECOMPILE, "nvrtcCreateProgram: %s", nvrtcGetErrorString(r));
    r = nvrtcCompileProgram(prog, nopts, opts);
    if (r != NVRTC_SUCCESS) {
        size_t ls = 0;
        nvrtcGetProgramLogSize(prog, &ls);
        std::string log(ls, '\0');
        if (ls) nvrtcGetProgramLog(prog, &log[0]);
        nvrtcDestroyProgram(&prog);
        if (log.size() > 3500) log.resize(3500);
        return fail(OEQB_ECOMPILE, "NVRTC failed for %s: %s\n%s", label, nvrtcGetErrorString(r), log.c_str());
    }
    size_t cs = 0;
    nvrtcGetCUBINSize(prog, &cs);
    cubin.resize(cs);
    nvrtcGetCUBIN(prog, &cubin[0]);
    nvrtcDestroyProgram(&prog);
    write_file_atomic(path, cubin);
    if (g_log) fprintf(stderr, "[oeq_b200] %s: compiled %zu bytes of cubin\n", label, cs);
    return OEQB_OK;
}

struct Program {
    cudaLibrary_t lib = nullptr;
    std::map<std::string, cudaKernel_t> kernels;
    std::map<std::string, int> smem_set;  // kernel -> bitmask of devices whose smem attribute was raised
    std::string cubin;                    // kept alive for lazy per-context loading
    bool regs_ok = false;                 // tensor-core kernels: register count verified against the hand-over scheme
    bool regs_checked = false;            // multi-stream kernels: the same
};

struct Entry {
    Desc d;
    uint64_t desc_hash = 0;     // of the descriptor text this entry was built from: a key reused for another problem is refused
    size_t desc_len = 0;
    const void* seen_ptr = nullptr;   // last caller buffer whose contents were compared (callers pass the same buffer again)
    std::string header;
    std::unique_ptr<Program> prog[FAM_COUNT];
    std::unique_ptr<Cuts> tc_cuts[5];                     // how the tensor-core kernels' work is cut: large and small sets of mode 0, of mode 1, dW
    std::unique_ptr<Program> prog_single[FAM_COUNT];   // the same families built with one edge stream per CTA
    bool tc_off = false;                                // a tensor-core program did not compile to what the host expects
    bool streams_off = false;                           // a multi-stream kernel came out with the wrong register count
};

std::map<int64_t, std::unique_ptr<Entry>> g_entries;

// Caller holds g_mutex.
int get_entry(const void* desc, size_t len, int64_t key, Entry** out) {
    auto it = g_entries.find(key);
    if (it != g_entries.end()) {
        Entry* have = it->second.get();
        if (desc && len > 0 && !(desc == have->seen_ptr && len == have->desc_len)) {
            if (len != have->desc_len || fnv1a(std::string((const char*)desc, len)) != have->desc_hash)
                return fail(OEQB_EINVAL, "key %lld was first used with a different descriptor: keys must identify one problem",
                            (long long)key);
            have->seen_ptr = desc;
        }
        *out = have;
        return OEQB_OK;
    }
    if (!desc || len == 0) return fail(OEQB_EINVAL, "descriptor is empty");
    auto e = std::make_unique<Entry>();
    e->desc_hash = fnv1a(std::string((const char*)desc, len));
    e->desc_len = len;
    e->seen_ptr = desc;
    std::string why;
    if (!parse_desc((const char*)desc, len, e->d, why)) return fail(OEQB_EPARSE, "descriptor: %s", why.c_str());
    e->header = emit_header(e->d);
    *out = e.get();
    g_entries[key] = std::move(e);
    return OEQB_OK;
}

// Compiles (or takes from the cubin cache) and loads one program.
int load_program(const std::string& src, const char* label, Program* p) {
    std::string cache_path;
    int rc = compile_cubin(src, label, p->cubin, &cache_path);
    if (rc) return rc;
    cudaError_t ce = cudaLibraryLoadData(&p->lib, p->cubin.data(), nullptr, nullptr, 0, nullptr, nullptr, 0);
    if (ce != cudaSuccess && !cache_path.empty()) {
        // a truncated or foreign file in the cache: drop it and compile afresh, once
        cudaGetLastError();
        remove(cache_path.c_str());
        if (g_log) fprintf(stderr, "[oeq_b200] %s: cached cubin %s did not load (%s); recompiling\n", label, cache_path.c_str(),
                           cudaGetErrorString(ce));
        if ((rc = compile_cubin(src, label, p->cubin, nullptr))) return rc;
        ce = cudaLibraryLoadData(&p->lib, p->cubin.data(), nullptr, nullptr, 0, nullptr, nullptr, 0);
    }
    if (ce != cudaSuccess) {
        cudaGetLastError();
        return fail(OEQB_ECOMPILE, "cudaLibraryLoadData(%s): %s", label, cudaGetErrorString(ce));
    }
    return OEQB_OK;
}

// Held by a thread that compiles without g_mutex: threads that want new programs wait for one another, so that each is compiled once.
std::mutex g_compile_mutex;

// As get_program, but `lock` (on g_mutex, held) is left while the program compiles: the other operators of the process go on.  An entry lasts as long
// as the process and its description does not change.
int program_off_lock(std::unique_lock<std::mutex>& lock, Entry* e, int fam) {
    if (e->prog[fam]) return OEQB_OK;
    lock.unlock();
    std::lock_guard<std::mutex> compiling(g_compile_mutex);
    lock.lock();
    if (e->prog[fam]) return OEQB_OK;
    lock.unlock();
    auto fresh = std::make_unique<Program>();
    const int rc = load_program(family_source(e->d, e->header, fam), family_name(fam), fresh.get());
    lock.lock();
    if (!rc && !e->prog[fam]) e->prog[fam] = std::move(fresh);   // (get_program may have compiled it meanwhile)
    return rc;
}

// Caller holds g_mutex.
int get_program(Entry* e, int fam, Program** out, bool allow_streams = true) {
    std::unique_ptr<Program>& slot = allow_streams ? e->prog[fam] : e->prog_single[fam];
    if (slot) { *out = slot.get(); return OEQB_OK; }
    auto p = std::make_unique<Program>();
    if (int rc = load_program(family_source(e->d, e->header, fam, allow_streams), family_name(fam), p.get())) return rc;
    *out = p.get();
    slot = std::move(p);
    return OEQB_OK;
}

std::map<cudaKernel_t, std::string> g_kernel_names;   // of the specialised kernels (guarded by g_mutex, as what follows)
std::set<std::string> g_recorded;                     // those launched since the option "record" was set

// Caller holds g_mutex.
int get_kernel(Program* p, const char* name, size_t smem, cudaKernel_t* out) {
    auto it = p->kernels.find(name);
    if (it == p->kernels.end()) {
        cudaKernel_t k;
        cudaError_t ce = cudaLibraryGetKernel(&k, p->lib, name);
        if (ce != cudaSuccess) {
            cudaGetLastError();   // (not for the next caller to find: this problem may be served by other kernels)
            return fail(OEQB_ECOMPILE, "kernel %s not found: %s", name, cudaGetErrorString(ce));
        }
        it = p->kernels.emplace(name, k).first;
        g_kernel_names[k] = name;
    }
    if (smem > 48 * 1024) {
        int dev = 0;
        CUDA_TRY(cudaGetDevice(&dev));
        int& mask = p->smem_set[name];
        if (!(mask & (1 << dev))) {
            CUDA_TRY(cudaFuncSetAttribute((const void*)it->second, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
            mask |= 1 << dev;
        }
    }
    *out = it->second;
    return OEQB_OK;
}

int launch(cudaKernel_t k, dim3 grid, unsigned block, size_t smem, void** args, cudaStream_t st) {
    const auto name = g_kernel_names.find(k);
    cudaError_t ce = cudaLaunchKernel((const void*)k, grid, dim3(block), args, smem, st);
    if (ce != cudaSuccess) return fail(OEQB_ECUDA, "launch of %s failed: %s", name != g_kernel_names.end() ? name->second.c_str() : "a kernel", cudaGetErrorString(ce));
    g_launches.fetch_add(1, std::memory_order_relaxed);
    if (g_record && name != g_kernel_names.end()) g_recorded.insert(name->second);
    return OEQB_OK;
}

int sm_count() {
    static int cached[64] = {0};
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return 148;
    if (!cached[dev]) {
        int n = 0;
        if (cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || n <= 0) n = 148;
        cached[dev] = n;
    }
    return cached[dev];
}

// ------------------------------------------------------------------------------------------ generic path
struct FwdParams {
    const void* x; const void* y; const void* W; void* z;
    const void* rows; const void* cols;
    long long n_units; long long n_edges;
    int unit_mode; int out_mode;
};
struct BwdParams {
    const void* x; const void* y_dx; const void* y_dw; const void* W; const void* g;
    void* dx; void* dy; void* dW;
    const void* rows; const void* cols; const void* perm;
    long long n_units; long long n_edges;
    int unit_mode; int accum;
    void* dW_part;
};
enum { UNIT_ITEM = 0, UNIT_EDGE = 1, UNIT_SEGMENT = 2 };
enum { OUT_STORE = 0, OUT_ADD = 1, OUT_ATOMIC = 2 };

unsigned generic_grid(long long units) {
    long long want = (units + 3) / 4;  // 4 warps per block
    long long cap = (long long)sm_count() * 16;
    if (want < 1) want = 1;
    return (unsigned)(want < cap ? want : cap);
}

int generic_forward(Entry* e, FwdParams p, cudaStream_t st) {
    if (p.n_units <= 0) return OEQB_OK;
    Program* prog;
    int rc = get_program(e, FAM_GENERIC, &prog);
    if (rc) return rc;
    cudaKernel_t k;
    if ((rc = get_kernel(prog, "oeq_generic_forward", 0, &k))) return rc;
    void* args[] = {&p};
    return launch(k, generic_grid(p.n_units), 128, 0, args, st);
}

int keep_pool_memory();

// dW (+)= the rows of partial sums, in order
int dw_reduce(Entry* e, const void* part, long long rows, void* dW, int accum, cudaStream_t st) {
    Program* prog;
    cudaKernel_t k;
    if (int rc = get_program(e, FAM_DW_REDUCE, &prog)) return rc;
    if (int rc = get_kernel(prog, "oeq_generic_dw_reduce", 0, &k)) return rc;
    void* args[] = {&part, &rows, &dW, &accum};
    return launch(k, (unsigned)((e->d.wn + 31) / 32), 256, 0, args, st);
}

int generic_backward(Entry* e, BwdParams p, cudaStream_t st) {
    if (p.n_units <= 0) return OEQB_OK;
    Program* prog;
    int rc = get_program(e, FAM_GENERIC, &prog);
    if (rc) return rc;
    if (e->d.shared && p.unit_mode != UNIT_SEGMENT) {
        // shared weights: path-major kernel that sums dW over a chunk of items in registers and stores the chunk's sums
        // as one row of a partials matrix; a second kernel adds the rows in chunk order, so dW is bitwise reproducible
        // (the chunking does not depend on the grid).  The matrix lives in stream-ordered scratch for the call.
        // The kernel adds to dX, so for the tensor product dX has to start at zero (the convolution zeroes it anyway).
        const Desc& d = e->d;
        if (p.unit_mode == UNIT_ITEM && !p.accum)
            CUDA_TRY(cudaMemsetAsync(p.dx, 0, (size_t)p.n_edges * d.dim[0] * d.elt(), st));
        cudaKernel_t ks;
        if ((rc = get_kernel(prog, "oeq_generic_backward_shared", 0, &ks))) return rc;
        int chunk = 32;
        long long chunks = (p.n_edges + chunk - 1) / chunk;
        void* part = nullptr;
        if ((rc = keep_pool_memory())) return rc;
        CUDA_TRY(cudaMallocAsync(&part, (size_t)chunks * d.wn * d.elt(), st));
        p.dW_part = part;
        void* args[] = {&p, &chunk};
        rc = launch(ks, generic_grid(chunks), 128, 0, args, st);
        // the entry points zero dW before the first pass, so the reduce always adds to what is there
        if (!rc) rc = dw_reduce(e, part, chunks, p.dW, 1, st);
        cudaFreeAsync(part, st);
        return rc;
    }
    cudaKernel_t k;
    if ((rc = get_kernel(prog, "oeq_generic_backward", 0, &k))) return rc;
    void* args[] = {&p};
    return launch(k, generic_grid(p.n_units), 128, 0, args, st);
}

// ------------------------------------------------------------------------------- 'uvw' with a weight row per item
// Where a block per item pays.  It has a fixed price (three or four barriers, four warps that start and end together: 1 to 2 ns an
// item on a full chip), and the general kernel, a warp per item, has none.  In the forward pass that kernel's time goes with the number
// of weight tile rows it walks (25 to 40 ps each); in the backward pass with the weights, whose gradients it stores strided, and with
// the paths.  Few items leave the chip empty, and four warps then finish an item sooner than one.  Measured over 1 to 23 paths,
// multiplicities 1 to 128, 500 to 200,000 items, us, general / block (same results from both):
//   forward   4 paths 8 x 8, 100,000 items 73 / 163;    4 paths 32 x 8 216 / 175;     11 paths 16 x 16 419 / 433;   11 paths 32 x 32, 10,000 items 122 / 92
//   backward  1 path 8 x 8, 100,000 items 71 / 159;     4 paths 8 x 8 244 / 202;      11 paths 1 x 1 322 / 247;     1 path 8 x 8, 5,000 items 9.4 / 9.1
// The lines below are within 1.6 of the faster kernel wherever they take the block, and within 2.3 (10 to 20 us calls) where they do not.
bool item_forward_pays(const Desc& d, long long batch) {
    if (!d.item || g_force_generic) return false;
    size_t rows = 0;
    for (auto& I : d.ins) rows += d.L[0][I.a].mul;
    return batch <= 600 || rows >= (d.dtype == 2 ? 24 + 4 * d.ins.size() : 48 + 8 * d.ins.size());
}
bool item_backward_pays(const Desc& d, long long batch) {
    return d.item && !g_force_generic && (batch <= 4800 || d.ins.size() >= 8 || d.wn >= (d.dtype == 2 ? 512 : 256));
}

struct ItemFwdParams {
    const void* x; const void* y; const void* W; void* z;
    long long items;
    int add;
};
struct ItemBwdParams {
    const void* x; const void* y_dx; const void* y_dw; const void* W; const void* g;
    void* dx; void* dy; void* dW;
    long long items;
    int add;
};
int item_launch(Entry* e, const char* name, size_t row, void* params, long long items, cudaStream_t st) {
    Program* prog;
    if (int rc = get_program(e, FAM_UVW_ITEM, &prog)) return rc;
    cudaKernel_t k;
    // (the kernels' static arrays and the row together may exceed 48 KB: the attribute is then needed whatever the row alone takes)
    if (int rc = get_kernel(prog, name, row ? std::max<size_t>(row, 48 * 1024 + 16) : 0, &k)) return rc;
    void* args[] = {params};
    return launch(k, (unsigned)std::min<long long>(items, 1 << 30), 128, row, args, st);
}
int item_forward(Entry* e, const void* x, const void* y, const void* W, void* z, long long items, int add, cudaStream_t st) {
    ItemFwdParams p{x, y, W, z, items, add};
    return item_launch(e, "oeq_uvw_item_forward", 0, &p, items, st);
}
int item_backward(Entry* e, const void* x, const void* y_dx, const void* y_dw, const void* W, const void* g, void* dx, void* dy,
                  void* dW, long long items, int add, cudaStream_t st) {
    ItemBwdParams p{x, y_dx, y_dw, W, g, dx, dy, dW, items, add};
    return item_launch(e, "oeq_uvw_item_backward", item_row_bytes(e->d), &p, items, st);
}

// ------------------------------------------------------------------------------- 'uvw' in doubles, shared weights
struct F64FwdParams { const void* x; const void* y; const void* W; void* z; long long batch; int accum; };
struct F64BwdParams { const void* x; const void* y; const void* W; const void* g; void* dx; void* dy; long long batch; int accum; };
struct F64DwParams { const void* x; const void* y; const void* g; void* part; long long batch; int chunk; };
int f64_launch(Entry* e, const char* name, dim3 grid, void* params, cudaStream_t st) {
    Program* prog;
    if (int rc = get_program(e, FAM_UVW_F64, &prog)) return rc;
    cudaKernel_t k;
    if (int rc = get_kernel(prog, name, 0, &k)) return rc;
    void* args[] = {params};
    return launch(k, grid, 128, 0, args, st);
}
int f64_forward(Entry* e, const void* x, const void* y, const void* W, void* z, long long batch, int accum, cudaStream_t st) {
    int tiles = 0;
    for (auto& b : e->d.L[2]) tiles += b.mul / 32;
    F64FwdParams p{x, y, W, z, batch, accum};
    return f64_launch(e, "oeq_uvw_f64_forward", dim3((unsigned)((batch + 31) / 32), (unsigned)tiles), &p, st);
}
// dW is added to (the caller zeroes it); dx and dy are stored, or added to with accum
int f64_backward(Entry* e, const void* x, const void* y_dx, const void* y_dw, const void* W, const void* g, void* dx, void* dy,
                 void* dW, long long batch, int accum, cudaStream_t st) {
    const Desc& d = e->d;
    F64BwdParams p{x, y_dx, W, g, dx, dy, batch, accum};
    int rc = f64_launch(e, "oeq_uvw_f64_backward", dim3((unsigned)((batch + 7) / 8)), &p, st);
    if (rc) return rc;
    // Items per row of partial sums, by the batch alone (so results do not depend on the device): about 80 rows keep the chip
    // busy with few paths, and a row costs wn doubles written and read once.
    int chunk = (int)std::min<long long>(std::max<long long>((batch + 79) / 80, 16), 4096);
    chunk = (chunk + 3) & ~3;
    long long chunks = (batch + chunk - 1) / chunk;
    if ((rc = keep_pool_memory())) return rc;
    void* part = nullptr;
    CUDA_TRY(cudaMallocAsync(&part, (size_t)chunks * d.wn * sizeof(double), st));
    F64DwParams q{x, y_dw, g, part, batch, chunk};
    rc = f64_launch(e, "oeq_uvw_f64_backward_dw", dim3((unsigned)chunks, (unsigned)((d.f64mm + 3) / 4)), &q, st);
    if (!rc) rc = dw_reduce(e, part, chunks, dW, 1, st);
    cudaFreeAsync(part, st);
    return rc;
}

// ------------------------------------------------------------------------------- channel-parallel path
struct FastParams {
    const void* X; const void* Y; const void* W; const void* G;
    void* Z; void* dX; void* dY; void* dW; void* scratch;
    const void* rows; const void* cols;
    long long N; long long E;
    int* status;
    int accum;         // forward kernels: add to the output rows instead of overwriting them
    int pad;
    const void* X2; const void* Y2; const void* W2;   // fused second-order forward
    const void* eorder;                               // unsorted edge lists: position -> edge id, grouped by receiver
};

constexpr size_t kAlign = 256;
size_t round_up(size_t v) { return (v + kAlign - 1) / kAlign * kAlign; }

// One host-mapped status word per device: kernels store a non-zero code when a bounded wait runs out.
int* g_status_host[64] = {nullptr};
int* g_status_dev[64] = {nullptr};

int status_word(int** dev_ptr) {
    int dev = 0;
    CUDA_TRY(cudaGetDevice(&dev));
    if (dev < 0 || dev >= 64) return fail(OEQB_EINVAL, "device index %d out of range", dev);
    if (!g_status_host[dev]) {
        int* h = nullptr;
        CUDA_TRY(cudaHostAlloc((void**)&h, 64, cudaHostAllocMapped));
        memset(h, 0, 64);
        int* dptr = nullptr;
        CUDA_TRY(cudaHostGetDevicePointer((void**)&dptr, h, 0));
        g_status_host[dev] = h;
        g_status_dev[dev] = dptr;
    }
    const int code = *(volatile int*)g_status_host[dev];
    if (code != 0) {
        *(volatile int*)g_status_host[dev] = 0;
        if (code == gprep::STATUS_BAD_INDEX)
            return fail(OEQB_EINVAL, "an earlier call was given an index array (rows / cols / transpose_perm, or the nodes' elements) with a "
                                     "value out of range, or a receiver list that is not sorted; its outputs are invalid");
        if (code == symc::STATUS_CHANGED)
            return fail(OEQB_EINVAL, "a captured symmetric contraction was replayed with other coupling tensors than it was captured "
                                     "with; its outputs are invalid: capture it again");
        return fail(OEQB_EKERNEL, "an earlier kernel gave up a bounded wait (code %d); its outputs are invalid", code);
    }
    if (dev_ptr) *dev_ptr = g_status_dev[dev];
    return OEQB_OK;
}

// Groups an unsorted edge list by receiver into ws (layout: [order: E indices][scratch of the grouping]); *order receives
// the position -> edge id list.  Returns OEQB_OK, or a negative number when the workspace is too small (the caller then
// takes the path that needs none).
size_t atomic_order_bytes(const Desc& d, long long N, long long E) {
    return round_up((size_t)(E > 0 ? E : 1) * (d.idx == 3 ? 4 : 8)) + gprep::group_workspace_bytes(N, E);
}
int group_by_receiver(const Desc& d, long long N, long long E, const void* rows, void* ws, long long ws_bytes,
                      cudaStream_t st, const void** order) {
    if (!ws || ws_bytes < (long long)atomic_order_bytes(d, N, E) || ((uintptr_t)ws & 15u)) return -1;
    int* status = nullptr;
    if (int rc = status_word(&status)) return rc;
    void* scratch = (char*)ws + round_up((size_t)E * (d.idx == 3 ? 4 : 8));
    long long launches = 0;
    bool ok;
    if (d.idx == 3) ok = gprep::group_by_key<int>((const int*)rows, nullptr, E, N, (int*)ws, nullptr, nullptr, scratch, status, st, nullptr, &launches);
    else ok = gprep::group_by_key<long long>((const long long*)rows, nullptr, E, N, (long long*)ws, nullptr, nullptr, scratch, status, st, nullptr, &launches);
    g_launches.fetch_add(launches, std::memory_order_relaxed);
    if (!ok) return fail(OEQB_ECUDA, "grouping the edge list by receiver failed: %s", cudaGetErrorString(cudaGetLastError()));
    *order = ws;
    return OEQB_OK;
}

bool aligned16(std::initializer_list<const void*> ptrs) {
    for (const void* p : ptrs)
        if (((uintptr_t)p & 15u) != 0) return false;
    return true;
}

bool use_fast(const Desc& d) { return d.fast && !g_force_generic; }


// kernel: 0 fwd_tp, 1 fwd_det, 2 fwd_atomic, 3 bwd_tp, 4 bwd_det, 5 bwd_atomic
int fast_launch(Entry* e, int kernel, FastParams p, cudaStream_t st, int* status_override = nullptr, bool dbl = false) {
    static const char* names1[6] = {"oeq_fast_forward_tp", "oeq_fast_forward_det", "oeq_fast_forward_atomic",
                                    "oeq_fast_backward_tp", "oeq_fast_backward_det", "oeq_fast_backward_atomic"};
    static const char* names2[6] = {"oeq_fast_double_backward_A_tp", "oeq_fast_double_backward_A_det", "",
                                    "oeq_fast_double_backward_B_tp", "oeq_fast_double_backward_B_det",
                                    "oeq_fast_double_backward_B_atomic"};
    const char* const* names = dbl ? names2 : names1;
    const Desc& d = e->d;
    int rc;
    if (status_override) p.status = status_override;
    else if ((rc = status_word(&p.status))) return rc;
    Program* prog;
    const bool fwd3 = dbl && kernel < 2;   // fused second-order forward (batch and sorted-convolution variants)
    const int fam = fwd3 ? FAM_FAST_FWD3_TP + kernel : dbl ? FAM_FAST_BWD2_TP + (kernel - 3) : FAM_FAST_FWD_TP + kernel;
    cudaKernel_t k;
    int V = family_streams(d, fam, !e->streams_off);
    if (V > 1) {
        // One CTA per SM with V consumer warpgroups and a producer warpgroup that hands registers over (setmaxnreg).
        // The hand-over only balances when the launch allocates exactly 65536 / threads registers per thread: a kernel
        // compiled to anything else is not used (its consumers would wait for registers that are never released).
        if ((rc = get_program(e, fam, &prog, true))) return rc;
        if ((rc = get_kernel(prog, names[kernel], d.fast_smemV, &k))) return rc;
        if (!prog->regs_checked) {
            cudaFuncAttributes attr;
            CUDA_TRY(cudaFuncGetAttributes(&attr, (const void*)k));
            const int threads = V * 128 + 128, want = 65536 / threads / 8 * 8;
            prog->regs_checked = true;
            if (attr.numRegs != want || attr.maxThreadsPerBlock < threads) {
                if (g_log) fprintf(stderr, "[oeq_b200] %s: multi-stream kernel has %d registers (%d needed); using the "
                                           "two-CTA variant\n", family_name(fam), attr.numRegs, want);
                e->streams_off = true;
                V = 1;
            }
        }
    }
    if (V > 1) {
        long long grid = sm_count();
        const long long work = ((p.E > 0 ? p.E : 1) + V - 1) / V;
        if (grid > work) grid = work;
        void* args[] = {&p};
        return launch(k, (unsigned)grid, (unsigned)(V * 128 + 128), d.fast_smemV, args, st);
    }
    const bool bwd1 = kernel >= 3 && !dbl;   // first-order backward: its own stage count and residency
    const size_t smem = dbl ? d.fast_smem4 : (kernel == 2 ? d.fast_smem3 : bwd1 ? d.fastb_smem : d.fast_smem);
    if ((rc = get_program(e, fam, &prog, false))) return rc;
    if ((rc = get_kernel(prog, names[kernel], smem, &k))) return rc;
    long long grid = (long long)sm_count() * (bwd1 ? d.fastb_ctas : d.fast_ctas);
    const long long work = p.E > 0 ? p.E : 1;
    if (grid > work) grid = work;
    void* args[] = {&p};
    const unsigned consumers = kernel < 3 ? (unsigned)(d.fast_ng * d.fast_U / d.fast_ch) : (unsigned)(d.fast_bwd_ng * d.fast_U);
    const int producers = fast_producers(dbl ? d.fast_S4 : (kernel == 2 ? d.fast_S3 : bwd1 ? d.fastb_S : d.fast_S));
    return launch(k, (unsigned)grid, consumers + 32 * producers, smem, args, st);
}

// dX[c] = sum of the per-edge rows in scratch over the sender's edges, in sender-major list order.  Two steps: the sender
// offsets (once), then the row sums for a range of senders [c_begin, c_end).
int fast_scatter_offsets(Entry* e, const void* cols, const void* perm, long long N, long long E, void* colptr, cudaStream_t st) {
    int rc;
    Program* prog;
    if ((rc = get_program(e, FAM_FAST_SCATTER, &prog))) return rc;
    cudaKernel_t k1;
    if ((rc = get_kernel(prog, "oeq_fixup_backward_offsets", 0, &k1))) return rc;
    void* args[] = {(void*)&cols, (void*)&perm, &E, &N, &colptr};
    return launch(k1, (unsigned)((E + 1 + 255) / 256), 256, 0, args, st);
}

int fast_scatter_rows(Entry* e, const void* scratch, const void* perm, const void* colptr, long long c_begin, long long c_end,
                      void* dX, cudaStream_t st) {
    if (c_end <= c_begin) return OEQB_OK;
    int rc;
    Program* prog;
    if ((rc = get_program(e, FAM_FAST_SCATTER, &prog))) return rc;
    cudaKernel_t k2;
    if ((rc = get_kernel(prog, "oeq_fixup_backward_reduce", 0, &k2))) return rc;
    long long grid = (long long)sm_count() * 8;
    if (grid > c_end - c_begin) grid = c_end - c_begin;
    void* args[] = {(void*)&scratch, (void*)&perm, (void*)&colptr, &c_begin, &c_end, &dX};
    return launch(k2, (unsigned)grid, 256, 0, args, st);
}

int fast_scatter(Entry* e, const void* scratch, const void* cols, const void* perm, long long N, long long E, void* colptr,
                 void* dX, cudaStream_t st) {
    if (int rc = fast_scatter_offsets(e, cols, perm, N, E, colptr, st)) return rc;
    return fast_scatter_rows(e, scratch, perm, colptr, 0, N, dX, st);
}

// ------------------------------------------------------------------- scratch that nobody has to allocate
// Backing store of oeqb_conv_backward_noalloc: a fixed array that is part of the library image, so every GPU that
// loads the library holds these bytes until the process exits.  In host code the name below is only a handle for
// the symbol; the device address is looked up once per device with cudaGetSymbolAddress.
static __device__ __align__(256) unsigned char g_noalloc_scratch[OEQB_NOALLOC_SCRATCH_BYTES];
void* g_noalloc_ptr[64] = {nullptr};

int noalloc_scratch(void** out) {
    int dev = 0;
    CUDA_TRY(cudaGetDevice(&dev));
    if (dev < 0 || dev >= 64) return fail(OEQB_EINVAL, "device index %d out of range", dev);
    if (!g_noalloc_ptr[dev]) {
        void* p = nullptr;
        cudaError_t ce = cudaGetSymbolAddress(&p, g_noalloc_scratch);
        if (ce != cudaSuccess || !p)
            return fail(OEQB_ECUDA, "cudaGetSymbolAddress(built-in scratch) failed on device %d: %s", dev, cudaGetErrorString(ce));
        g_noalloc_ptr[dev] = p;
    }
    *out = g_noalloc_ptr[dev];
    return OEQB_OK;
}

// ------------------------------------------------------------------------------------ tensor-core 'uvw'
struct TcParams {
    CUtensorMap src;
    const void* y; const void* W; void* dst;
    const void* x; void* dy;
    long long batch;
    int accum;
    int* status;
    int parts;
    int cut[kTcMaxParts + 1];
};
struct TcDwParams {
    CUtensorMap x; CUtensorMap g;
    const void* y; void* part;
    long long batch;
    int* status;
    int splits;
    int cut[kTcMaxParts + 1];
};

// SM cycles of an instance of a set (mode 0 and 1): per chunk the slowest of MMAs (12 of N / 2 cycles each), conversion and sums.
double tc_instance_cost(const Desc& d, int mode, int n) {
    const TcPlan& p = *d.tc_plan[mode];
    const TcPlan::Set& t = p.sets[p.inst[n].first];
    const std::vector<Block>& S = d.L[mode == 0 ? 0 : 2];
    double cost = 1000;
    for (auto& v : t.visits) {
        double pairs = 0;
        for (int i : v.ins) pairs += (double)ik_pairs(d.ins[i]).size();
        const Block& A = S[v.src];
        const double sums = 80 + 2 * pairs / A.d() * (p.tw / 2 * (mode == 1 ? 2 : 1) + 2);
        cost += (double)(A.mul / 32 * A.d()) * std::max(std::max(6.0 * p.tw * v.ins.size(), 280.0), sums);
    }
    return cost;
}
constexpr int kTcCutsDw = 4;
Cuts& tc_cuts(Entry* e, int which) {   // 2 * mode + (0 large sets, 1 small ones), or kTcCutsDw: of the groups, whose costs alone are used
    std::unique_ptr<Cuts>& slot = e->tc_cuts[which];
    if (slot) return *slot;
    slot = std::make_unique<Cuts>();
    const Desc& d = e->d;
    if (which == kTcCutsDw) {
        const std::vector<TcSub> subs = tc_subpaths(d);
        for (auto& g : tc_dw_groups(d)) slot->cost.push_back(2 * 600.0 * d.L[2][d.ins[subs[g[0]].ins].o].d() + 1000);   // two halves of a tile, a chunk per component
    } else {
        const TcPlan& p = *d.tc_plan[which / 2];
        for (int n = which % 2 ? p.ncoarse : 0; n < (which % 2 ? (int)p.inst.size() : p.ncoarse); ++n) slot->cost.push_back(tc_instance_cost(d, which / 2, n));
        cut_into_parts(*slot);
    }
    return *slot;
}
int tc_family(int mode, int list, bool parts) {
    const int fam[3][2] = {{FAM_UVW_TC, FAM_UVW_TC_DX}, {FAM_UVW_TC_PARTS, FAM_UVW_TC_DX_PARTS}, {FAM_UVW_TC_SMALL, FAM_UVW_TC_DX_SMALL}};
    return fam[list ? 2 : parts ? 1 : 0][mode];
}
// How the sets of `tiles` tiles are walked: which list of instances, and in how many parts (1: by one CTA per tile): whatever leaves the busiest
// CTA least to do when units are dealt out in turn.  Beside its sets a unit fills and drains the pipeline (about 3,000 cycles).
// 30 paths of 32 x 32, 20 tiles on 148 SMs: 20 us a forward in parts where a tile takes one CTA 40 us; 391 tiles: 119 us in one part.
int tc_parts(Entry* e, int mode, long long tiles, int* list) {
    const int sms = sm_count();
    *list = 0;
    if (tiles >= 16LL * sms) return 1;
    const Cuts* lists[2] = {&tc_cuts(e, 2 * mode), &tc_cuts(e, 2 * mode + 1)};
    return best_parts(lists, tiles, 3000.0, mode == 1 ? 1500.0 : 0.0, sms, list);
}

int keep_pool_memory();
void note_slow_path(const char* where, const char* why);

// The map of a [rows, cols] array of floats for copies of 32 columns x box_rows rows (cols a multiple of 32, 16-byte aligned).
int encode_map(CUtensorMap* map, const void* data, long long rows, long long cols, unsigned box_rows, bool swizzled) {
    typedef CUresult (*Encode)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*, const cuuint32_t*, const cuuint32_t*,
                               CUtensorMapInterleave, CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
    static Encode encode = nullptr;
    if (!encode) {
        void* f = nullptr;
        cudaDriverEntryPointQueryResult found;
        CUDA_TRY(cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &f, 12000, cudaEnableDefault, &found));
        if (!f || found != cudaDriverEntryPointSuccess) return fail(OEQB_ECUDA, "the driver has no cuTensorMapEncodeTiled");
        encode = (Encode)f;
    }
    const cuuint64_t dims[2] = {(cuuint64_t)cols, (cuuint64_t)rows}, strides[1] = {(cuuint64_t)cols * 4};
    const cuuint32_t box[2] = {32, box_rows}, step[2] = {1, 1};
    auto run = [&] {
        return encode(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 2, const_cast<void*>(data), dims, strides, box, step, CU_TENSOR_MAP_INTERLEAVE_NONE,
                      swizzled ? CU_TENSOR_MAP_SWIZZLE_128B : CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    };
    CUresult r = run();
    if (r == CUDA_ERROR_INVALID_CONTEXT) {   // the thread's first use of the device: the runtime's context is not current yet
        int dev = 0;
        CUDA_TRY(cudaGetDevice(&dev));
        CUDA_TRY(cudaSetDevice(dev));
        r = run();
    }
    if (r != CUDA_SUCCESS) return fail(OEQB_ECUDA, "cuTensorMapEncodeTiled(%lld x %lld) failed: %d", rows, cols, (int)r);
    return OEQB_OK;
}

// The kernel of a program, and whether it is what the host expects.  The warpgroups hand registers over (setmaxnreg): the shares only add up when the
// launch gives every thread 65536 / 512 of them.
int tc_kernel(Entry* e, int mode, int list, bool parts, cudaKernel_t* k, Program** prog) {
    static const char* names[2][2] = {{"oeq_uvw_tc_forward", "oeq_uvw_tc_forward_parts"}, {"oeq_uvw_tc_backward_dx", "oeq_uvw_tc_backward_dx_parts"}};
    const char* name = names[mode][parts];
    if (int rc = get_program(e, tc_family(mode, list, parts), prog)) return rc;
    if (int rc = get_kernel(*prog, name, e->d.tc_plan[mode]->smem, k)) return rc;
    if (!(*prog)->regs_ok) {
        cudaFuncAttributes attr;
        CUDA_TRY(cudaFuncGetAttributes(&attr, (const void*)*k));
        if (attr.numRegs != 128) return fail(OEQB_ECOMPILE, "%s was compiled to %d registers instead of 128: its register hand-over would not end", name, attr.numRegs);
        (*prog)->regs_ok = true;
    }
    return OEQB_OK;
}
// Compiles what a call on `batch` items needs before anything of it is launched, without g_mutex (`lock`, held).  OEQB_ECOMPILE: there is no usable
// program (noted once); the general kernels serve the problem from then on.
int tc_prepare(std::unique_lock<std::mutex>& lock, Entry* e, bool forward, bool backward, long long batch) {
    if (e->tc_off) return OEQB_ECOMPILE;
    int rc = OEQB_OK;
    for (int mode = forward ? 0 : 1; mode <= (backward ? 1 : 0) && !rc; ++mode) {
        int list;
        cudaKernel_t k;
        Program* prog;
        const bool parts = tc_parts(e, mode, (batch + 127) / 128, &list) > 1;
        if (!(rc = program_off_lock(lock, e, tc_family(mode, list, parts)))) rc = tc_kernel(e, mode, list, parts, &k, &prog);
    }
    if (backward && !rc) rc = program_off_lock(lock, e, FAM_UVW_TC_DW);
    if (backward && !rc) rc = program_off_lock(lock, e, FAM_DW_REDUCE);
    if (rc == OEQB_ECOMPILE) {
        e->tc_off = true;
        note_slow_path("uvw on the tensor cores", g_err.c_str());
    }
    return rc;
}

// mode 0: dst = z from (src = x, y, W); mode 1: dst = dx from (src = g, y, W), and dy with x
int tc_launch(Entry* e, const void* src, const void* y, const void* W, void* dst, const void* x, void* dy, long long batch, int accum, cudaStream_t st, int mode) {
    const Desc& d = e->d;
    TcParams p{{}, y, W, dst, x, dy, batch, accum, nullptr, 1, {0}};
    int rc = encode_map(&p.src, src, batch, d.dim[mode == 0 ? 0 : 2], 128, true);
    if (rc) return rc;
    if (!accum && (mode == 0 ? d.tc_zero_z : d.tc_zero_dx))
        CUDA_TRY(cudaMemsetAsync(dst, 0, (size_t)batch * d.dim[mode == 0 ? 2 : 0] * sizeof(float), st));
    if ((rc = status_word(&p.status))) return rc;
    const size_t smem = d.tc_plan[mode]->smem;
    const long long tiles = (batch + 127) / 128;
    int list = 0;
    p.parts = tc_parts(e, mode, tiles, &list);
    const Cuts& c = tc_cuts(e, 2 * mode + list);
    for (int i = 0; i <= p.parts; ++i) p.cut[i] = c.cut[p.parts][i];
    const bool parts = p.parts > 1;
    Program* prog;
    cudaKernel_t k, ks = nullptr;
    if ((rc = tc_kernel(e, mode, list, parts, &k, &prog))) return rc;
    const unsigned grid = (unsigned)std::min<long long>(sm_count(), tiles * p.parts);
    // stream-ordered scratch: an aligned copy of weights that start at an odd place (the kernel's loads are of 16 bytes), and the parts' sums of
    // dy, rows that a second kernel adds in order
    const bool copy_w = ((uintptr_t)W & 15u) != 0, rows = mode == 1 && parts;
    const size_t w_bytes = copy_w ? round_up((size_t)d.wn * sizeof(float)) : 0, row_bytes = rows ? (size_t)p.parts * batch * d.dim[1] * sizeof(float) : 0;
    char* scratch = nullptr;
    if (rows && (rc = get_kernel(prog, "oeq_uvw_tc_backward_dy_parts", 0, &ks))) return rc;
    if (w_bytes + row_bytes > 0) {
        if ((rc = keep_pool_memory())) return rc;
        CUDA_TRY(cudaMallocAsync((void**)&scratch, w_bytes + row_bytes, st));
    }
    if (copy_w) {
        p.W = scratch;
        const cudaError_t ce = cudaMemcpyAsync(scratch, W, (size_t)d.wn * sizeof(float), cudaMemcpyDeviceToDevice, st);
        if (ce != cudaSuccess) rc = fail(OEQB_ECUDA, "cudaMemcpyAsync: %s", cudaGetErrorString(ce));
    }
    if (rows) p.dy = scratch + w_bytes;
    void* args[] = {&p};
    if (!rc) rc = launch(k, grid, 512, smem, args, st);   // TC_THREADS
    if (!rc && rows) {
        long long n = batch * d.dim[1];
        void* sargs[] = {&p.dy, &dy, &n, &p.parts, &p.accum};
        rc = launch(ks, (unsigned)((n + 255) / 256), 256, 0, sargs, st);
    }
    if (scratch) cudaFreeAsync(scratch, st);
    return rc;
}

// Keep freed stream-ordered scratch in the device's pool: by default the pool gives memory back to the driver at every
// synchronisation and the next call pays for mapping it again.
int keep_pool_memory() {
    static bool pool_kept[64] = {false};
    int dev = 0;
    CUDA_TRY(cudaGetDevice(&dev));
    if (dev >= 0 && dev < 64 && !pool_kept[dev]) {
        cudaMemPool_t pool;
        CUDA_TRY(cudaDeviceGetDefaultMemPool(&pool, dev));
        uint64_t keep = UINT64_MAX;
        CUDA_TRY(cudaMemPoolSetAttribute(pool, cudaMemPoolAttrReleaseThreshold, &keep));
        pool_kept[dev] = true;
    }
    return OEQB_OK;
}

// dW = sum over the batch, on the tensor cores: the sums of every tile of 64 items are one row of a partials matrix (the
// tensor cores' accumulation truncates, so it is kept that short), oeq_generic_dw_reduce adds the rows in order.
int tc_backward_dw(Entry* e, const void* x, const void* y, const void* g, void* dW, long long batch, int accum, cudaStream_t st) {
    int rc;
    const Desc& d = e->d;
    TcDwParams p{{}, {}, y, nullptr, batch, nullptr, 1, {0}};
    if ((rc = encode_map(&p.x, x, batch, d.dim[0], 32, false)) || (rc = encode_map(&p.g, g, batch, d.dim[2], 32, false))) return rc;
    if ((rc = status_word(&p.status))) return rc;
    Program* prog;
    if ((rc = get_program(e, FAM_UVW_TC_DW, &prog))) return rc;
    cudaKernel_t k;
    const size_t smem = d.tc_dw_smem;
    if ((rc = get_kernel(prog, "oeq_uvw_tc_backward_dw", smem, &k))) return rc;
    long long tiles = (batch + 63) / 64;
    if ((rc = keep_pool_memory())) return rc;
    void* part = nullptr;
    CUDA_TRY(cudaMallocAsync(&part, (size_t)tiles * d.wn * sizeof(float), st));   // one row per tile of 64 items
    p.part = part;
    void* args[] = {&p};
    // A launch takes 16 groups (each writes its groups' part of every tile's row), a unit of work at most eight (their accumulators and the
    // A operands fill the tensor memory).  Of the ways to cut them: the one whose busiest CTA has least to do (a unit fills and drains, 3,000 cycles).
    const std::vector<double>& cost = tc_cuts(e, kTcCutsDw).cost;
    for (int g0 = 0; g0 < d.tc_ngrp && !rc; g0 += 16) {
        const int n = std::min(16, d.tc_ngrp - g0), sms = sm_count();
        double best = 0;
        for (int per = std::min(8, n); per >= 1; --per) {
            const int S = (n + per - 1) / per;
            double part_cost[kTcMaxParts];
            int cut[kTcMaxParts + 1];
            for (int s = 0; s <= S; ++s) cut[s] = (int)((long long)n * s / S);
            for (int s = 0; s < S; ++s) { part_cost[s] = 0; for (int i = cut[s]; i < cut[s + 1]; ++i) part_cost[s] += cost[g0 + i]; }
            const double t = busiest_load(tiles * S, S, part_cost, 3000.0, sms);
            if (best == 0 || t < 0.95 * best) { best = t; p.splits = S; for (int s = 0; s <= S; ++s) p.cut[s] = g0 + cut[s]; }
        }
        rc = launch(k, (unsigned)std::min<long long>(sms, tiles * p.splits), 21 * 32, smem, args, st);   // TC_THREADS
    }
    if (!rc) rc = dw_reduce(e, part, tiles, dW, accum, st);
    cudaFreeAsync(part, st);
    return rc;
}

// 'uvw' backward on the tensor cores; mask selects the outputs (1 dx, 2 dy, 4 dW).  dx is contracted with y_dx, dW with
// y_dw (they differ in the second-order pass); accum adds to the outputs.
int tc_backward(Entry* e, int mask, const void* x, const void* y_dx, const void* y_dw, const void* W, const void* g, void* dx,
                void* dy, void* dW, long long batch, int accum, cudaStream_t st) {
    if (mask & 3)     // dx and dy
        if (int rc = tc_launch(e, g, y_dx, W, dx, x, dy, batch, accum, st, 1)) return rc;
    if (mask & 4)     // dW: reduction over the batch on the tensor cores, fixed-order sum of the CTAs' rows
        if (int rc = tc_backward_dw(e, x, y_dw, g, dW, batch, accum, st)) return rc;
    return OEQB_OK;
}

// A problem that the specialised kernels serve took a slower route: counted (oeqb_slow_path_count) and, with the log
// option, reported, so that a performance cliff caused by an unaligned buffer or a missing workspace is visible.
std::atomic<long long> g_slow_paths{0};
void note_slow_path(const char* where, const char* why) {
    g_slow_paths.fetch_add(1, std::memory_order_relaxed);
    if (g_log) fprintf(stderr, "[oeq_b200] %s: %s\n", where, why);
}

// Index validation of a convolution call (caller holds g_mutex).  The channel-parallel kernels turn rows / cols /
// transpose_perm straight into addresses of bulk copies, so a bad entry would be a wild access on a shared GPU.  One
// small kernel checks the arrays, the host waits for it and reads the status word, and the call is refused with
// OEQB_EINVAL before any of the main kernels is launched.  The wait makes this a synchronising step, so by default it runs
// once per edge list (identified by its addresses and sizes; option "validate": 0 never, 2 every call) and never while
// the stream is being captured.
struct GraphKey {
    int dev; const void* rows; const void* cols; const void* perm; long long E, N; int sorted;
    bool operator<(const GraphKey& o) const {
        return std::tie(dev, rows, cols, perm, E, N, sorted) < std::tie(o.dev, o.rows, o.cols, o.perm, o.E, o.N, o.sorted);
    }
};
std::set<GraphKey> g_validated;

int validate_graph(const Desc& d, long long N, long long NS, long long E, const void* rows, const void* cols, const void* perm,
                   bool need_sorted, cudaStream_t st, const char* what) {
    if (g_validate <= 0 || E <= 0) return OEQB_OK;
    GraphKey key{0, rows, cols, perm, E, N * 0x100000001LL + NS, need_sorted ? 1 : 0};
    CUDA_TRY(cudaGetDevice(&key.dev));
    if (g_validate == 1 && g_validated.count(key)) return OEQB_OK;
    cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
    if (cudaStreamIsCapturing(st, &cap) != cudaSuccess || cap != cudaStreamCaptureStatusNone) return OEQB_OK;
    int* status = nullptr;
    if (int rc = status_word(&status)) return rc;
    const unsigned grid = (unsigned)((E + 255) / 256 < 2048 ? (E + 255) / 256 : 2048);
    if (d.idx == 3) gprep::validate_edges<int><<<grid, 256, 0, st>>>((const int*)rows, (const int*)cols, (const int*)perm, E, N, NS, need_sorted, status);
    else gprep::validate_edges<long long><<<grid, 256, 0, st>>>((const long long*)rows, (const long long*)cols, (const long long*)perm, E, N, NS, need_sorted, status);
    g_launches.fetch_add(1, std::memory_order_relaxed);
    CUDA_TRY(cudaGetLastError());
    CUDA_TRY(cudaStreamSynchronize(st));
    int dev = key.dev;
    const int code = *(volatile int*)g_status_host[dev];
    if (code == gprep::STATUS_BAD_INDEX) {
        *(volatile int*)g_status_host[dev] = 0;
        return fail(OEQB_EINVAL, "%s: rows must lie in [0, %lld) and cols in [0, %lld)%s%s; nothing was launched", what, N, NS,
                    need_sorted ? ", rows must be sorted (deterministic convolution)" : "",
                    perm ? ", transpose_perm in [0, n_edges)" : "");
    }
    if (g_validated.size() >= 256) g_validated.clear();
    g_validated.insert(key);
    return OEQB_OK;
}

int check_ptrs(std::initializer_list<const void*> ptrs, const char* what) {
    for (const void* p : ptrs)
        if (!p) return fail(OEQB_EINVAL, "%s: null pointer argument", what);
    return OEQB_OK;
}

}  // namespace

// =============================================================================================== C ABI
extern "C" {

const char* oeqb_last_error(void) { return g_err.c_str(); }
const char* oeqb_version(void) { return "oeq_b200 0.1 (sm_100a)"; }
int64_t oeqb_launch_count(void) { return g_launches.load(); }

int oeqb_set_option(const char* name, const char* value) {
    if (!name || !value) return fail(OEQB_EINVAL, "oeqb_set_option: null argument");
    std::lock_guard<std::mutex> lock(g_mutex);
    std::string n = name;
    if (n == "cache_dir") set_cache_dir(value);
    else if (n == "force_generic") g_force_generic = atoi(value) != 0;
    else if (n == "log") g_log = atoi(value) != 0;
    else if (n == "record") { g_record = atoi(value) != 0; if (g_record) g_recorded.clear(); }
    else if (n == "single_group") g_single_group = atoi(value) != 0;
    else if (n == "single_producer") g_single_producer = atoi(value) != 0;
    else if (n == "streams") g_streams = atoi(value);
    else if (n == "streams_forward") g_streams_fwd = atoi(value) != 0;
    else if (n == "validate") g_validate = atoi(value);
    else if (n == "no_tc") g_no_tc = atoi(value) != 0;
    else if (n == "tc_backward") g_tc_backward = atoi(value) & 7;
    else return fail(OEQB_EINVAL, "unknown option '%s'", name);
    return OEQB_OK;
}

int oeqb_launched_kernels(char* buf, size_t cap, size_t* needed) {
    if (!needed || (cap && !buf)) return fail(OEQB_EINVAL, "oeqb_launched_kernels: null argument");
    std::lock_guard<std::mutex> lock(g_mutex);
    std::string all;
    for (const std::string& n : g_recorded) all += n + "\n";
    *needed = all.size() + 1;
    if (cap) {
        const size_t n = std::min(all.size(), cap - 1);
        memcpy(buf, all.data(), n);
        buf[n] = '\0';
    }
    return OEQB_OK;
}

int oeqb_query(const void* desc, size_t desc_len, int64_t key, oeqb_kernel_prop* out) {
    if (!out) return fail(OEQB_EINVAL, "oeqb_query: null output");
    std::lock_guard<std::mutex> lock(g_mutex);
    Entry* e;
    int rc = get_entry(desc, desc_len, key, &e);
    if (rc) return rc;
    const Desc& d = e->d;
    memset(out, 0, sizeof *out);
    out->L1_dim = d.dim[0]; out->L2_dim = d.dim[1]; out->L3_dim = d.dim[2]; out->weight_numel = d.wn;
    out->shared_weights = d.shared; out->irrep_dtype = d.dtype; out->weight_dtype = d.dtype; out->idx_dtype = d.idx;
    out->is_conv = d.conv; out->deterministic = d.det; out->kahan = d.kahan; out->is_uvw = d.uvw;
    out->fast_path = (d.fast && !g_force_generic) ? 1 : ((d.tc && !g_force_generic && !g_no_tc) ? 2 : 0);
    return OEQB_OK;
}

int oeqb_emit_source(const void* desc, size_t desc_len, const char* kind, char* buf, size_t cap, size_t* needed) {
    if (!desc || !kind) return fail(OEQB_EINVAL, "oeqb_emit_source: null argument");
    Desc d;
    std::string why;
    if (!parse_desc((const char*)desc, desc_len, d, why)) return fail(OEQB_EPARSE, "descriptor: %s", why.c_str());
    int fam = family_from_name(kind);
    if (fam < 0) return fail(OEQB_EINVAL, "unknown kernel family '%s'", kind);
    std::string src = family_source(d, emit_header(d), fam);
    if (needed) *needed = src.size() + 1;
    if (buf && cap) {
        size_t n = src.size() < cap - 1 ? src.size() : cap - 1;
        memcpy(buf, src.data(), n);
        buf[n] = '\0';
    }
    return OEQB_OK;
}

int oeqb_precompile(const void* desc, size_t desc_len, int64_t key) {
    (void)key;
    if (!desc) return -fail(OEQB_EINVAL, "oeqb_precompile: null descriptor");
    Desc d;
    std::string why;
    if (!parse_desc((const char*)desc, desc_len, d, why)) return -fail(OEQB_EPARSE, "descriptor: %s", why.c_str());
    std::lock_guard<std::mutex> lock(g_mutex);
    const std::string header = emit_header(d);
    int done = 0;
    for (int fam = 0; fam < FAM_COUNT; ++fam) {
        if (fam == FAM_UVW_TC || fam == FAM_UVW_TC_PARTS || fam == FAM_UVW_TC_SMALL) { if (!d.tc) continue; }
        else if (fam >= FAM_UVW_TC_DX && fam <= FAM_UVW_TC_DX_SMALL) { if (!d.tc_bwd) continue; }
        else if (fam == FAM_UVW_ITEM) { if (!d.item) continue; }
        else if (fam == FAM_UVW_F64) { if (!d.f64mm) continue; }
        else if (fam == FAM_DW_REDUCE) { if (!d.shared) continue; }
        else if (fam != FAM_GENERIC && !d.fast) continue;
        if (fam >= FAM_FAST_BWD2_TP && fam <= FAM_FAST_BWD2_ATOMIC && d.fast_S4 < 3) continue;
        if (fam == FAM_FAST_FWD_ATOMIC && d.fast_S3 < 2) continue;
        if ((fam == FAM_FAST_FWD3_TP || fam == FAM_FAST_FWD3_DET) && d.fast_S4 < 3) continue;
        std::string cubin;
        int rc = compile_cubin(family_source(d, header, fam), family_name(fam), cubin);
        if (rc) return -rc;
        ++done;
        if (family_streams(d, fam, true) > 1) {   // the one-stream variant too: it is the fallback
            rc = compile_cubin(family_source(d, header, fam, false), family_name(fam), cubin);
            if (rc) return -rc;
            ++done;
        }
    }
    return done;
}

// (the launches cover 8 items per block: the x extent of a grid ends at 2^31 - 1)
static bool f64_route(const Desc& d, int64_t batch) { return d.f64mm > 0 && !g_force_generic && batch <= (1LL << 33); }

int oeqb_tp_forward(const void* desc, size_t desc_len, int64_t key, int64_t batch, const void* x, const void* y,
                    const void* W, void* z, void* stream) {
    if (batch < 0) return fail(OEQB_EINVAL, "oeqb_tp_forward: negative batch");
    if (batch == 0) return OEQB_OK;
    if (int rc = check_ptrs({x, y, W, z}, "oeqb_tp_forward")) return rc;
    std::unique_lock<std::mutex> lock(g_mutex);
    Entry* e;
    if (int rc = get_entry(desc, desc_len, key, &e)) return rc;
    if (use_fast(e->d) && aligned16({x, W})) {
        FastParams f{x, y, W, nullptr, z, nullptr, nullptr, nullptr, nullptr, nullptr, nullptr, batch, batch, nullptr};
        return fast_launch(e, 0, f, (cudaStream_t)stream);
    }
    if (e->d.tc && !g_force_generic && !g_no_tc && aligned16({x, z})) {
        const int rc = tc_prepare(lock, e, true, false, batch);
        if (rc != OEQB_ECOMPILE) return rc ? rc : tc_launch(e, x, y, W, z, nullptr, nullptr, batch, 0, (cudaStream_t)stream, 0);
    }
    if (f64_route(e->d, batch)) return f64_forward(e, x, y, W, z, batch, 0, (cudaStream_t)stream);
    if (item_forward_pays(e->d, batch) && aligned16({W})) return item_forward(e, x, y, W, z, batch, 0, (cudaStream_t)stream);
    FwdParams p{x, y, W, z, nullptr, nullptr, batch, batch, UNIT_ITEM, OUT_STORE};
    return generic_forward(e, p, (cudaStream_t)stream);
}

int oeqb_tp_backward(const void* desc, size_t desc_len, int64_t key, int64_t batch, const void* x, const void* y,
                     const void* W, const void* g, void* dx, void* dy, void* dW, void* stream) {
    if (batch < 0) return fail(OEQB_EINVAL, "oeqb_tp_backward: negative batch");
    if (int rc = check_ptrs({x, y, W, g, dx, dy, dW}, "oeqb_tp_backward")) return rc;
    std::unique_lock<std::mutex> lock(g_mutex);
    Entry* e;
    if (int rc = get_entry(desc, desc_len, key, &e)) return rc;
    cudaStream_t st = (cudaStream_t)stream;
    const Desc& d = e->d;
    if (d.shared) CUDA_TRY(cudaMemsetAsync(dW, 0, d.wn * d.elt(), st));
    if (batch == 0) return OEQB_OK;
    if (use_fast(d) && aligned16({x, W, dx})) {
        FastParams f{x, y, W, g, nullptr, dx, dy, dW, nullptr, nullptr, nullptr, batch, batch, nullptr};
        return fast_launch(e, 3, f, st);
    }
    if (f64_route(d, batch)) return f64_backward(e, x, y, y, W, g, dx, dy, dW, batch, 0, st);
    if (item_backward_pays(d, batch) && aligned16({W, dW})) return item_backward(e, x, y, y, W, g, dx, dy, dW, batch, 0, st);
    int tcb = (d.tc_bwd && !g_force_generic && !g_no_tc && aligned16({x, dx, g})) ? g_tc_backward : 0;
    if (tcb)
        if (int rc = tc_prepare(lock, e, false, true, batch)) {
            if (rc != OEQB_ECOMPILE) return rc;
            tcb = 0;
        }
    if (tcb != 7) {
        CUDA_TRY(cudaMemsetAsync(dy, 0, batch * d.dim[1] * d.elt(), st));
        BwdParams p{x, y, y, W, g, dx, dy, dW, nullptr, nullptr, nullptr, batch, batch, UNIT_ITEM, 0};
        if (int rc = generic_backward(e, p, st)) return rc;
    }
    return tc_backward(e, tcb, x, y, y, W, g, dx, dy, dW, batch, 0, st);
}

int oeqb_tp_double_backward(const void* desc, size_t desc_len, int64_t key, int64_t batch, const void* x,
                            const void* y, const void* W, const void* g, const void* x2, const void* y2,
                            const void* W2, void* dx, void* dy, void* dW, void* dg, void* stream) {
    if (batch < 0) return fail(OEQB_EINVAL, "oeqb_tp_double_backward: negative batch");
    if (int rc = check_ptrs({x, y, W, g, x2, y2, W2, dx, dy, dW, dg}, "oeqb_tp_double_backward")) return rc;
    std::unique_lock<std::mutex> lock(g_mutex);
    Entry* e;
    if (int rc = get_entry(desc, desc_len, key, &e)) return rc;
    cudaStream_t st = (cudaStream_t)stream;
    const Desc& d = e->d;
    if (d.shared) CUDA_TRY(cudaMemsetAsync(dW, 0, d.wn * d.elt(), st));
    if (batch == 0) return OEQB_OK;
    int rc;
    if (use_fast(d) && d.fast_S4 >= 3 && aligned16({x, x2, W, W2, dx})) {
        // same decomposition on the channel-parallel kernels: three forward passes (store, add, add) and two
        // second-order backward passes (the second adds); see the general path below for the algebra
        if (d.fast_S4 >= 3 && aligned16({dg})) {   // all three terms of dg in one pass
            FastParams f{x, y, W, nullptr, dg, nullptr, nullptr, nullptr, nullptr, nullptr, nullptr, batch, batch, nullptr};
            f.X2 = x2; f.Y2 = y2; f.W2 = W2;
            if ((rc = fast_launch(e, 0, f, st, nullptr, true))) return rc;
        } else {
            FastParams f{x2, y, W, nullptr, dg, nullptr, nullptr, nullptr, nullptr, nullptr, nullptr, batch, batch, nullptr};
            if ((rc = fast_launch(e, 0, f, st))) return rc;
            f.X = x; f.Y = y2; f.accum = 1;
            if ((rc = fast_launch(e, 0, f, st))) return rc;
            f.Y = y; f.W = W2;
            if ((rc = fast_launch(e, 0, f, st))) return rc;
        }
        FastParams b{x, y, W, g, nullptr, dx, dy, dW, nullptr, nullptr, nullptr, batch, batch, nullptr};
        b.X2 = x2; b.Y2 = y2; b.W2 = W2;   // both second-order backward terms in one pass
        return fast_launch(e, 3, b, st, nullptr, true);
    }
    if (d.tc_bwd && !g_force_generic && !g_no_tc && g_tc_backward == 7 && aligned16({x, x2, dx, dg, g}) &&
        (rc = tc_prepare(lock, e, true, true, batch)) != OEQB_ECOMPILE) {
        // the same five passes on the tensor-core kernels (the second and later ones add to their outputs)
        if (rc) return rc;
        if ((rc = tc_launch(e, x2, y, W, dg, nullptr, nullptr, batch, 0, st, 0))) return rc;
        if ((rc = tc_launch(e, x, y2, W, dg, nullptr, nullptr, batch, 1, st, 0))) return rc;
        if ((rc = tc_launch(e, x, y, W2, dg, nullptr, nullptr, batch, 1, st, 0))) return rc;
        if ((rc = tc_backward(e, 7, x2, y2, y, W, g, dx, dy, dW, batch, 0, st))) return rc;
        return tc_backward(e, 7, x, y, y2, W2, g, dx, dy, dW, batch, 1, st);
    }
    if (f64_route(d, batch)) {   // the five passes of the general path below
        if ((rc = f64_forward(e, x2, y, W, dg, batch, 0, st))) return rc;
        if ((rc = f64_forward(e, x, y2, W, dg, batch, 1, st))) return rc;
        if ((rc = f64_forward(e, x, y, W2, dg, batch, 1, st))) return rc;
        if ((rc = f64_backward(e, x2, y2, y, W, g, dx, dy, dW, batch, 0, st))) return rc;
        return f64_backward(e, x, y, y2, W2, g, dx, dy, dW, batch, 1, st);
    }
    // dg = F(x2, y, W) + F(x, y2, W) + F(x, y, W2): the product is linear in each argument
    if (item_forward_pays(d, batch) && aligned16({W, W2})) {
        if ((rc = item_forward(e, x2, y, W, dg, batch, 0, st))) return rc;
        if ((rc = item_forward(e, x, y2, W, dg, batch, 1, st))) return rc;
        if ((rc = item_forward(e, x, y, W2, dg, batch, 1, st))) return rc;
    } else {
        FwdParams f{x2, y, W, dg, nullptr, nullptr, batch, batch, UNIT_ITEM, OUT_STORE};
        if ((rc = generic_forward(e, f, st))) return rc;
        f.x = x; f.y = y2; f.out_mode = OUT_ADD;
        if ((rc = generic_forward(e, f, st))) return rc;
        f.y = y; f.W = W2;
        if ((rc = generic_forward(e, f, st))) return rc;
    }
    // (dx, dy, dW) = mixed second derivatives contracted with g
    if (item_backward_pays(d, batch) && aligned16({W, W2, dW})) {
        if ((rc = item_backward(e, x2, y2, y, W, g, dx, dy, dW, batch, 0, st))) return rc;
        return item_backward(e, x, y, y2, W2, g, dx, dy, dW, batch, 1, st);
    }
    CUDA_TRY(cudaMemsetAsync(dy, 0, batch * d.dim[1] * d.elt(), st));
    BwdParams b{x2, y2, y, W, g, dx, dy, dW, nullptr, nullptr, nullptr, batch, batch, UNIT_ITEM, 0};
    if ((rc = generic_backward(e, b, st))) return rc;
    b.x = x; b.y_dx = y; b.y_dw = y2; b.W = W2; b.accum = 1;
    return generic_backward(e, b, st);
}

int64_t oeqb_conv_workspace_bytes(const void* desc, size_t desc_len, int64_t key, int direction, int64_t n_nodes,
                                  int64_t n_edges) {
    if (n_nodes < 0 || n_edges < 0 || direction < 0 || direction > 2)
        return -(int64_t)fail(OEQB_EINVAL, "oeqb_conv_workspace_bytes: bad argument");
    std::lock_guard<std::mutex> lock(g_mutex);
    Entry* e;
    if (int rc = get_entry(desc, desc_len, key, &e)) return -(int64_t)rc;
    const Desc& d = e->d;
    // Deterministic backward on the channel-parallel path: one dX row per edge plus the sender offsets.
    if ((direction == 1 || (direction == 2 && d.fast_S4 >= 3)) && d.conv && d.det && use_fast(d))
        return (int64_t)(round_up((size_t)n_edges * d.dim[0] * d.elt()) + round_up((size_t)(n_nodes + 1) * 8));
    // Unsorted (atomic) convolutions on the channel-parallel path: room to group the edge list by receiver first.
    if (d.conv && !d.det && use_fast(d) && n_edges > 0) return (int64_t)atomic_order_bytes(d, n_nodes, n_edges);
    return 0;
}

static int conv_check(const Desc& d, int64_t n_nodes, int64_t n_edges, const void* perm, const char* what) {
    if (n_nodes < 0 || n_edges < 0) return fail(OEQB_EINVAL, "%s: negative size", what);
    if (!d.conv) return fail(OEQB_EINVAL, "%s: descriptor was not built for a convolution", what);
    if (d.det && n_edges > 0 && !perm) return fail(OEQB_EINVAL, "%s: deterministic mode needs transpose_perm", what);
    return OEQB_OK;
}

static int conv_backward_impl(const void* desc, size_t desc_len, int64_t key, int64_t n_receivers, int64_t n_nodes,
                              int64_t n_edges, const void* X, const void* Y, const void* W, const void* G, void* dX,
                              void* dY, void* dW, const void* rows, const void* cols, const void* transpose_perm,
                              void* workspace, int64_t workspace_bytes, void* stream, bool defer_rows);

int oeqb_conv_forward(const void* desc, size_t desc_len, int64_t key, int64_t n_nodes, int64_t n_edges,
                      const void* X, const void* Y, const void* W, void* Z, const void* rows, const void* cols,
                      const void* transpose_perm, void* workspace, int64_t workspace_bytes, void* stream) {
    return oeqb_conv_forward_rect(desc, desc_len, key, n_nodes, n_nodes, n_edges, X, Y, W, Z, rows, cols, transpose_perm,
                                  workspace, workspace_bytes, stream);
}

int oeqb_conv_forward_rect(const void* desc, size_t desc_len, int64_t key, int64_t n_nodes, int64_t n_senders,
                           int64_t n_edges, const void* X, const void* Y, const void* W, void* Z, const void* rows,
                           const void* cols, const void* transpose_perm, void* workspace, int64_t workspace_bytes,
                           void* stream) {
    if (n_senders < 0) return fail(OEQB_EINVAL, "oeqb_conv_forward_rect: negative size");
    std::lock_guard<std::mutex> lock(g_mutex);
    Entry* e;
    if (int rc = get_entry(desc, desc_len, key, &e)) return rc;
    const Desc& d = e->d;
    if (int rc = conv_check(d, n_nodes, n_edges, transpose_perm, "oeqb_conv_forward")) return rc;
    if (n_nodes == 0) return OEQB_OK;
    if (int rc = check_ptrs({X, Z}, "oeqb_conv_forward")) return rc;
    if (n_edges > 0) if (int rc = check_ptrs({Y, W, rows, cols}, "oeqb_conv_forward")) return rc;
    cudaStream_t st = (cudaStream_t)stream;
    if (int rc = validate_graph(d, n_nodes, n_senders, n_edges, rows, cols, nullptr, d.det != 0, st, "oeqb_conv_forward")) return rc;
    const bool fast = use_fast(d) && n_edges > 0 && aligned16({X, W});
    if (use_fast(d) && n_edges > 0 && !fast) note_slow_path("oeqb_conv_forward", "X or W is not 16-byte aligned: general kernels");
    if (d.det) {
        if (fast) {
            FastParams f{X, Y, W, nullptr, Z, nullptr, nullptr, nullptr, nullptr, rows, cols, n_nodes, n_edges, nullptr};
            return fast_launch(e, 1, f, st);
        }
        FwdParams p{X, Y, W, Z, rows, cols, n_nodes, n_edges, UNIT_SEGMENT, OUT_STORE};
        return generic_forward(e, p, st);
    }
    if (fast) {
        // Group the edges by receiver on the device, then run the sorted-list kernel through that order: each
        // receiver row is summed in registers and written once, instead of one 50 KB read-modify-write per edge.
        const void* order = nullptr;
        const int grc = group_by_receiver(d, n_nodes, n_edges, rows, workspace, workspace_bytes, st, &order);
        if (grc > 0) return grc;
        if (grc == 0) {
            FastParams f{X, Y, W, nullptr, Z, nullptr, nullptr, nullptr, nullptr, rows, cols, n_nodes, n_edges, nullptr};
            f.eorder = order;
            return fast_launch(e, 1, f, st);
        }
        note_slow_path("oeqb_conv_forward", "no workspace for grouping the edges by receiver: per-edge scatter");
    }
    CUDA_TRY(cudaMemsetAsync(Z, 0, n_nodes * d.dim[2] * d.elt(), st));
    if (fast && d.fast_S3 >= 2 && aligned16({Z})) {
        FastParams f{X, Y, W, nullptr, Z, nullptr, nullptr, nullptr, nullptr, rows, cols, n_nodes, n_edges, nullptr};
        return fast_launch(e, 2, f, st);
    }
    FwdParams p{X, Y, W, Z, rows, cols, n_edges, n_edges, UNIT_EDGE, OUT_ATOMIC};
    return generic_forward(e, p, st);
}

int oeqb_conv_backward(const void* desc, size_t desc_len, int64_t key, int64_t n_nodes, int64_t n_edges,
                       const void* X, const void* Y, const void* W, const void* G, void* dX, void* dY, void* dW,
                       const void* rows, const void* cols, const void* transpose_perm, void* workspace,
                       int64_t workspace_bytes, void* stream) {
    return oeqb_conv_backward_rect(desc, desc_len, key, n_nodes, n_nodes, n_edges, X, Y, W, G, dX, dY, dW, rows, cols,
                                   transpose_perm, workspace, workspace_bytes, stream);
}

int oeqb_conv_backward_rect(const void* desc, size_t desc_len, int64_t key, int64_t n_receivers, int64_t n_nodes,
                            int64_t n_edges, const void* X, const void* Y, const void* W, const void* G, void* dX,
                            void* dY, void* dW, const void* rows, const void* cols, const void* transpose_perm,
                            void* workspace, int64_t workspace_bytes, void* stream) {
    return conv_backward_impl(desc, desc_len, key, n_receivers, n_nodes, n_edges, X, Y, W, G, dX, dY, dW, rows, cols,
                              transpose_perm, workspace, workspace_bytes, stream, /*defer_rows=*/false);
}

int oeqb_conv_backward_edges(const void* desc, size_t desc_len, int64_t key, int64_t n_receivers, int64_t n_nodes,
                             int64_t n_edges, const void* X, const void* Y, const void* W, const void* G, void* dY,
                             void* dW, const void* rows, const void* cols, const void* transpose_perm, void* workspace,
                             int64_t workspace_bytes, void* stream) {
    // dX is not touched by this step; a non-null placeholder satisfies the common argument checks
    return conv_backward_impl(desc, desc_len, key, n_receivers, n_nodes, n_edges, X, Y, W, G, workspace, dY, dW, rows, cols,
                              transpose_perm, workspace, workspace_bytes, stream, /*defer_rows=*/true);
}

int oeqb_conv_backward_rows(const void* desc, size_t desc_len, int64_t key, int64_t n_nodes, int64_t n_edges,
                            int64_t row_begin, int64_t row_end, const void* transpose_perm, void* workspace,
                            int64_t workspace_bytes, void* dX, void* stream) {
    if (row_begin < 0 || row_end > n_nodes || row_begin > row_end)
        return fail(OEQB_EINVAL, "oeqb_conv_backward_rows: bad row range [%lld, %lld) of %lld", (long long)row_begin,
                    (long long)row_end, (long long)n_nodes);
    std::lock_guard<std::mutex> lock(g_mutex);
    Entry* e;
    if (int rc = get_entry(desc, desc_len, key, &e)) return rc;
    const Desc& d = e->d;
    if (!(d.conv && d.det && use_fast(d)))
        return fail(OEQB_EUNSUPPORTED, "oeqb_conv_backward_rows: only after oeqb_conv_backward_edges (deterministic "
                                       "convolutions on the channel-parallel kernels)");
    const size_t scratch_bytes = round_up((size_t)n_edges * d.dim[0] * d.elt());
    const size_t need = scratch_bytes + round_up((size_t)(n_nodes + 1) * 8);
    if (!workspace || workspace_bytes < (int64_t)need || !dX || !transpose_perm || !aligned16({workspace, dX}))
        return fail(OEQB_EINVAL, "oeqb_conv_backward_rows: needs the workspace of the matching oeqb_conv_backward_edges call "
                                 "(%zu bytes), dX and transpose_perm", need);
    return fast_scatter_rows(e, workspace, transpose_perm, (char*)workspace + scratch_bytes, row_begin, row_end, dX,
                             (cudaStream_t)stream);
}

static int conv_backward_impl(const void* desc, size_t desc_len, int64_t key, int64_t n_receivers, int64_t n_nodes,
                              int64_t n_edges, const void* X, const void* Y, const void* W, const void* G, void* dX,
                              void* dY, void* dW, const void* rows, const void* cols, const void* transpose_perm,
                              void* workspace, int64_t workspace_bytes, void* stream, bool defer_rows) {
    if (n_receivers < 0) return fail(OEQB_EINVAL, "oeqb_conv_backward_rect: negative size");
    std::lock_guard<std::mutex> lock(g_mutex);
    Entry* e;
    if (int rc = get_entry(desc, desc_len, key, &e)) return rc;
    const Desc& d = e->d;
    if (int rc = conv_check(d, n_nodes, n_edges, transpose_perm, "oeqb_conv_backward")) return rc;
    cudaStream_t st = (cudaStream_t)stream;
    if (d.shared) { if (!dW) return fail(OEQB_EINVAL, "oeqb_conv_backward: null dW"); CUDA_TRY(cudaMemsetAsync(dW, 0, d.wn * d.elt(), st)); }
    if (n_nodes == 0) return OEQB_OK;
    if (int rc = check_ptrs({X, G, dX}, "oeqb_conv_backward")) return rc;
    if (n_edges > 0) {
        if (int rc = check_ptrs({Y, W, dY, dW, rows, cols}, "oeqb_conv_backward")) return rc;
        if (int rc = validate_graph(d, n_receivers, n_nodes, n_edges, rows, cols, d.det ? transpose_perm : nullptr, d.det != 0, st, "oeqb_conv_backward")) return rc;
    }
    const bool fast = use_fast(d) && n_edges > 0 && aligned16({X, W, G, dX, workspace});
    if (use_fast(d) && n_edges > 0 && !fast) note_slow_path("oeqb_conv_backward", "an operand is not 16-byte aligned: general kernels");
    if (d.det && fast) {
        const size_t scratch_bytes = round_up((size_t)n_edges * d.dim[0] * d.elt());
        const size_t need = scratch_bytes + round_up((size_t)(n_nodes + 1) * 8);
        if (!workspace || workspace_bytes < (int64_t)need)
            return fail(OEQB_EINVAL, "oeqb_conv_backward: workspace of %lld bytes is smaller than the %zu required",
                        (long long)workspace_bytes, need);
        void* colptr = (char*)workspace + scratch_bytes;
        FastParams f{X, Y, W, G, nullptr, dX, dY, dW, workspace, rows, cols, n_nodes, n_edges, nullptr};
        if (int rc = fast_launch(e, 4, f, st)) return rc;
        if (defer_rows) return fast_scatter_offsets(e, cols, transpose_perm, n_nodes, n_edges, colptr, st);
        return fast_scatter(e, workspace, cols, transpose_perm, n_nodes, n_edges, colptr, dX, st);
    }
    if (defer_rows)
        return fail(OEQB_EUNSUPPORTED, "oeqb_conv_backward_edges: this problem (or these buffers) is not served by the "
                                       "deterministic channel-parallel kernels; call oeqb_conv_backward");
    if (!d.det && fast) {
        CUDA_TRY(cudaMemsetAsync(dX, 0, n_nodes * d.dim[0] * d.elt(), st));
        FastParams f{X, Y, W, G, nullptr, dX, dY, dW, nullptr, rows, cols, n_nodes, n_edges, nullptr};
        // walked receiver by receiver (grouped on the device), a receiver's gradient row is read once, not once per edge
        const int grc = group_by_receiver(d, n_nodes, n_edges, rows, workspace, workspace_bytes, st, &f.eorder);
        if (grc > 0) return grc;
        if (grc < 0) note_slow_path("oeqb_conv_backward", "no workspace for grouping the edges by receiver");
        return fast_launch(e, 5, f, st);
    }
    if (n_edges > 0) CUDA_TRY(cudaMemsetAsync(dY, 0, n_edges * d.dim[1] * d.elt(), st));
    if (d.det) {
        BwdParams p{X, Y, Y, W, G, dX, dY, dW, rows, cols, transpose_perm, n_nodes, n_edges, UNIT_SEGMENT, 0};
        return generic_backward(e, p, st);
    }
    CUDA_TRY(cudaMemsetAsync(dX, 0, n_nodes * d.dim[0] * d.elt(), st));
    BwdParams p{X, Y, Y, W, G, dX, dY, dW, rows, cols, nullptr, n_edges, n_edges, UNIT_EDGE, 0};
    return generic_backward(e, p, st);
}

int oeqb_conv_double_backward(const void* desc, size_t desc_len, int64_t key, int64_t n_nodes, int64_t n_edges,
                              const void* X, const void* Y, const void* W, const void* G, const void* X2,
                              const void* Y2, const void* W2, void* dX, void* dY, void* dW, void* dG,
                              const void* rows, const void* cols, const void* transpose_perm, void* workspace,
                              int64_t workspace_bytes, void* stream) {
    std::lock_guard<std::mutex> lock(g_mutex);
    Entry* e;
    if (int rc = get_entry(desc, desc_len, key, &e)) return rc;
    const Desc& d = e->d;
    if (int rc = conv_check(d, n_nodes, n_edges, transpose_perm, "oeqb_conv_double_backward")) return rc;
    cudaStream_t st = (cudaStream_t)stream;
    if (d.shared) { if (!dW) return fail(OEQB_EINVAL, "oeqb_conv_double_backward: null dW"); CUDA_TRY(cudaMemsetAsync(dW, 0, d.wn * d.elt(), st)); }
    if (n_nodes == 0) return OEQB_OK;
    if (int rc = check_ptrs({X, G, X2, dX, dG}, "oeqb_conv_double_backward")) return rc;
    if (n_edges > 0) {
        if (int rc = check_ptrs({Y, W, Y2, W2, dY, dW, rows, cols}, "oeqb_conv_double_backward")) return rc;
        if (int rc = validate_graph(d, n_nodes, n_nodes, n_edges, rows, cols, d.det ? transpose_perm : nullptr, d.det != 0, st, "oeqb_conv_double_backward")) return rc;
    }
    int rc;
    if (use_fast(d) && d.fast_S4 >= 3 && (d.det || d.fast_S3 >= 2) && n_edges > 0 && aligned16({X, X2, W, W2, G, dX, dG, workspace})) {
        // channel-parallel kernels: dG from one fused second-order forward pass (three terms), (dX, dY, dW) from one
        // fused second-order backward pass.  An unsorted edge list is grouped by receiver first and then walked through
        // that order by the same kernels as a sorted one; without room for the grouping it takes three accumulating
        // forward passes with a per-edge scatter.
        const int kb = d.det ? 4 : 5;
        void* colptr = nullptr;
        const void* order = nullptr;
        if (d.det) {
            const size_t scratch_bytes = round_up((size_t)n_edges * d.dim[0] * d.elt());
            const size_t need = scratch_bytes + round_up((size_t)(n_nodes + 1) * 8);
            if (!workspace || workspace_bytes < (int64_t)need)
                return fail(OEQB_EINVAL, "oeqb_conv_double_backward: workspace of %lld bytes is smaller than the %zu required",
                            (long long)workspace_bytes, need);
            colptr = (char*)workspace + scratch_bytes;
        } else {
            const int grc = group_by_receiver(d, n_nodes, n_edges, rows, workspace, workspace_bytes, st, &order);
            if (grc > 0) return grc;
            if (grc < 0) note_slow_path("oeqb_conv_double_backward", "no workspace for grouping the edges by receiver");
            CUDA_TRY(cudaMemsetAsync(dX, 0, n_nodes * d.dim[0] * d.elt(), st));
        }
        if (d.det || order) {   // all three terms of dG in one pass over receiver-grouped edges
            FastParams f{X, Y, W, nullptr, dG, nullptr, nullptr, nullptr, nullptr, rows, cols, n_nodes, n_edges, nullptr};
            f.X2 = X2; f.Y2 = Y2; f.W2 = W2; f.eorder = order;
            if ((rc = fast_launch(e, 1, f, st, nullptr, true))) return rc;
        } else {
            CUDA_TRY(cudaMemsetAsync(dG, 0, n_nodes * d.dim[2] * d.elt(), st));
            FastParams f{X2, Y, W, nullptr, dG, nullptr, nullptr, nullptr, nullptr, rows, cols, n_nodes, n_edges, nullptr};
            if ((rc = fast_launch(e, 2, f, st))) return rc;
            f.X = X; f.Y = Y2; f.accum = 1;
            if ((rc = fast_launch(e, 2, f, st))) return rc;
            f.Y = Y; f.W = W2;
            if ((rc = fast_launch(e, 2, f, st))) return rc;
        }
        FastParams b{X, Y, W, G, nullptr, dX, dY, dW, workspace, rows, cols, n_nodes, n_edges, nullptr};
        b.X2 = X2; b.Y2 = Y2; b.W2 = W2; b.eorder = order;   // both second-order backward terms in one pass
        if ((rc = fast_launch(e, kb, b, st, nullptr, true))) return rc;
        if (d.det) return fast_scatter(e, workspace, cols, transpose_perm, n_nodes, n_edges, colptr, dX, st);
        return OEQB_OK;
    }
    if (n_edges > 0) CUDA_TRY(cudaMemsetAsync(dY, 0, n_edges * d.dim[1] * d.elt(), st));
    if (d.det) {
        FwdParams f{X2, Y, W, dG, rows, cols, n_nodes, n_edges, UNIT_SEGMENT, OUT_STORE};
        if ((rc = generic_forward(e, f, st))) return rc;
        f.x = X; f.y = Y2; f.out_mode = OUT_ADD;
        if ((rc = generic_forward(e, f, st))) return rc;
        f.y = Y; f.W = W2;
        if ((rc = generic_forward(e, f, st))) return rc;
        BwdParams b{X2, Y2, Y, W, G, dX, dY, dW, rows, cols, transpose_perm, n_nodes, n_edges, UNIT_SEGMENT, 0};
        if ((rc = generic_backward(e, b, st))) return rc;
        b.x = X; b.y_dx = Y; b.y_dw = Y2; b.W = W2; b.accum = 1;
        return generic_backward(e, b, st);
    }
    CUDA_TRY(cudaMemsetAsync(dG, 0, n_nodes * d.dim[2] * d.elt(), st));
    CUDA_TRY(cudaMemsetAsync(dX, 0, n_nodes * d.dim[0] * d.elt(), st));
    FwdParams f{X2, Y, W, dG, rows, cols, n_edges, n_edges, UNIT_EDGE, OUT_ATOMIC};
    if ((rc = generic_forward(e, f, st))) return rc;
    f.x = X; f.y = Y2;
    if ((rc = generic_forward(e, f, st))) return rc;
    f.y = Y; f.W = W2;
    if ((rc = generic_forward(e, f, st))) return rc;
    BwdParams b{X2, Y2, Y, W, G, dX, dY, dW, rows, cols, nullptr, n_edges, n_edges, UNIT_EDGE, 0};
    if ((rc = generic_backward(e, b, st))) return rc;
    b.x = X; b.y_dx = Y; b.y_dw = Y2; b.W = W2; b.accum = 1;
    return generic_backward(e, b, st);
}


int oeqb_conv_backward_noalloc(const void* desc, size_t desc_len, int64_t key, int64_t n_nodes, int64_t n_edges,
                               const void* X, const void* Y, const void* W, const void* G, void* dX, void* dY, void* dW,
                               const void* rows, const void* cols, const void* transpose_perm, void* stream) {
    std::lock_guard<std::mutex> lock(g_mutex);
    Entry* e;
    if (int rc = get_entry(desc, desc_len, key, &e)) return rc;
    const Desc& d = e->d;
    if (int rc = conv_check(d, n_nodes, n_edges, transpose_perm, "oeqb_conv_backward_noalloc")) return rc;
    if (!(d.det && use_fast(d)))
        return fail(OEQB_EUNSUPPORTED, "oeqb_conv_backward_noalloc: only deterministic convolutions served by the "
                                       "channel-parallel kernels use scratch; call oeqb_conv_backward for this problem");
    if (n_nodes == 0 || n_edges == 0)
        return fail(OEQB_EINVAL, "oeqb_conv_backward_noalloc: empty graph; call oeqb_conv_backward");
    const size_t scratch_bytes = round_up((size_t)n_edges * d.dim[0] * d.elt());
    const size_t colptr_bytes = round_up((size_t)(n_nodes + 1) * 8);
    const size_t need = scratch_bytes + colptr_bytes + kAlign;   // last slot: the kernels' status word
    if (need > (size_t)OEQB_NOALLOC_SCRATCH_BYTES)
        return fail(OEQB_EINVAL, "oeqb_conv_backward_noalloc: this graph needs %zu bytes of scratch (%lld edges x %lld-float "
                                 "rows + %lld sender offsets) but the built-in array holds %zu; use oeqb_conv_backward "
                                 "with a caller-provided workspace",
                    need, (long long)n_edges, (long long)d.dim[0], (long long)n_nodes + 1, (size_t)OEQB_NOALLOC_SCRATCH_BYTES);
    if (int rc = check_ptrs({X, Y, W, G, dX, dY, dW, rows, cols}, "oeqb_conv_backward_noalloc")) return rc;
    if (!aligned16({X, W, G, dX}))
        return fail(OEQB_EINVAL, "oeqb_conv_backward_noalloc: X, W, G and dX must be 16-byte aligned");
    void* base = nullptr;
    if (int rc = noalloc_scratch(&base)) return rc;
    cudaStream_t st = (cudaStream_t)stream;
    void* colptr = (char*)base + scratch_bytes;
    // The kernels' status word sits in the last slot of the array, wherever the graph's rows end, so that
    // oeqb_noalloc_status can find it without knowing the sizes of the call that wrote it.
    int* status = (int*)((char*)base + (size_t)OEQB_NOALLOC_SCRATCH_BYTES - kAlign);
    // The array keeps whatever the previous call left.  Per-edge rows and sender offsets are overwritten in full by
    // the kernels below; only the status word has to start at zero.
    CUDA_TRY(cudaMemsetAsync(status, 0, sizeof(int), st));
    FastParams f{X, Y, W, G, nullptr, dX, dY, dW, base, rows, cols, n_nodes, n_edges, nullptr};
    if (int rc = fast_launch(e, 4, f, st, status)) return rc;
    return fast_scatter(e, base, cols, transpose_perm, n_nodes, n_edges, colptr, dX, st);
}

int oeqb_selftest_bounded_wait(const void* desc, size_t desc_len, int64_t key, void* stream) {
    std::lock_guard<std::mutex> lock(g_mutex);
    Entry* e;
    if (int rc = get_entry(desc, desc_len, key, &e)) return rc;
    if (!use_fast(e->d)) return fail(OEQB_EUNSUPPORTED, "oeqb_selftest_bounded_wait: the descriptor is not served by the channel-parallel kernels");
    int* status = nullptr;
    if (int rc = status_word(&status)) return rc;
    Program* prog;
    if (int rc = get_program(e, FAM_FAST_SCATTER, &prog)) return rc;
    cudaKernel_t k;
    if (int rc = get_kernel(prog, "oeq_selftest_starved_wait", 0, &k)) return rc;
    cudaStream_t st = (cudaStream_t)stream;
    int* left = nullptr;
    CUDA_TRY(cudaMallocAsync((void**)&left, sizeof(int), st));
    CUDA_TRY(cudaMemsetAsync(left, 0, sizeof(int), st));
    void* args[] = {&status, &left};
    int rc = launch(k, 1, 64, 0, args, st);
    int came_back = 0;
    if (!rc) {
        CUDA_TRY(cudaMemcpyAsync(&came_back, left, sizeof(int), cudaMemcpyDeviceToHost, st));
        CUDA_TRY(cudaStreamSynchronize(st));
    }
    cudaFreeAsync(left, st);
    if (rc) return rc;
    // the kernel must have returned (it did: the synchronisation came back), every thread must have left, and the status
    // word must carry the code; reading it clears it
    const int seen = status_word(nullptr);
    if (came_back != 64) return fail(OEQB_EKERNEL, "oeqb_selftest_bounded_wait: %d of 64 threads came back", came_back);
    if (seen != OEQB_EKERNEL) return fail(OEQB_EKERNEL, "oeqb_selftest_bounded_wait: the starved wait did not report through the status word");
    return OEQB_OK;
}

int oeqb_stream_is_capturing(void* stream) {
    cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
    if (cudaStreamIsCapturing((cudaStream_t)stream, &cap) != cudaSuccess) return -fail(OEQB_ECUDA, "cudaStreamIsCapturing failed");
    return cap != cudaStreamCaptureStatusNone;
}

int oeqb_check_status(void) {
    std::lock_guard<std::mutex> lock(g_mutex);
    return status_word(nullptr);
}

int64_t oeqb_slow_path_count(void) { return g_slow_paths.load(); }

int64_t oeqb_graph_workspace_bytes(int64_t n_nodes, int64_t n_edges) {
    if (n_nodes < 0 || n_edges < 0) return -(int64_t)fail(OEQB_EINVAL, "oeqb_graph_workspace_bytes: negative size");
    return (int64_t)gprep::group_workspace_bytes(n_nodes, n_edges);
}

int oeqb_prepare_graph(int idx_dtype, int64_t n_nodes, int64_t n_edges, const void* rows, const void* cols,
                       void* sorted_rows, void* sorted_cols, void* order, void* transpose_perm, void* workspace,
                       int64_t workspace_bytes, void* stream) {
    if (idx_dtype != 3 && idx_dtype != 4) return fail(OEQB_EINVAL, "oeqb_prepare_graph: idx_dtype must be 3 (int32) or 4 (int64)");
    if (n_nodes < 0 || n_edges < 0) return fail(OEQB_EINVAL, "oeqb_prepare_graph: negative size");
    if (n_edges == 0) return OEQB_OK;
    if (n_nodes == 0) return fail(OEQB_EINVAL, "oeqb_prepare_graph: edges without nodes");
    if (int rc = check_ptrs({rows, cols, sorted_rows, sorted_cols, order, transpose_perm, workspace}, "oeqb_prepare_graph")) return rc;
    if (workspace_bytes < (int64_t)gprep::group_workspace_bytes(n_nodes, n_edges) || ((uintptr_t)workspace & 15u))
        return fail(OEQB_EINVAL, "oeqb_prepare_graph: workspace of %lld bytes is smaller than the %zu required (or not 16-byte aligned)",
                    (long long)workspace_bytes, gprep::group_workspace_bytes(n_nodes, n_edges));
    std::lock_guard<std::mutex> lock(g_mutex);
    int* status = nullptr;
    if (int rc = status_word(&status)) return rc;
    cudaStream_t st = (cudaStream_t)stream;
    long long launches = 0;
    bool ok;
    // pass 1: by (row, col) -> order, sorted rows / cols; pass 2: the sorted list by (col, row) -> transpose_perm
    if (idx_dtype == 3) {
        ok = gprep::group_by_key<int>((const int*)rows, (const int*)cols, n_edges, n_nodes, (int*)order, (int*)sorted_rows,
                                      (int*)sorted_cols, workspace, status, st, nullptr, &launches) &&
             gprep::group_by_key<int>((const int*)sorted_cols, (const int*)sorted_rows, n_edges, n_nodes, (int*)transpose_perm,
                                      nullptr, nullptr, workspace, status, st, nullptr, &launches);
    } else {
        ok = gprep::group_by_key<long long>((const long long*)rows, (const long long*)cols, n_edges, n_nodes, (long long*)order,
                                            (long long*)sorted_rows, (long long*)sorted_cols, workspace, status, st, nullptr, &launches) &&
             gprep::group_by_key<long long>((const long long*)sorted_cols, (const long long*)sorted_rows, n_edges, n_nodes,
                                            (long long*)transpose_perm, nullptr, nullptr, workspace, status, st, nullptr, &launches);
    }
    g_launches.fetch_add(launches, std::memory_order_relaxed);
    if (!ok) return fail(OEQB_ECUDA, "oeqb_prepare_graph: kernel launch failed: %s", cudaGetErrorString(cudaGetLastError()));
    return OEQB_OK;
}

namespace {
int plan_bounds(const char* who, int32_t world, const int64_t* bounds, int64_t n_nodes, pplan::Bounds* B) {
    if (world < 1 || world > pplan::MAX_WORLD) return fail(OEQB_EINVAL, "%s: world must be 1 ... %d", who, pplan::MAX_WORLD);
    B->world = world;
    for (int q = 0; q <= world; ++q) {
        B->b[q] = bounds ? bounds[q] : (q == 0 ? 0 : n_nodes);
        if (B->b[q] < 0 || B->b[q] > n_nodes || (q > 0 && B->b[q] < B->b[q - 1])) return fail(OEQB_EINVAL, "%s: bounds must ascend within [0, n_nodes]", who);
    }
    return OEQB_OK;
}
}  // namespace

int64_t oeqb_plan_workspace_bytes(int64_t n_nodes, int64_t n_edges, int64_t n_receivers, int64_t n_owned, int32_t world) {
    if (n_nodes < 0 || n_edges < 0 || n_receivers < 0 || n_owned < 0 || world < 1) return -(int64_t)fail(OEQB_EINVAL, "oeqb_plan_workspace_bytes: bad argument");
    return (int64_t)pplan::layout(n_nodes, n_edges, n_receivers, n_owned, world).total;
}

int oeqb_plan_count(int64_t n_nodes, int64_t n_edges, const void* rows, const void* cols, int64_t recv_begin, int64_t recv_end,
                    int64_t own_begin, int64_t own_end, int32_t world, int32_t rank, const int64_t* bounds, void* workspace,
                    int64_t workspace_bytes, int64_t* counts, void* stream) {
    pplan::Bounds B;
    if (int rc = plan_bounds("oeqb_plan_count", world, bounds, n_nodes, &B)) return rc;
    if (n_nodes < 0 || n_edges < 0 || recv_begin < 0 || recv_end < recv_begin || recv_end > n_nodes || own_begin < 0 || own_end < own_begin ||
        own_end > n_nodes || rank < 0 || rank >= world)
        return fail(OEQB_EINVAL, "oeqb_plan_count: bad range");
    if (int rc = check_ptrs({workspace, counts}, "oeqb_plan_count")) return rc;
    if (n_edges > 0) if (int rc = check_ptrs({rows, cols}, "oeqb_plan_count")) return rc;
    const size_t need = pplan::layout(n_nodes, n_edges, recv_end - recv_begin, own_end - own_begin, world).total;
    if (workspace_bytes < (int64_t)need || ((uintptr_t)workspace & 15u))
        return fail(OEQB_EINVAL, "oeqb_plan_count: workspace of %lld bytes is smaller than the %zu required (or not 16-byte aligned)",
                    (long long)workspace_bytes, need);
    long long launches = 0;
    const bool ok = pplan::count((const long long*)rows, (const long long*)cols, n_nodes, n_edges, recv_begin, recv_end, own_begin, own_end, B,
                                 rank, workspace, (long long*)counts, (cudaStream_t)stream, &launches);
    g_launches.fetch_add(launches, std::memory_order_relaxed);
    if (!ok) return fail(OEQB_ECUDA, "oeqb_plan_count: %s", cudaGetErrorString(cudaGetLastError()));
    return OEQB_OK;
}

int oeqb_plan_fill(int64_t n_nodes, int64_t n_edges, const void* rows, const void* cols, int64_t recv_begin, int64_t recv_end,
                   int64_t own_begin, int64_t own_end, int32_t world, const int64_t* bounds, int64_t e0, int64_t e1, int64_t n_halo,
                   void* workspace, int64_t workspace_bytes, void* halo_ids, void* send_ids, void* rows_local, void* cols_local,
                   void* perm_local, void* stream) {
    pplan::Bounds B;
    if (int rc = plan_bounds("oeqb_plan_fill", world, bounds, n_nodes, &B)) return rc;
    if (e0 < 0 || e1 < e0 || e1 > n_edges || n_halo < 0 || n_halo > n_nodes) return fail(OEQB_EINVAL, "oeqb_plan_fill: bad sizes");
    if (int rc = check_ptrs({workspace}, "oeqb_plan_fill")) return rc;
    if (e1 > e0) if (int rc = check_ptrs({rows, cols, rows_local, cols_local, perm_local}, "oeqb_plan_fill")) return rc;
    const size_t need = pplan::layout(n_nodes, n_edges, recv_end - recv_begin, own_end - own_begin, world).total;
    if (workspace_bytes < (int64_t)need) return fail(OEQB_EINVAL, "oeqb_plan_fill: workspace too small");
    std::lock_guard<std::mutex> lock(g_mutex);
    int* status = nullptr;
    if (int rc = status_word(&status)) return rc;
    long long launches = 0;
    const bool ok = pplan::fill((const long long*)rows, (const long long*)cols, n_nodes, n_edges, recv_begin, recv_end, own_begin, own_end, B, e0,
                                e1, n_halo, workspace, (long long*)halo_ids, (long long*)send_ids, (long long*)rows_local,
                                (long long*)cols_local, (long long*)perm_local, status, (cudaStream_t)stream, &launches);
    g_launches.fetch_add(launches, std::memory_order_relaxed);
    if (!ok) return fail(OEQB_ECUDA, "oeqb_plan_fill: %s", cudaGetErrorString(cudaGetLastError()));
    return OEQB_OK;
}

int oeqb_group_mm(int dtype, int ragged_inner, int64_t num_groups, int64_t num_features, int64_t M, int64_t K,
                  const int64_t* ragged_counts, const void* A, const void* B, void* C, void* stream) {
    if (dtype != 1 && dtype != 2) return fail(OEQB_EINVAL, "oeqb_group_mm: dtype must be 1 (float32) or 2 (float64)");
    if (ragged_inner < 0 || ragged_inner > 2) return fail(OEQB_EINVAL, "oeqb_group_mm: ragged_inner must be 0, 1 or 2");
    if (num_groups < 0 || num_features < 0 || M < 0 || K < 0) return fail(OEQB_EINVAL, "oeqb_group_mm: negative size");
    if (num_groups > gmm::MAX_GROUPS) return fail(OEQB_EUNSUPPORTED, "oeqb_group_mm: at most %d groups", gmm::MAX_GROUPS);
    if (K > 64) return fail(OEQB_EUNSUPPORTED, "oeqb_group_mm: K = %lld exceeds 64", (long long)K);
    if (num_features > 65535) return fail(OEQB_EUNSUPPORTED, "oeqb_group_mm: more than 65535 feature channels");
    if (num_groups == 0 || num_features == 0 || (M == 0 && ragged_inner != 2)) return OEQB_OK;
    if (!ragged_counts) return fail(OEQB_EINVAL, "oeqb_group_mm: null ragged_counts");
    gmm::Offsets offs;
    offs.n_groups = (int)num_groups;
    offs.off[0] = 0;
    for (int64_t g = 0; g < num_groups; ++g) {
        if (ragged_counts[g] < 0) return fail(OEQB_EINVAL, "oeqb_group_mm: negative group size");
        offs.off[g + 1] = offs.off[g] + ragged_counts[g];
    }
    const long long n_nodes = offs.off[num_groups];
    cudaStream_t st = (cudaStream_t)stream;
    const size_t elt = dtype == 2 ? 8 : 4;
    if (ragged_inner == 1) {
        // groups without nodes keep zeros; the kernel writes every row of a non-empty group
        if (int rc = check_ptrs({C}, "oeqb_group_mm")) return rc;
        if (K == 0) return OEQB_OK;
    }
    if (n_nodes == 0) {
        if (ragged_inner == 1) CUDA_TRY(cudaMemsetAsync(C, 0, (size_t)num_groups * num_features * M * K * elt, st));
        return OEQB_OK;
    }
    if (int rc = check_ptrs({A, B, C}, "oeqb_group_mm")) return rc;
    if (ragged_inner == 2) {
        if (K == 0) return OEQB_OK;
        if (M == 0) { CUDA_TRY(cudaMemsetAsync(C, 0, (size_t)n_nodes * num_features * K * elt, st)); return OEQB_OK; }
    }
    if (K == 0) { CUDA_TRY(cudaMemsetAsync(C, 0, (size_t)n_nodes * num_features * M * elt, st)); return OEQB_OK; }
    cudaError_t ce = dtype == 2 ? gmm::dispatch<double>(ragged_inner, offs, n_nodes, num_features, (int)M, (int)K, A, B, C, st)
                                : gmm::dispatch<float>(ragged_inner, offs, n_nodes, num_features, (int)M, (int)K, A, B, C, st);
    if (ce != cudaSuccess) return fail(OEQB_ECUDA, "oeqb_group_mm: kernel launch failed: %s", cudaGetErrorString(ce));
    g_launches.fetch_add(1, std::memory_order_relaxed);
    return OEQB_OK;
}

extern "C++" {
namespace {
struct SymTerm { int w, i, j, k; };
struct SymPlan {
    int G, F, ell, n_out, out_dim;
    uint64_t key;
    symc::Sets sets;
    int out_col[symc::MAX_OUT], out_stride[symc::MAX_OUT];
    // chunks of the weight gradient's terms: at most 56 (28 doubles) running sums per thread
    int chunks(int dtype) const { return (sets.terms + (dtype == 2 ? 28 : 56) - 1) / (dtype == 2 ? 28 : 56); }
    int chunk(int dtype) const { return (sets.terms + chunks(dtype) - 1) / chunks(dtype); }
    // slices of an element's nodes in the weight gradient: sixteen warps per SM, eight nodes or more each
    int slices(int dtype, long long n) const {
        const long long warps = (long long)G * ((F + 31) / 32) * chunks(dtype);
        const long long want = (16 * 148 + warps - 1) / warps, most = n / (8LL * G) + 1;
        return (int)std::min<long long>(std::min(want, most), 64);
    }
    size_t coef_bytes(size_t elt) const { return round_up((size_t)G * ((sets.terms + 3) / 4) * F * 4 * elt); }
    size_t part_bytes(int dtype, long long n) const { return round_up((size_t)slices(dtype, n) * G * sets.terms * F * (dtype == 2 ? 8 : 4)); }
};

int symcon_plan(const int32_t* meta, int n_meta, SymPlan* p) {
    if (!meta || n_meta < 9) return fail(OEQB_EINVAL, "oeqb_symcon: bad meta");
    memset(p, 0, sizeof *p);
    p->G = meta[0]; p->F = meta[1]; p->ell = meta[2]; p->n_out = meta[3]; p->sets.n_sets = meta[4];
    p->out_dim = meta[5]; p->sets.terms = meta[6]; p->sets.F = p->F;
    p->key = (uint64_t)(uint32_t)meta[7] | (uint64_t)(uint32_t)meta[8] << 32;
    if (p->G < 1 || p->G > gmm::MAX_GROUPS || p->F < 1 || p->F > 65535 || p->ell < 1 || p->ell > symc::MAX_ELL || p->n_out < 1 || p->n_out > symc::MAX_OUT ||
        p->sets.n_sets < 1 || p->sets.n_sets > symc::MAX_SETS || p->sets.terms < 1 || p->sets.terms > symc::MAX_TERMS ||
        n_meta < 9 + 2 * p->sets.n_sets + 2 * p->n_out)
        return fail(OEQB_EINVAL, "oeqb_symcon: bad meta");
    const int32_t* m = meta + 9;
    int rows = 0, u = 0;
    for (int s = 0; s < p->sets.n_sets; ++s) {
        p->sets.k[s] = *m++;
        p->sets.t0[s] = rows;
        rows += *m++;
        p->sets.t1[s] = rows;
        p->sets.u[s] = u;
        if (p->sets.k[s] < 0 || rows < p->sets.t0[s]) return fail(OEQB_EINVAL, "oeqb_symcon: bad meta");
        u += p->sets.k[s] * (rows - p->sets.t0[s]);
    }
    if (rows != p->sets.terms) return fail(OEQB_EINVAL, "oeqb_symcon: bad meta");
    for (int w = 0; w < p->n_out; ++w) { p->out_col[w] = *m++; p->out_stride[w] = *m++; }
    return OEQB_OK;
}

// The straight-line code of kernels/sym_poly.cuh for one list of terms (sorted: first order, then by the first two factors, by
// component, by the third factor).
std::string emit_sym(const SymPlan& p, int dtype, const SymTerm* t) {
    std::ostringstream s;
    const int n = p.sets.terms, ell = p.ell, chunk = p.chunk(dtype), chunks = p.chunks(dtype);
    s << "typedef " << (dtype == 2 ? "double" : "float") << " T;\n#define OEQ_DEV __device__ __forceinline__\n"
      << "constexpr int ELL = " << ell << ", NOUT = " << p.n_out << ", TERMS = " << n << ", QUADS = " << (n + 3) / 4 << ", CHUNK = " << chunk
      << ", CHUNKS = " << chunks << ";\nstruct __align__(16) T4 { T x, y, z, w; };\n";
    const char comp[4] = {'x', 'y', 'z', 'w'};
    auto coef = [&](int q) { return "c" + std::to_string(q / 4) + "." + comp[q % 4]; };
    auto load = [&](int q) { if (q % 4 == 0) s << "  const T4 c" << q / 4 << " = c[" << q / 4 << "];\n"; };
    for (int grad = 0; grad < 2; ++grad) {
        if (!grad) s << "OEQ_DEV void sym_eval(const T (&x)[ELL], const T4* c, T (&P)[NOUT]) {\n  for (int w = 0; w < NOUT; ++w) P[w] = T(0);\n";
        else s << "OEQ_DEV void sym_grad(const T (&x)[ELL], const T (&cot)[NOUT], const T4* c, T (&dx)[ELL]) {\n";
        for (int q = 0; q < n;) {
            if (t[q].j == ell) {
                load(q);
                if (!grad) s << "  P[" << t[q].w << "] = fma(" << coef(q) << ", x[" << t[q].i << "], P[" << t[q].w << "]);\n";
                else s << "  dx[" << t[q].i << "] = fma(cot[" << t[q].w << "], " << coef(q) << ", dx[" << t[q].i << "]);\n";
                ++q;
                continue;
            }
            const int i = t[q].i, j = t[q].j, pair = q;
            s << "  const T xx" << pair << " = x[" << i << "] * x[" << j << "];\n";
            if (grad) s << "  T s" << pair << " = T(0);\n";
            while (q < n && t[q].i == i && t[q].j == j) {
                const int w = t[q].w, at = q;
                s << "  T r" << at << " = T(0);\n";
                if (grad) s << "  const T g" << at << " = cot[" << w << "] * xx" << pair << ";\n";
                for (; q < n && t[q].i == i && t[q].j == j && t[q].w == w; ++q) {
                    load(q);
                    if (t[q].k == ell) { s << "  r" << at << " += " << coef(q) << ";\n"; continue; }
                    s << "  r" << at << " = fma(" << coef(q) << ", x[" << t[q].k << "], r" << at << ");";
                    if (grad) s << " dx[" << t[q].k << "] = fma(" << coef(q) << ", g" << at << ", dx[" << t[q].k << "]);";
                    s << "\n";
                }
                if (!grad) s << "  P[" << w << "] = fma(xx" << pair << ", r" << at << ", P[" << w << "]);\n";
                else s << "  s" << pair << " = fma(cot[" << w << "], r" << at << ", s" << pair << ");\n";
            }
            if (grad)
                s << "  dx[" << i << "] = fma(s" << pair << ", x[" << j << "], dx[" << i << "]); dx[" << j << "] = fma(s" << pair << ", x[" << i
                  << "], dx[" << j << "]);\n";
        }
        s << "}\n";
    }
    s << "template <int N> struct SymChunk;\n";
    for (int c = 0; c < chunks; ++c) {
        s << "template <> struct SymChunk<" << c << "> { static OEQ_DEV void add(const T (&x)[ELL], const T (&cot)[NOUT], T (&m)[CHUNK]) {\n";
        for (int q = c * chunk; q < n && q < (c + 1) * chunk; ++q) {
            const int at = q - c * chunk;
            const bool fresh = at == 0 || t[q].i != t[q - 1].i || t[q].j != t[q - 1].j || t[q].w != t[q - 1].w;
            if (t[q].j == ell) { s << "  m[" << at << "] = fma(cot[" << t[q].w << "], x[" << t[q].i << "], m[" << at << "]);\n"; continue; }
            if (at == 0 || t[q].i != t[q - 1].i || t[q].j != t[q - 1].j)
                s << "  const T xx" << t[q].i << "_" << t[q].j << " = x[" << t[q].i << "] * x[" << t[q].j << "];\n";
            if (fresh) s << "  const T g" << t[q].i << "_" << t[q].j << "_" << t[q].w << " = cot[" << t[q].w << "] * xx" << t[q].i << "_" << t[q].j << ";\n";
            s << "  m[" << at << "] ";
            if (t[q].k == ell) s << "+= g" << t[q].i << "_" << t[q].j << "_" << t[q].w << ";\n";
            else s << "= fma(g" << t[q].i << "_" << t[q].j << "_" << t[q].w << ", x[" << t[q].k << "], m[" << at << "]);\n";
        }
        s << "} };\n";
    }
    return s.str();
}

std::map<std::pair<uint64_t, int>, std::unique_ptr<Program>> g_sym_programs;   // by (key of the terms, dtype)

// Takes g_mutex, and leaves it while it compiles (about a second per hundred terms): the other operators of the process go on.
int symcon_program(const SymPlan& p, int dtype, const int32_t* terms, Program** out) {
    const std::pair<uint64_t, int> key{p.key, dtype};
    auto known = [&] {
        std::lock_guard<std::mutex> lock(g_mutex);
        auto it = g_sym_programs.find(key);
        if (it != g_sym_programs.end()) *out = it->second.get();
        return it != g_sym_programs.end();
    };
    if (known()) return OEQB_OK;
    std::lock_guard<std::mutex> compiling(g_compile_mutex);
    if (known()) return OEQB_OK;
    if (int rc = check_ptrs({terms}, "oeqb_symcon")) return rc;
    const SymTerm* t = (const SymTerm*)terms;
    for (int q = 0; q < p.sets.terms; ++q)
        if (t[q].w < 0 || t[q].w >= p.n_out || t[q].i < 0 || t[q].i >= p.ell || t[q].j < t[q].i || t[q].j > p.ell || t[q].k < t[q].j || t[q].k > p.ell)
            return fail(OEQB_EINVAL, "oeqb_symcon: bad term");
    auto fresh = std::make_unique<Program>();
    if (int rc = load_program(emit_sym(p, dtype, t) + K_COMMON + K_SYM_POLY, "symmetric_contraction", fresh.get())) return rc;
    std::lock_guard<std::mutex> lock(g_mutex);
    *out = (g_sym_programs[key] = std::move(fresh)).get();
    return OEQB_OK;
}

struct SymParams {
    const int* group; long long n;
    int G, F, out_dim, slices;
    const void* x; const void* cot; const void* coef;
    void* out; void* dx; void* part;
    int out_cols[2 * symc::MAX_OUT];   // n_out columns, then n_out strides (the kernel's arrays have exactly n_out entries)
};
SymParams symcon_params(const SymPlan& p, const int32_t* group, long long n) {
    SymParams a{};
    a.group = group; a.n = n; a.G = p.G; a.F = p.F; a.out_dim = p.out_dim;
    for (int w = 0; w < p.n_out; ++w) { a.out_cols[w] = p.out_col[w]; a.out_cols[p.n_out + w] = p.out_stride[w]; }
    return a;
}
int symcon_launch(Program* prog, const char* name, dim3 grid, unsigned block, SymParams& a, cudaStream_t st) {
    cudaKernel_t k;
    if (int rc = get_kernel(prog, name, 0, &k)) return rc;
    void* args[] = {&a};
    return launch(k, grid, block, 0, args, st);
}
// Caller holds g_mutex.
int symcon_group(const int64_t* keys, long long n, int G, int32_t* group, cudaStream_t st) {
    int* status = nullptr;
    if (int rc = status_word(&status)) return rc;
    CUDA_TRY(symc::run_group((const long long*)keys, n, G, group, status, gprep::STATUS_BAD_INDEX, st));
    g_launches.fetch_add(1, std::memory_order_relaxed);
    return OEQB_OK;
}
// as SYM_WPB in kernels/sym_poly.cuh
unsigned symcon_wpb(const SymPlan& p, size_t elt) { return 8 * (size_t)((p.sets.terms + 3) / 4) * 4 * elt <= 48000 ? 8 : 1; }
}  // namespace
}

int64_t oeqb_symcon_group_ints(int64_t n_nodes, int64_t n_elements) {
    if (n_nodes < 0 || n_elements < 1 || n_elements > gmm::MAX_GROUPS) return -(int64_t)fail(OEQB_EINVAL, "oeqb_symcon_group_ints: bad size");
    return symc::group_ints(n_nodes, (int)n_elements);
}

int64_t oeqb_symcon_bytes(int dtype, const int32_t* meta, int n_meta, int direction, int64_t n_nodes) {
    if ((dtype != 1 && dtype != 2) || n_nodes < 0) return -(int64_t)fail(OEQB_EINVAL, "oeqb_symcon_bytes: bad argument");
    SymPlan p;
    if (int rc = symcon_plan(meta, n_meta, &p)) return -(int64_t)rc;
    return (int64_t)(direction == 0 ? p.coef_bytes(dtype == 2 ? 8 : 4) : p.part_bytes(dtype, n_nodes));
}

int oeqb_symcon_compare(int n, const void* const* a, const void* const* b, const int64_t* bytes, int32_t* changed, void* stream) {
    if (n < 0 || n > symc::MAX_SETS) return fail(OEQB_EINVAL, "oeqb_symcon_compare: bad size");
    if (int rc = check_ptrs({a, b, bytes}, "oeqb_symcon_compare")) return rc;
    symc::Pairs p{};
    for (int i = 0; i < n; ++i) {
        if (bytes[i] < 0 || bytes[i] % 4) return fail(OEQB_EINVAL, "oeqb_symcon_compare: bad size");
        if (bytes[i] == 0) continue;
        if (int rc = check_ptrs({a[i], b[i]}, "oeqb_symcon_compare")) return rc;
        p.a[p.n] = (const unsigned*)a[i];
        p.b[p.n] = (const unsigned*)b[i];
        p.words[p.n++] = bytes[i] / 4;
    }
    std::lock_guard<std::mutex> lock(g_mutex);
    int* status = nullptr;
    if (int rc = status_word(&status)) return rc;
    cudaStream_t st = (cudaStream_t)stream;
    if (p.n == 0) return OEQB_OK;
    CUDA_TRY(changed ? symc::run_compare(p, changed, 1, st) : symc::run_compare(p, status, symc::STATUS_CHANGED, st));
    g_launches.fetch_add(1, std::memory_order_relaxed);
    return OEQB_OK;
}

int oeqb_symcon_group(int64_t n_nodes, int64_t n_elements, const int64_t* keys, int32_t* group, void* stream) {
    if (n_nodes < 0 || n_nodes > (1LL << 30) || n_elements < 1 || n_elements > gmm::MAX_GROUPS) return fail(OEQB_EINVAL, "oeqb_symcon_group: bad size");
    if (n_nodes == 0) return OEQB_OK;
    if (int rc = check_ptrs({keys, group}, "oeqb_symcon_group")) return rc;
    std::lock_guard<std::mutex> lock(g_mutex);
    return symcon_group(keys, n_nodes, (int)n_elements, group, (cudaStream_t)stream);
}

int oeqb_symcon_forward(int dtype, const int32_t* meta, int n_meta, const int32_t* terms, const int32_t* place, const void* U, int64_t n_nodes,
                        const int64_t* keys, const void* x, const void* const* weights, int32_t* group, void* coef, void* out, void* stream) {
    if (dtype != 1 && dtype != 2) return fail(OEQB_EINVAL, "oeqb_symcon_forward: dtype must be 1 (float32) or 2 (float64)");
    SymPlan p;
    if (int rc = symcon_plan(meta, n_meta, &p)) return rc;
    if (n_nodes == 0) return OEQB_OK;
    if (n_nodes < 0 || n_nodes > (1LL << 30)) return fail(OEQB_EINVAL, "oeqb_symcon_forward: bad size");
    if (int rc = check_ptrs({place, U, x, weights, group, coef, out}, "oeqb_symcon_forward")) return rc;
    if (!aligned16({x, coef})) return fail(OEQB_EINVAL, "oeqb_symcon_forward: x is not 16-byte aligned");
    Program* prog;
    if (int rc = symcon_program(p, dtype, terms, &prog)) return rc;
    std::lock_guard<std::mutex> lock(g_mutex);
    p.sets.place = place;
    symc::Pointers w{};
    for (int s = 0; s < p.sets.n_sets; ++s) w.p[s] = (void*)weights[s];
    cudaStream_t st = (cudaStream_t)stream;
    if (keys)
        if (int rc = symcon_group(keys, n_nodes, p.G, group, st)) return rc;
    CUDA_TRY(dtype == 2 ? symc::run_coefficients<double>(p.sets, p.G, (const double*)U, w, (double*)coef, st)
                        : symc::run_coefficients<float>(p.sets, p.G, (const float*)U, w, (float*)coef, st));
    g_launches.fetch_add(1, std::memory_order_relaxed);
    SymParams a = symcon_params(p, group, n_nodes);
    a.x = x; a.coef = coef; a.out = out;
    const unsigned wpb = symcon_wpb(p, dtype == 2 ? 8 : 4);
    return symcon_launch(prog, "oeq_sym_forward", dim3((unsigned)symc::max_tiles(n_nodes, p.G), (p.F + wpb - 1) / wpb), 32 * wpb, a, st);
}

int oeqb_symcon_backward(int dtype, const int32_t* meta, int n_meta, const int32_t* terms, const int32_t* place, const void* U, int64_t n_nodes,
                         const int32_t* group, const void* coef, const void* x, const void* cot, void* workspace, void* dx,
                         void* const* dweights, void* stream) {
    if (dtype != 1 && dtype != 2) return fail(OEQB_EINVAL, "oeqb_symcon_backward: dtype must be 1 (float32) or 2 (float64)");
    SymPlan p;
    if (int rc = symcon_plan(meta, n_meta, &p)) return rc;
    if (n_nodes < 0 || n_nodes > (1LL << 30)) return fail(OEQB_EINVAL, "oeqb_symcon_backward: bad size");
    const size_t elt = dtype == 2 ? 8 : 4;
    cudaStream_t st = (cudaStream_t)stream;
    if (int rc = check_ptrs({dweights}, "oeqb_symcon_backward")) return rc;
    if (n_nodes == 0) {
        for (int s = 0; s < p.sets.n_sets; ++s) if (p.sets.k[s] > 0) CUDA_TRY(cudaMemsetAsync(dweights[s], 0, (size_t)p.G * p.sets.k[s] * p.F * elt, st));
        return OEQB_OK;
    }
    if (int rc = check_ptrs({place, U, group, coef, x, cot, workspace, dx}, "oeqb_symcon_backward")) return rc;
    if (!aligned16({x, coef, dx})) return fail(OEQB_EINVAL, "oeqb_symcon_backward: an operand is not 16-byte aligned");
    Program* prog;
    if (int rc = symcon_program(p, dtype, terms, &prog)) return rc;
    std::lock_guard<std::mutex> lock(g_mutex);
    p.sets.place = place;
    symc::Pointers dw{};
    for (int s = 0; s < p.sets.n_sets; ++s) dw.p[s] = dweights[s];
    SymParams a = symcon_params(p, group, n_nodes);
    a.x = x; a.cot = cot; a.coef = coef; a.dx = dx; a.part = workspace;
    a.slices = p.slices(dtype, n_nodes);
    const unsigned wpb = symcon_wpb(p, elt);
    if (int rc = symcon_launch(prog, "oeq_sym_backward_x", dim3((unsigned)symc::max_tiles(n_nodes, p.G), (p.F + wpb - 1) / wpb), 32 * wpb, a, st)) return rc;
    if (int rc = symcon_launch(prog, "oeq_sym_backward_c", dim3((unsigned)(((long long)p.G * ((p.F + 31) / 32) * a.slices + 3) / 4), (unsigned)p.chunks(dtype)), 128, a, st)) return rc;
    CUDA_TRY(dtype == 2 ? symc::run_gradient_w<double>(p.sets, p.G, (const double*)U, (const double*)workspace, a.slices, dw, st)
                        : symc::run_gradient_w<float>(p.sets, p.G, (const float*)U, (const float*)workspace, a.slices, dw, st));
    g_launches.fetch_add(1, std::memory_order_relaxed);
    return OEQB_OK;
}

int oeqb_noalloc_status(void) {
    std::lock_guard<std::mutex> lock(g_mutex);
    void* base = nullptr;
    if (int rc = noalloc_scratch(&base)) return rc;
    int code = 0;
    // 4 bytes out of the built-in array into a stack variable: a copy, not an allocation
    CUDA_TRY(cudaMemcpy(&code, (char*)base + (size_t)OEQB_NOALLOC_SCRATCH_BYTES - kAlign, sizeof(int), cudaMemcpyDeviceToHost));
    if (code != 0)
        return fail(OEQB_EKERNEL, "oeqb_conv_backward_noalloc: a kernel of the last call on this device gave up a bounded "
                                  "wait (code %d); its outputs are invalid", code);
    return OEQB_OK;
}

}  // extern "C"
