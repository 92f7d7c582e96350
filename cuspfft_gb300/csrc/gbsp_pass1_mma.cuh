// gbsp_pass1_mma.cuh -- pass 1 as a contraction on the tensor cores.
//
// A Bluestein row of a tile that starts at u0 is written u = u0 + i + 128*d
// (i < 128), so that
//   S[u][c] = sum_{r in column c} W^{(i - 64)*r} * W^{(u0 + 64 + 128*d)*r}
// is, for one column, the product of a (rows i) x (nonzeros) and a
// (nonzeros) x (blocks d) complex matrix: one table lookup per (i, r) and per
// (d, r) instead of one per (u, r), and W^{-e*r} is the conjugate of W^{e*r}.  As a real product, A[i] = [ar, ai] per
// nonzero and B has the two rows [br, -bi] (real part) and [bi, br]
// (imaginary part) per d: M = 128 i, N = 2 * d, K = 2 per nonzero.
//
// Every factor is an FP32 table entry, split into three FP16 parts
// w = h + m + l: h to 2^-7, m to 2^-18, l the rest (all times 64, so that l
// keeps its bits).  The h*h products are multiples of 2^-14, so their FP32
// accumulation in TMEM, whose rounding is not to nearest, is exact while a
// partial sum stays below 1024.  A rounded factor is at most 1 + 2^-7.5 long,
// so that holds for any sum of up to 1012 nonzeros; columns of more than 1024
// (MM_MAX_DEGREE) take the FP32 kernel, and between the two a sum past 1024,
// which has 2^-13 as its own FP32 step, is cut to that step in the last one or
// two K-steps (at most 6e-8 of it each).  The products h*m, m*h, m*m, h*l, l*h
// go to a second accumulator, 2^-8 as large on random rows and at most 7 where
// all of a column's factors are rounded the same way, which its rounding
// shifts by 8e-8 of the sum at worst (m*l and l*l are below 2^-26 each).  What
// is left is the rounding of the two table entries: on columns of 2 to 1000
// nonzeros the sums are 2-4e-8 (relative L2) from FP64, where FP32 sums of
// recurrence twiddles are 0.9-1.3e-7.
//
// A row's split depends on its tile only through u0 mod 128, so tiles that
// start at a multiple of 128 rows give the same bits as one tile.
//
// One persistent CTA per SM, 22 warps.  Work item: a window of columns x a
// block of up to 128 * 32 rows: 4 columns x 32 d, 8 x 16 or 16 x 8, whose
// accumulators (two per column) fill TMEM.
//   warps 0-11   look up, split and store the operands of a chunk in shared
//                memory (two stages)
//   warps 12-19  write an item's results, while the next item's first two
//                chunks are made
//   warp 20      takes items from the queue and fills chunk descriptors (up to
//                four K-steps of eight nonzeros): the plan holds the row
//                indices, as fractions of the circle, padded to whole K-steps
//                per column, so a chunk is one bulk copy
//   warp 21      issues the MMAs, those that share an A part in a row, so that
//                A stays in the collector buffer
// No pipe is full (8219^2 on GB300: LSU data pipe 49 %, instruction issue
// 38 %, tensor pipe 12 %, DRAM the S write alone):
// a CTA is a chain of operands, MMA and epilogue, and shared memory is its
// longest link, so: operands are K-major without
// swizzle (8 x 16-byte core matrices, K halves 2 KB (A) or 1 KB (B) apart), a
// thread's four nonzeros one 16-byte conflict-free store per part; and table
// entry p sits at p ^ (p / 16 % 16), because the lookups i*r of consecutive i
// step by r and an even step would meet few banks (conflicts 3x on average).
// The lanes of a warp write 32 consecutive rows of S, a thread's four columns
// of a row as one 32-byte store (rows 32 apart, one page each, were 2x slower
// on 40421 columns).  Against the FP32 kernel on GB300: 8219^2 0.34 -> 0.24 ms,
// 16706^2 1.19 -> 0.68, 40421^2 4.5 -> 2.31, 70001 x 1201 1.21 -> 0.47.
#pragma once
#include <cuda_fp16.h>
#include "gbsp_kernels.cuh"

namespace gbsp {

constexpr int MM_GEN_WARPS = 12;
constexpr int MM_EPI_WARPS = 8;
constexpr int MM_PRODUCER = MM_GEN_WARPS + MM_EPI_WARPS, MM_ISSUER = MM_PRODUCER + 1;
constexpr int MM_THREADS = (MM_ISSUER + 1) * 32;
constexpr int MM_MAXWIN = 16;     // columns per item
constexpr int MM_MAXD = 32;       // blocks d an item can hold
constexpr int MM_BLOCKD = 32;     // ... and does
constexpr int MM_ROWS = 128;      // rows i (M of the MMA)
constexpr int MM_KSTEPS = 4;      // K-steps (8 nonzeros each) per chunk
constexpr int MM_STAGES = 2;
constexpr int MM_DESCS = 8;
constexpr int MM_ITEMS = 16;      // item records in flight (more than descriptors + 1)
constexpr int MM_A_BYTES = MM_ROWS * 32;       // one part of A, one K-step
constexpr int MM_B_BYTES = 2 * MM_MAXD * 32;   // one part of B, one K-step
constexpr int MM_KSTEP_BYTES = 3 * (MM_A_BYTES + MM_B_BYTES);
constexpr int MM_STAGE_BYTES = MM_KSTEPS * MM_KSTEP_BYTES;
constexpr int MM_MAX_DEGREE = 1024;          // nonzeros of a column (h*h sums exact up to 1012, see above)
constexpr uint32_t MM_PAD = 0xffffffffu;     // no fraction of rows < 2^31
constexpr float MM_SCALE = 64.f;             // table entries in shared memory
constexpr float MM_UNSCALE = 1.f / (MM_SCALE * MM_SCALE);
constexpr int MM_TMEM_COLS = 512;
constexpr long long MM_WAIT_CLOCKS = 2000000000ll;  // a wait gives up after about a second

GBSP_HD constexpr size_t p1_mma_smem_bytes(size_t ntab) {
    return (size_t)MM_STAGES * MM_STAGE_BYTES + ((ntab + 15) & ~(size_t)15) * 8;
}

// One matrix's inputs for one tile of Bluestein rows [u0, u0 + tile_rows).
struct P1MmaArgs {
    const uint32_t* kfrac;  // ceil(r * 2^32 / rows) per nonzero, each column padded to whole K-steps (MM_PAD)
    const int* kptr;        // first K-step of every column, padded to whole windows of MM_MAXWIN, + 1
    const float2* row_tab;  // in layout `gtab` (FULL, HALF or TWO), at least as fine as `tab`
    const float2* chirp;    // nullptr: raw column sums
    float2* S;
    size_t s_pitch;
    int gtab, tab, ntab, cols, s_cols, rows, u0, tile_rows;
    int nfull, nd_rest;     // row blocks: nfull of MM_MAXD * 128 rows, then one of nd_rest * 128
    int step_full, step_rest;  // columns per item in these
    uint32_t magic;
    unsigned long long magic64;
    unsigned int* queue;    // [0] next item, [1] CTAs done (zeroed by the last one out)
    int* err;
};

// Row blocks of 32 d, and what is left as one smaller block with a wider
// window (8219 rows: 32 d + 14 rows; two equal blocks would look every A up
// twice).
GBSP_HD constexpr int p1_mma_win(int nd) { return nd <= 8 ? 16 : nd <= 16 ? 8 : 4; }
GBSP_HD inline int p1_mma_windows(int s_cols, int step) { return (s_cols + step - 1) / step; }
GBSP_HD inline long p1_mma_items(const P1MmaArgs& a) {
    return (long)a.nfull * p1_mma_windows(a.s_cols, a.step_full) +
           (a.nd_rest ? p1_mma_windows(a.s_cols, a.step_rest) : 0);
}
// A window's nonzeros are one SM's chain, so with fewer items than SMs (`sms`)
// a window takes fewer columns than it holds, the widest first: down to four,
// the epilogue's 32-byte stores, or to one where the chain is longer than the
// stores (from 32 nonzeros a column, `degree`) or there is an SM for each.
// GB300, all columns a window holds and fewer: 12001 rows x 64 columns of 200
// nonzeros 81 -> 25 us, 4097 x 64 of 24 16 -> 14; 8001 x 300 of 100 33 -> 29
// (of 4, with two columns a window, 16 -> 19).
GBSP_HD inline void p1_mma_tiling(P1MmaArgs* a, int sms, int degree) {
    const int nd = (a->tile_rows + MM_ROWS - 1) / MM_ROWS;
    a->nfull = nd / MM_BLOCKD;
    a->nd_rest = nd % MM_BLOCKD;
    const int least = (degree >= 32 || (a->nfull + 1) * a->s_cols <= sms) ? 1 : 4;
    a->step_full = a->nfull ? p1_mma_win(MM_BLOCKD) : least;
    a->step_rest = a->nd_rest ? p1_mma_win(a->nd_rest) : least;
    for (;;) {
        P1MmaArgs b = *a;
        int& step = b.step_rest >= b.step_full ? b.step_rest : b.step_full;
        if (step <= least) return;
        step /= 2;
        if (p1_mma_items(b) > sms) return;
        *a = b;
    }
}

// ---------------------------------------------------------------------------
// tcgen05 helpers (inline PTX)
// ---------------------------------------------------------------------------
namespace tc {
__device__ __forceinline__ void alloc(uint32_t* dst, uint32_t cols) {  // whole warp
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(dst)), "r"(cols)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void dealloc(uint32_t addr, uint32_t cols) {  // the same warp
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(addr), "r"(cols) : "memory");
}
__device__ __forceinline__ void fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
// arrives on bar when every MMA this thread has issued is complete
__device__ __forceinline__ void commit(uint64_t* bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_u32(bar))
                 : "memory");
}
// shared-memory matrix descriptor, K-major, no swizzle: lbo = bytes between
// the two 16-byte K halves, 128 bytes between groups of eight rows
__device__ __forceinline__ uint64_t smem_desc(uint32_t addr, uint32_t lbo) {
    return (uint64_t)(addr >> 4) | ((uint64_t)(lbo >> 4) << 16) | ((uint64_t)(128 >> 4) << 32) | (1ull << 46);
}
// FP16 x FP16 -> FP32, both operands K-major, M = 128, N a multiple of 16
__device__ __forceinline__ uint32_t idesc(int n) {
    return (1u << 4) | ((uint32_t)(n / 8) << 17) | ((uint32_t)(MM_ROWS / 16) << 24);
}
// COLL: what becomes of A's collector buffer
enum Coll { FILL, USE, LASTUSE, DISCARD };
template <Coll COLL>
__device__ __forceinline__ void mma(uint32_t d, uint64_t a, uint64_t b, uint32_t id, bool accumulate) {
#define GBSP_TC_MMA(op)                                                                                      \
    asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.u32 p, %4, 0;\n\t"                                         \
                 "tcgen05.mma.cta_group::1.kind::f16.collector::a::" op " [%0], %1, %2, %3, p;\n\t}" ::"r"(d), \
                 "l"(a), "l"(b), "r"(id), "r"((uint32_t)accumulate)                                          \
                 : "memory")
    if constexpr (COLL == FILL) GBSP_TC_MMA("fill");
    else if constexpr (COLL == USE) GBSP_TC_MMA("use");
    else if constexpr (COLL == LASTUSE) GBSP_TC_MMA("lastuse");
    else GBSP_TC_MMA("discard");
#undef GBSP_TC_MMA
}
__device__ __forceinline__ bool elect() {  // one lane of the warp, the same every time
    uint32_t ok;
    asm volatile("{\n\t.reg .pred p;\n\telect.sync _|p, 0xffffffff;\n\tselp.u32 %0, 1, 0, p;\n\t}" : "=r"(ok));
    return ok != 0;
}
// four consecutive FP32 columns of this warp's 32 lanes
__device__ __forceinline__ void ld4(float (&v)[4], uint32_t addr) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x4.b32 {%0, %1, %2, %3}, [%4];"
                 : "=f"(v[0]), "=f"(v[1]), "=f"(v[2]), "=f"(v[3])
                 : "r"(addr));
}
__device__ __forceinline__ void wait_ld() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }
}  // namespace tc

__device__ __forceinline__ void mbar_arrive(uint64_t* bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}
// a try_wait that sleeps for up to a millisecond (spinning warps would take
// issue slots from the working ones)
__device__ __forceinline__ bool mm_try_wait(uint64_t* bar, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2, %3;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(smem_u32(bar)), "r"(parity), "r"(1000000u)
        : "memory");
    return ok != 0;
}
// true when the phase completed; false after MM_WAIT_CLOCKS, or as soon as
// another warp has given up (then *dead is set and every role stops)
__device__ __forceinline__ bool mm_wait(uint64_t* bar, uint32_t parity, volatile int* dead) {
    if (mm_try_wait(bar, parity)) return true;
    const long long t0 = clock64();
    for (uint32_t i = 1;; i++) {
        if (mm_try_wait(bar, parity)) return true;
        if (i % 8 == 0 && (*dead || clock64() - t0 > MM_WAIT_CLOCKS)) break;
    }
    *dead = 1;
    return false;
}
// the same for a whole warp, whose lanes go on or stop together
__device__ __forceinline__ bool mm_wait_warp(uint64_t* bar, uint32_t parity, volatile int* dead) {
    return __all_sync(0xffffffffu, mm_wait(bar, parity, dead));
}

// One chunk: up to MM_KSTEPS K-steps of one item.
struct __align__(16) MmDesc {
    uint32_t fr[MM_KSTEPS * 8];
    int nk, mat, item, flags, cstride;
    uint32_t kcode;              // a byte per K-step: its column, + MM_MAXWIN on the column's first
};
constexpr int MM_FIRST = 1, MM_LAST = 2, MM_END = 4;

struct MmItem {
    float2 chirp[MM_MAXWIN];  // times MM_UNSCALE
    float2* S;                // first row, first column
    size_t s_pitch;
    int ub;                   // B's phases are (ub + 128 * d) * r
    int na, nd, win, rows_left, ncol, used, vec;  // used: bit j = column j has nonzeros
};

struct MmShared {
    MmDesc desc[MM_DESCS];
    MmItem item[MM_ITEMS];
    uint64_t desc_full[MM_DESCS], desc_empty[MM_DESCS];
    uint64_t gen_full[MM_STAGES], stage_empty[MM_STAGES];
    uint64_t acc_full, acc_empty, tab_ready, drain;
    uint32_t tmem;
    int dead, n_items;  // n_items: how many items there were, once known
};

// The three FP16 parts of a scaled table entry, as (re, im) pairs.
struct MmSplit {
    uint32_t h, m, l;
};
__device__ __forceinline__ uint32_t mm_pack(float2 v) {
    const __half2 p = __floats2half2_rn(v.x, v.y);
    return *reinterpret_cast<const uint32_t*>(&p);
}
__device__ __forceinline__ MmSplit mm_split(float2 w) {
    // adding and subtracting 1.5 * 2^23 * step rounds to a multiple of step
    const float2 M1 = make_float2(1.5f * 4194304.f, 1.5f * 4194304.f);  // step 2^-1  (2^-7 unscaled)
    const float2 N1 = make_float2(-M1.x, -M1.y);
    const float2 M2 = make_float2(1.5f * 2048.f, 1.5f * 2048.f);        // step 2^-12 (2^-18 unscaled)
    const float2 N2 = make_float2(-M2.x, -M2.y);
    const float2 neg = make_float2(-1.f, -1.f);
    const float2 h = __fadd2_rn(__fadd2_rn(w, M1), N1);
    const float2 r = __ffma2_rn(h, neg, w);
    const float2 m = __fadd2_rn(__fadd2_rn(r, M2), N2);
    const float2 l = __ffma2_rn(m, neg, r);
    return MmSplit{mm_pack(h), mm_pack(m), mm_pack(l)};
}

struct MmMat {  // what operand generation needs of a matrix
    uint32_t rows, magic, hr;
    unsigned long long magic64;
    int tab;
};

// W^p from the table (see row_twiddle for the layouts), times MM_SCALE
__device__ __forceinline__ uint32_t mm_slot(uint32_t p) { return p ^ ((p >> 4) & 15u); }
template <int TAB>
__device__ __forceinline__ float2 mm_twiddle(const float2* tab, uint32_t p, uint32_t rows, uint32_t hr) {
    if (TAB == TAB_FULL) return tab[mm_slot(p)];
    if (TAB == TAB_TWO) return cmul(tab[mm_slot(TWO_LO + (p >> TWO_LO_BITS))], tab[mm_slot(p & (TWO_LO - 1))]);
    const bool hi = p > hr;
    float2 w = tab[mm_slot(hi ? rows - p : p)];
    w.y = hi ? -w.y : w.y;
    return w;
}

// Operands of warp-task (v, g): vector v of the chunk (four nonzeros: K-step
// v/2, K half v%2); g = 0: the d of B, g = 1: rows 64 -+ e of A, e = 33 + lane,
// g = 2: e = 1 + lane.  Row 64 (e = 0) takes the place of row 128.
//
// Phases: with f = ceil(r * 2^32 / rows), x * f mod 2^32 is the fraction of
// the circle of x * r, too large by less than x, so its product with rows has
// (x * r) mod rows as its high word while x * rows < 2^32: always for A
// (x <= 64), and for B (x < rows) unless BIG.
template <int TAB, bool BIG>
__device__ __forceinline__ void mm_gen(const MmDesc& d, const MmItem& it, const MmMat& mt, const float2* tab,
                                       unsigned char* stage, int v, int g, int lane) {
    const uint4 f = *reinterpret_cast<const uint4*>(&d.fr[4 * v]);
    const uint32_t f4[4] = {f.x, f.y, f.z, f.w};
    const int e = (g == 1 ? MM_ROWS / 4 + 1 : 1) + lane;
    const int lo = MM_ROWS / 2 - e, up = e == MM_ROWS / 2 ? e : MM_ROWS / 2 + e;
    if (g == 0 ? lane >= it.nd : lo >= it.na) return;
    const uint32_t u = g == 0 ? mod_magic((uint32_t)(it.ub + MM_ROWS * lane), mt.rows, mt.magic) : (uint32_t)e;
    // padding looks some entry up and is zeroed afterwards: no branch keeps
    // the four lookups apart
    MmSplit s[4];
#pragma unroll
    for (int i = 0; i < 4; i++) {
        uint32_t p;
        if (BIG && g == 0) p = mulmod_rows<true>(u, __umulhi(f4[i], mt.rows), mt.rows, mt.magic, mt.magic64);
        else p = __umulhi(u * f4[i], mt.rows);
        s[i] = mm_split(mm_twiddle<TAB>(tab, p, mt.rows, mt.hr));
    }
    if (f4[3] == MM_PAD) {  // a column's last vector
#pragma unroll
        for (int i = 0; i < 4; i++)
            if (f4[i] == MM_PAD) s[i] = MmSplit{0u, 0u, 0u};
    }
    unsigned char* ks = stage + (v >> 1) * MM_KSTEP_BYTES;
    constexpr uint32_t SG = 0x80000000u;
    if (g != 0) {
        uint4* a = reinterpret_cast<uint4*>(ks + (v & 1) * (MM_A_BYTES / 2));
        constexpr int PART = MM_A_BYTES / 16;
        a[lo] = make_uint4(s[0].h ^ SG, s[1].h ^ SG, s[2].h ^ SG, s[3].h ^ SG);
        a[lo + PART] = make_uint4(s[0].m ^ SG, s[1].m ^ SG, s[2].m ^ SG, s[3].m ^ SG);
        a[lo + 2 * PART] = make_uint4(s[0].l ^ SG, s[1].l ^ SG, s[2].l ^ SG, s[3].l ^ SG);
        if (up >= it.na) return;
        if (up == MM_ROWS / 2) {
            const uint32_t one = mm_pack(make_float2(MM_SCALE, 0.f));
#pragma unroll
            for (int i = 0; i < 4; i++) s[i] = MmSplit{f4[i] != MM_PAD ? one : 0u, 0u, 0u};
        }
        a[up] = make_uint4(s[0].h, s[1].h, s[2].h, s[3].h);
        a[up + PART] = make_uint4(s[0].m, s[1].m, s[2].m, s[3].m);
        a[up + 2 * PART] = make_uint4(s[0].l, s[1].l, s[2].l, s[3].l);
    } else {
        // row 2d: (br, -bi); row 2d+1: (bi, br)
        uint4* b = reinterpret_cast<uint4*>(ks + 3 * MM_A_BYTES + (v & 1) * (MM_B_BYTES / 2)) + 2 * lane;
        auto put = [&](uint32_t x0, uint32_t x1, uint32_t x2, uint32_t x3) {
            b[0] = make_uint4(x0 ^ SG, x1 ^ SG, x2 ^ SG, x3 ^ SG);
            b[1] = make_uint4(__byte_perm(x0, 0u, 0x1032), __byte_perm(x1, 0u, 0x1032), __byte_perm(x2, 0u, 0x1032),
                              __byte_perm(x3, 0u, 0x1032));
            b += MM_B_BYTES / 16;
        };
        put(s[0].h, s[1].h, s[2].h, s[3].h);
        put(s[0].m, s[1].m, s[2].m, s[3].m);
        put(s[0].l, s[1].l, s[2].l, s[3].l);
    }
}

// TMEM -> S: a warp reads the TMEM lanes of its quarter (rows i), in sixteen
// units of four columns x two blocks d; it takes units x0, x0 + 2, ...
__device__ __forceinline__ void mm_epilogue(const MmItem& it, uint32_t tmem, int quarter, int x0, int lane) {
    const int i0 = quarter * 32;
    const uint32_t base = tmem + ((uint32_t)i0 << 16);
    const int nq = MM_MAXWIN / (it.win / 4);    // units per four columns: 16, 8 or 4
    const int cstride = MM_TMEM_COLS / it.win;  // TMEM columns of one column of the window
    float2* const S = it.S + (size_t)(i0 + lane) * it.s_pitch;
    const size_t dstep = MM_ROWS * it.s_pitch;
    const int left = it.rows_left - (i0 + lane);
    for (int x = x0; x < MM_MAXWIN; x += MM_EPI_WARPS / 4) {
        const int cg = x / nq * 4, dq = x % nq * 2;
        if (dq >= it.nd || cg >= it.ncol) continue;  // warp-uniform
        float v0[4][4], v1[4][4];  // (re, im) of two d
#pragma unroll
        for (int j = 0; j < 4; j++) {
            const uint32_t t = base + (cg + j) * cstride + 2 * dq;
            tc::ld4(v0[j], t);
            tc::ld4(v1[j], t + cstride / 2);
        }
        float2 ch[4];
#pragma unroll
        for (int j = 0; j < 4; j++) ch[j] = it.chirp[cg + j];
        tc::wait_ld();
        const bool vec = it.vec && cg + 4 <= it.ncol;
        const bool all = (it.used >> cg & 15) == 15;
        float2* dst = S + dq * dstep + cg;
#pragma unroll
        for (int i = 0; i < 2; i++, dst += dstep) {
            if (dq + i >= it.nd || (dq + i) * MM_ROWS >= left) continue;
            float2 o[4];
#pragma unroll
            for (int j = 0; j < 4; j++) {
                const float2 v = make_float2(v0[j][2 * i] + v1[j][2 * i], v0[j][2 * i + 1] + v1[j][2 * i + 1]);
                o[j] = cmul(v, ch[j]);
                if (!all && !(it.used >> (cg + j) & 1)) o[j] = make_float2(0.f, 0.f);
            }
            if (vec) {
                asm volatile("st.global.v8.f32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"l"(dst), "f"(o[0].x),
                             "f"(o[0].y), "f"(o[1].x), "f"(o[1].y), "f"(o[2].x), "f"(o[2].y), "f"(o[3].x), "f"(o[3].y)
                             : "memory");
            } else {
#pragma unroll
                for (int j = 0; j < 4; j++)
                    if (cg + j < it.ncol) dst[j] = o[j];
            }
        }
    }
}

// BATCH: args / item_begin list nmat matrices whose items share one queue
// (which must be 0 at launch); else `one` is the matrix.
template <bool BATCH>
__global__ void __launch_bounds__(MM_THREADS, 1)
k_twiddle_mma(P1MmaArgs one, const P1MmaArgs* __restrict__ args, const long* __restrict__ item_begin, int nmat,
              unsigned int* queue) {
    extern __shared__ __align__(1024) unsigned char mm_smem[];
    __shared__ MmShared sh;
    float2* tab = reinterpret_cast<float2*>(mm_smem + (size_t)MM_STAGES * MM_STAGE_BYTES);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    // the plan's table, brought to this kernel's layout
    auto load_table = [&](const P1MmaArgs& a, int tid, int nt) {
        for (int i = tid; i < a.ntab; i += nt) {
            const bool high = a.tab == TAB_TWO && i >= TWO_LO;
            int p = i;
            if (high && a.gtab != TAB_TWO) p = (int)((long long)(i - TWO_LO) * TWO_LO % a.rows);
            const bool conj = a.gtab == TAB_HALF && p > a.rows / 2;
            float2 w = a.row_tab[conj ? a.rows - p : p];
            if (conj) w.y = -w.y;
            if (a.tab != TAB_TWO || high) { w.x *= MM_SCALE; w.y *= MM_SCALE; }
            tab[mm_slot(i)] = w;
        }
    };
    pdl_trigger();
    if (!BATCH) load_table(one, threadIdx.x, MM_THREADS);
    for (int i = threadIdx.x; i < (int)((sizeof(sh.desc) + sizeof(sh.item)) / 4); i += MM_THREADS)
        reinterpret_cast<int*>(&sh)[i] = 0;
    if (threadIdx.x == 0) {
        for (int i = 0; i < MM_DESCS; i++) {
            mbar_init(&sh.desc_full[i], 1);
            mbar_init(&sh.desc_empty[i], MM_GEN_WARPS + 1);
        }
        for (int i = 0; i < MM_STAGES; i++) {
            mbar_init(&sh.gen_full[i], MM_GEN_WARPS);
            mbar_init(&sh.stage_empty[i], 1);
        }
        mbar_init(&sh.acc_full, 1);
        mbar_init(&sh.acc_empty, MM_EPI_WARPS);
        mbar_init(&sh.tab_ready, MM_GEN_WARPS);
        mbar_init(&sh.drain, 1);
        sh.dead = 0;
        sh.n_items = -1;
    }
    if (warp == MM_ISSUER) tc::alloc(&sh.tmem, MM_TMEM_COLS);
    tc::fence_before();
    pdl_wait();
    __syncthreads();
    tc::fence_after();
    const uint32_t tmem = sh.tmem;
    volatile int* dead = &sh.dead;

    if (warp == MM_PRODUCER) {
        // ---- descriptors
        const long total = BATCH ? item_begin[nmat] : p1_mma_items(one);
        // A CTA's first item is its own number, the others come from the queue.
        // Item k + 1 is taken when the operands of item k - 1 are made, no
        // earlier: the descriptors hold eight chunks, and CTAs that filled
        // them with items as soon as they started left others without any
        // (3449 rows x 1201 columns, 301 items on 152 SMs: 174 us or 221, by luck).
        struct Next {
            long it;
            int m, c0, row0, nd, step, k0, kend;
            float2 ch;
        } cur;
        int m = 0;
        auto take = [&](Next& o, long it) {
            o.it = it;
            o.m = m;
            if (o.it >= total) return;
            long first = 0;
            if (BATCH) {
                while (m + 1 < nmat && item_begin[m + 1] <= o.it) m++;
                first = item_begin[m];
                o.m = m;
            }
            const P1MmaArgs& a = BATCH ? args[m] : one;
            long i = o.it - first;
            int n_win = p1_mma_windows(a.s_cols, a.step_full);
            o.nd = MM_BLOCKD;
            o.step = a.step_full;
            o.row0 = 0;
            if (i >= (long)a.nfull * n_win) {
                i -= (long)a.nfull * n_win;
                o.nd = a.nd_rest;
                o.step = a.step_rest;
                o.row0 = a.nfull * MM_BLOCKD * MM_ROWS;
                n_win = p1_mma_windows(a.s_cols, o.step);
            }
            const int t = (int)(i / n_win);
            o.row0 += t * MM_BLOCKD * MM_ROWS;
            o.c0 = ((int)i - t * n_win) * o.step;
            const int j = min(lane, o.step - 1);
            o.k0 = a.kptr[o.c0];
            o.kend = a.kptr[o.c0 + j + 1];
            o.ch = make_float2(MM_UNSCALE, 0.f);
            if (a.chirp) {
                o.ch = o.c0 + j < a.cols ? a.chirp[o.c0 + j] : make_float2(0.f, 0.f);
                o.ch.x *= MM_UNSCALE;
                o.ch.y *= MM_UNSCALE;
            }
        };
        take(cur, blockIdx.x);
        int n = 0, items = 0;  // chunks and items written
        int before = 0;        // chunks up to the item before (its last one is before - 1)
        bool ok = true;
        while (ok && cur.it < total) {
            const P1MmaArgs& a = BATCH ? args[cur.m] : one;
            const int kend = cur.kend - cur.k0;
            const int nk = __shfl_sync(0xffffffffu, kend, 31);
            int kbeg = __shfl_up_sync(0xffffffffu, kend, 1);
            if (lane == 0) kbeg = 0;
            const unsigned used = __ballot_sync(0xffffffffu, kend > kbeg);
            const int nch = max(1, (nk + MM_KSTEPS - 1) / MM_KSTEPS);
            constexpr uint32_t kbytes = 8 * sizeof(uint32_t);
            const uint32_t* src = a.kfrac + (size_t)cur.k0 * 8;
            for (int c = 0; c < nch; c++, n++) {
                MmDesc& d = sh.desc[n % MM_DESCS];
                uint64_t* full = &sh.desc_full[n % MM_DESCS];
                if (n >= MM_DESCS && !mm_wait_warp(&sh.desc_empty[n % MM_DESCS], (n / MM_DESCS - 1) & 1, dead)) {
                    ok = false;
                    break;
                }
                if (c == 0) {
                    // (its ring slot was last used MM_ITEMS items ago, an
                    // item whose descriptors are all free again)
                    MmItem& q = sh.item[items % MM_ITEMS];
                    if (lane < MM_MAXWIN) q.chirp[lane] = cur.ch;
                    if (lane == 0) {
                        q.S = a.S + (size_t)cur.row0 * a.s_pitch + cur.c0;
                        q.s_pitch = a.s_pitch;
                        q.ub = a.u0 + cur.row0 + MM_ROWS / 2;
                        q.rows_left = a.tile_rows - cur.row0;
                        q.na = min(MM_ROWS, q.rows_left);
                        q.nd = cur.nd;
                        q.win = p1_mma_win(cur.nd);
                        q.ncol = min(cur.step, a.s_cols - cur.c0);
                        q.used = (int)used;
                        q.vec = (a.s_pitch & 3) == 0 && ((uintptr_t)a.S & 31) == 0;
                    }
                    __syncwarp();
                }
                uint32_t kcode = 0;
#pragma unroll
                for (int q = 0; q < MM_KSTEPS; q++) {
                    const int k = c * MM_KSTEPS + q;
                    const int col = __popc(__ballot_sync(0xffffffffu, kend <= k));
                    const bool beg = __any_sync(0xffffffffu, kbeg == k && kend > k);
                    kcode |= (uint32_t)((col & (MM_MAXWIN - 1)) + (beg ? MM_MAXWIN : 0)) << (8 * q);
                }
                if (lane == 0) {
                    const int n4 = min(MM_KSTEPS, nk - c * MM_KSTEPS);
                    d.nk = n4;
                    d.kcode = kcode;
                    d.cstride = MM_TMEM_COLS / p1_mma_win(cur.nd);
                    d.mat = cur.m;
                    d.item = items % MM_ITEMS;
                    d.flags = (c == 0 ? MM_FIRST : 0) | (c == nch - 1 ? MM_LAST : 0);
                    mbar_expect_tx(full, n4 * kbytes);
                    if (n4 > 0) {
                        fence_proxy_async_smem();
                        bulk_copy_g2s(d.fr, src + (size_t)c * MM_KSTEPS * 8, n4 * kbytes, full);
                    }
                }
            }
            if (!ok) break;
            items++;
            // (a slot written again since has been free in between)
            if (before > 0 && n < before + MM_DESCS &&
                !mm_wait_warp(&sh.desc_empty[(before - 1) % MM_DESCS], ((before - 1) / MM_DESCS) & 1, dead)) {
                ok = false;
                break;
            }
            before = n;
            unsigned int nx = 0;
            if (lane == 0) nx = atomicAdd(queue, 1u);
            take(cur, (long)gridDim.x + __shfl_sync(0xffffffffu, nx, 0));
        }
        // No copy may be in flight when the CTA ends.  The warps that use a
        // chunk wait for it, unless a wait gave up before.  (Before the end
        // mark, which moves its slot's barrier on by one phase more.)
        if (lane == 0) {
            int alone = 0;
            for (int k = max(0, n - MM_DESCS); k < n; k++)
                mm_wait(&sh.desc_full[k % MM_DESCS], (k / MM_DESCS) & 1, &alone);
        }
        __syncwarp();
        if (ok && n >= MM_DESCS) ok = mm_wait_warp(&sh.desc_empty[n % MM_DESCS], (n / MM_DESCS - 1) & 1, dead);
        if (ok && lane == 0) {
            sh.desc[n % MM_DESCS].flags = MM_END;
            mbar_arrive(&sh.desc_full[n % MM_DESCS]);
        }
        if (!BATCH && lane == 0) {
            // the last CTA out rearms the queue for the next launch
            __threadfence();
            if (atomicAdd(&queue[1], 1u) == gridDim.x - 1) {
                atomicExch(&queue[0], 0u);
                atomicExch(&queue[1], 0u);
            }
        }
    } else if (warp == MM_ISSUER) {
        // ---- MMA issue.  The whole warp runs the loop on uniform values (one
        // lane alone had to move every operand to a uniform register: 100
        // clocks an MMA), one elected lane issues.
        const uint32_t ring = smem_u32(mm_smem);
        int items = 0;
        for (int n = 0;; n++) {
            const int s = n % MM_STAGES;
            if (!mm_wait_warp(&sh.desc_full[n % MM_DESCS], (n / MM_DESCS) & 1, dead)) break;
            const MmDesc& d = sh.desc[n % MM_DESCS];
            const int flags = __shfl_sync(0xffffffffu, d.flags, 0), nk = __shfl_sync(0xffffffffu, d.nk, 0);
            const uint32_t kcode = __shfl_sync(0xffffffffu, d.kcode, 0);
            const uint32_t cstride = __shfl_sync(0xffffffffu, d.cstride, 0);
            if (flags & MM_END) break;
            if (lane == 0) mbar_arrive(&sh.desc_empty[n % MM_DESCS]);
            if (!mm_wait_warp(&sh.gen_full[s], (n / MM_STAGES) & 1, dead)) break;
            if ((flags & MM_FIRST) && items > 0 && !mm_wait_warp(&sh.acc_empty, (items - 1) & 1, dead)) break;
            tc::fence_after();
            if (tc::elect()) {
                const uint32_t id = tc::idesc(cstride / 2);
#pragma unroll
                for (int k = 0; k < MM_KSTEPS; k++) {
                    if (k >= nk) break;
                    const uint32_t a = ring + s * MM_STAGE_BYTES + k * MM_KSTEP_BYTES, b = a + 3 * MM_A_BYTES;
                    const uint32_t kc = kcode >> (8 * k) & 0xffu;
                    const uint32_t d0 = tmem + (kc & (MM_MAXWIN - 1)) * cstride, d1 = d0 + cstride / 2;
                    const bool acc = (kc & MM_MAXWIN) == 0;
                    const uint64_t ah = tc::smem_desc(a, MM_A_BYTES / 2);
                    const uint64_t bh = tc::smem_desc(b, MM_B_BYTES / 2);
                    const uint64_t am = ah + (MM_A_BYTES >> 4), al = am + (MM_A_BYTES >> 4);
                    const uint64_t bm = bh + (MM_B_BYTES >> 4), bl = bm + (MM_B_BYTES >> 4);
                    tc::mma<tc::FILL>(d0, ah, bh, id, acc);
                    tc::mma<tc::USE>(d1, ah, bm, id, acc);
                    tc::mma<tc::LASTUSE>(d1, ah, bl, id, true);
                    tc::mma<tc::FILL>(d1, am, bh, id, true);
                    tc::mma<tc::LASTUSE>(d1, am, bm, id, true);
                    tc::mma<tc::DISCARD>(d1, al, bh, id, true);
                }
                tc::commit(&sh.stage_empty[s]);
                if (flags & MM_LAST) tc::commit(&sh.acc_full);
            }
            __syncwarp();
            if (flags & MM_LAST) items++;
        }
        // the epilogue warps' end: one phase more, once they have seen the last
        if (items == 0 || mm_wait_warp(&sh.acc_empty, (items - 1) & 1, dead)) {
            if (lane == 0) {
                sh.n_items = items;
                mbar_arrive(&sh.acc_full);
            }
        }
        // nothing may be in flight when TMEM is released
        if (tc::elect()) {
            int alone = 0;
            tc::commit(&sh.drain);
            mm_wait(&sh.drain, 0, &alone);
        }
        __syncwarp();
    } else if (warp >= MM_GEN_WARPS) {
        // ---- epilogues
        for (int i = 0;; i++) {
            if (!mm_wait_warp(&sh.acc_full, i & 1, dead)) break;
            if (*(volatile int*)&sh.n_items == i) break;
            tc::fence_after();
            mm_epilogue(sh.item[i % MM_ITEMS], tmem, warp & 3, (warp - MM_GEN_WARPS) >> 2, lane);
            tc::fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(&sh.acc_empty);
        }
    } else {
        // ---- operands
        MmMat mt;
        int cur = -1;
        auto set_mat = [&](const P1MmaArgs& a) {
            mt.rows = (uint32_t)a.rows;
            mt.magic = a.magic;
            mt.magic64 = a.magic64;
            mt.hr = (uint32_t)a.rows / 2;
            mt.tab = a.tab + (a.rows > 65535 ? 4 : 0);
        };
        if (!BATCH) set_mat(one);
        const int g = warp % 3;
        for (int n = 0;; n++) {
            const int s = n % MM_STAGES;
            if (!mm_wait_warp(&sh.desc_full[n % MM_DESCS], (n / MM_DESCS) & 1, dead)) break;
            const MmDesc& d = sh.desc[n % MM_DESCS];
            const int flags = d.flags;
            if (flags & MM_END) break;
            if (BATCH && d.mat != cur) {
                cur = d.mat;
                // no warp may still read the table of the matrix before, and
                // none may read the new one before it is whole
                __syncwarp();
                if (lane == 0) mbar_arrive(&sh.tab_ready);
                if (!mm_wait_warp(&sh.tab_ready, 0, dead)) break;
                load_table(args[cur], threadIdx.x, MM_GEN_WARPS * 32);
                __syncwarp();
                if (lane == 0) mbar_arrive(&sh.tab_ready);
                if (!mm_wait_warp(&sh.tab_ready, 1, dead)) break;
                set_mat(args[cur]);
            }
            if (n >= MM_STAGES && !mm_wait_warp(&sh.stage_empty[s], (n / MM_STAGES - 1) & 1, dead)) break;
            // a warp keeps its part g and takes every fourth vector, from a
            // different one each chunk so that short chunks spread out
            const MmItem& it = sh.item[d.item];
            unsigned char* stage = mm_smem + (size_t)s * MM_STAGE_BYTES;
            if (g != 2 || it.na > MM_ROWS / 4) {
                for (int v = (warp / 3 + n) % (MM_GEN_WARPS / 3); v < 2 * d.nk; v += MM_GEN_WARPS / 3) {
                    switch (mt.tab) {
                        case TAB_FULL: mm_gen<TAB_FULL, false>(d, it, mt, tab, stage, v, g, lane); break;
                        case TAB_HALF: mm_gen<TAB_HALF, false>(d, it, mt, tab, stage, v, g, lane); break;
                        case TAB_TWO: mm_gen<TAB_TWO, false>(d, it, mt, tab, stage, v, g, lane); break;
                        case TAB_TWO + 4: mm_gen<TAB_TWO, true>(d, it, mt, tab, stage, v, g, lane); break;
                    }
                }
            }
            fence_proxy_async_smem();
            __syncwarp();
            if (lane == 0) {
                mbar_arrive(&sh.gen_full[s]);
                mbar_arrive(&sh.desc_empty[n % MM_DESCS]);
            }
        }
    }
    __syncthreads();
    if (warp == MM_ISSUER) {
        tc::fence_after();
        tc::dealloc(tmem, MM_TMEM_COLS);
    }
    if (threadIdx.x == 0 && *dead) atomicOr(BATCH ? args[0].err : one.err, ERR_TIMEOUT);
}

}  // namespace gbsp
