// Split-precision element contraction on the sm_100a tensor cores.
//
// V[e][p] = sum_q M[p][q] C[q][e] is evaluated with FP64 operands cut into
// INT8 slices of B bits (Ozaki scheme):
//   M[p][q] = R_p sum_a m_a[p][q] 2^-Ba      (row scale R_p, a = 1..S)
//   C[q][e] = Q_e sum_b c_b[q][e] 2^-Bb      (column scale Q_e)
//   V[e][p] ~ R_p Q_e sum_{a+b <= L} 2^-B(a+b) sum_q m_a c_b
// Each sum_q m_a c_b is an INT8 x INT8 product summed exactly in INT32 by
// tcgen05.mma (kind::i8); all pairs with the same level l = a+b accumulate
// in the same TMEM accumulator (still exact: at most S products of
// |m c| <= 2^14 per q, q <= 2^14).  The epilogue recombines the levels.
//
// Split tier: B = 8, the balanced base-256 digits -128 .. 127 of the operand
// rounded to an integer, S = 6, L = 7 (21 products).  FP32-level tier: B = 7,
// the operand truncated to signed 7-bit fields, scales the power of two above
// the largest magnitude, S = 5, L = 6 (15 products).
// A balanced digit carries a bit more than a truncated one, rounding has half
// the error of truncation, and the scale uses the largest value itself (to
// 2^-20): six balanced digits err 4 to 8 times less than seven truncated ones
// with L = 8, for 21 products instead of 28.  (Relative Frobenius error of
// the element matrices, order-2 elasticity on hexahedra / on tetrahedra /
// order-5 Helmholtz: 6.1e-14 / 1.8e-14 / 2.9e-14 against 5.0e-13 / 6.6e-14 /
// 2.1e-13.)  A step of mixed orders 1-5 on 48,000 tetrahedra, whose contraction
// the products bound: 1725 -> 1451 us.
//
// Level accumulators sit side by side in TMEM (level l at columns
// NE(l-2) .. NE(l-2)+NE-1, NE = 64 elements), and the column
// slices of one K step sit side by side in shared memory, so A slice a times
// the concatenation [c_1 | ... | c_k] (N = NE k <= 256) writes every pair
// (a, b) straight into level a+b's columns: for S = 6, 8 MMAs per K step
// instead of 21.
//
// Operands live in global memory already in the interleaved K-major layout
// that the UMMA "no swizzle" canonical form expects, blocked so that one K
// step of one tile is a single contiguous range (one bulk copy per operand):
//   A (rows of M):    [orient][ptile][kstep][slice][2][128][16 bytes]
//   B (columns of C): [tile][kstep][2][slice][NE][16 bytes]
// A core matrix (8 rows x 16 bytes) is 128 contiguous bytes; 8-row groups are
// SBO = 128 bytes apart, the two 16-byte K chunks of a step LBO bytes apart.
#pragma once

#include "engine_internal.h"
#include "split_digits.cuh"

#include <cstdint>

namespace slgpu {

constexpr int kSplitM = 128;     // element-matrix entries per tile (TMEM lanes)
constexpr int kSplitKStep = 32;  // bytes of K per pipeline stage (one MMA K)
constexpr int kSplitMaxS = 6;    // most slices per operand
constexpr int kSplitEpiWarps = 16;  // 4 per TMEM lane quarter, 16 columns each
constexpr int kSplitThreads = 64 + 32 * kSplitEpiWarps;
constexpr int kSplitABytes = 2 * kSplitM * 16;  // one slice of one K step of A

// Elements per tile: the columns of one accumulator level.  Six levels of 64
// fill 384 of the 512 TMEM columns, so there is one accumulator, and a tile's
// MMAs wait until the one before has been read.  Two accumulators of 32
// columns need no such wait, but A (the rows of M) is read twice as often and
// the MMAs are half as wide: 1.4 times slower with long K, no faster with
// short.
constexpr int kSplitNE = 64;
constexpr int kSplitStages = 6;                // shared-memory pipeline depth
constexpr int kSplitBBytes = 2 * kSplitNE * 16;  // one slice of one K step of B
constexpr int kSplitGroupB = 256 / kSplitNE;   // B slices per MMA (N <= 256)

// One group of a batched contraction launch.  Its work items are
// [w0, w0 + nwork) of the launch: item w0 + v is row tile v % ntp of element
// tile v / ntp.
struct SplitGroup {
    int Ppad, ntp, nk;      // padded rows, row tiles, K steps
    int nrows;              // rows of A computed
    int es, es2;            // values per element matrix of out, of out2
    const int2* rowmap;     // [nrows]: where row r's value goes in an element matrix of
                            // out, and its mirror in out2, or out (-1: nowhere); null:
                            // row r is value r, without a mirror
    double* out2;           // null, or the transposed partner group's element matrices
    const Tile* tiles;      // [nwork / ntp]
    const int8_t* A;        // row slices
    const int8_t* B;        // column slices
    const double* rowscale;  // [norient][Ppad]: R_p 2^(8 - B L)
    const double* colscale;  // [ntiles][64]: Q_e 2^-8 of each slot
    double* out;            // [nelem][es]
    int64_t w0, nwork;
};

// Groups of one launch (same S, L and NE), passed by value: every element
// group of a step runs in one persistent launch, whatever its entry count,
// Gauss points or element count.
constexpr int kSplitBatch = 24;
struct SplitParams {
    SplitGroup g[kSplitBatch];
    int ngroups;
    int64_t nwork;          // sum of the groups' work items
    unsigned int* error;    // set on a timed-out wait (host memory, written only then)
    unsigned long long* next;  // work items handed out after each CTA's first; zero at launch
    int f32;                // out and out2 hold floats (FP32-level steps): same entry order
};

// Work items passed from a CTA's producer to its MMA and epilogue roles.
constexpr int kSplitItems = 8;

// Group of work item w, advanced from the group of the CTA's previous item
// (a CTA's items increase, so each role walks the groups once).
__device__ __forceinline__ int split_group_of(const SplitParams& p, int gi, int64_t w)
{
    while (gi + 1 < p.ngroups && w >= p.g[gi + 1].w0) gi++;
    return gi;
}

// ---------------------------------------------------------------- slicing

// Order of K: q = g nterms + t, the terms of a Gauss point side by side (the
// slicing kernel has them in one thread).

// Row slices of M for one orientation: block per row p, threads over q.
// M[p][q] = T_t[o][i][g] * D_t[o][j][g] as in the FP64 contraction.
// Row r of A holds entry rowentry[r] of M (entry r without that array; -1: a
// zero row); rows from nrows to Ppad are zero.
struct RowSliceParams {
    const double* tables;
    const int64_t* tab_off;
    const int32_t* term_tf;
    const int32_t* term_dof;
    const int32_t* rowentry;
    int nterms, ngp, ntf, ndof, norient, Qpad, Ppad, nrows;
    int L;            // largest level
    int8_t* slices;   // [orient][ptile][kstep][S][2][128][16]
    double* rowscale; // [norient][Ppad]
};

// M[pe][q] (pe < 0: zero).
__device__ __forceinline__ double m_entry(const RowSliceParams& p, int o, int pe, int q)
{
    const int g = q / p.nterms, t = q - g * p.nterms, ngp = p.ngp;
    if (pe < 0 || g >= ngp)
        return 0.0;
    const int i = pe / p.ndof, j = pe - i * p.ndof;
    const double tv = p.tables[p.tab_off[p.term_tf[t]] + ((int64_t)o * p.ntf + i) * ngp + g];
    const int dt = p.term_dof[t];
    const double dv = dt >= 0 ? p.tables[p.tab_off[dt] + ((int64_t)o * p.ndof + j) * ngp + g] : 1.0;
    return tv * dv;
}

template <int B, int S>
__global__ void k_slice_rows(RowSliceParams p)
{
    const int pe = blockIdx.x, o = blockIdx.y;
    const int src = pe >= p.nrows ? -1 : p.rowentry != nullptr ? p.rowentry[pe] : pe;
    __shared__ int top, rounded;
    if (threadIdx.x == 0) {
        top = 0;
        rounded = 0;
    }
    // The thread's first kRowKeep entries stay in registers (Q <= 1024); later
    // ones are formed again in every pass.
    constexpr int kRowKeep = 4;
    double kept[kRowKeep];
#pragma unroll
    for (int k = 0; k < kRowKeep; k++) {
        const int q = threadIdx.x + k * blockDim.x;
        kept[k] = q < p.Qpad ? m_entry(p, o, src, q) : 0.0;
    }
    auto each = [&](auto f) {
#pragma unroll
        for (int k = 0; k < kRowKeep; k++)
            if ((int)(threadIdx.x + k * blockDim.x) < p.Qpad)
                f((int)(threadIdx.x + k * blockDim.x), kept[k]);
        for (int q = threadIdx.x + kRowKeep * blockDim.x; q < p.Qpad; q += blockDim.x) f(q, m_entry(p, o, src, q));
    };
    __syncthreads();
    // Magnitudes compare as their bit patterns (NaN above infinity).
    int mx = 0;
    each([&](int, double x) { mx = max(mx, __double2hiint(x) & 0x7fffffff); });
    atomicMax(&top, mx);
    __syncthreads();
    if constexpr (B == 8) {
        bool exact = true;
        each([&](int, double x) { exact = exact && split_exact(x, top); });
        if (!exact)
            rounded = 1;
        __syncthreads();
    }
    double unit, pre;
    const double f = split_scale<B, S>(top, B == 8 && rounded == 0, &unit, &pre);
    if (threadIdx.x == 0)
        p.rowscale[(int64_t)o * p.Ppad + pe] = ldexp(unit, 16 - B * p.L);
    const int ntp = p.Ppad / kSplitM, nk = p.Qpad / kSplitKStep;
    const int pt = pe / kSplitM, r = pe % kSplitM;
    each([&](int q, double x) {
        const unsigned long long u = split_digits<B, S>(x * pre, f);
        const int ks = q / kSplitKStep, c = (q / 16) & 1;
        for (int s = 0; s < S; s++)
            p.slices[(((((int64_t)o * ntp + pt) * nk + ks) * S + s) * 2 + c) * (kSplitM * 16) + r * 16 + (q & 15)] =
                (int8_t)((u >> (8 * (S - 1 - s))) ^ split_flip<B>());
    });
}

// Column slices of coefficients in memory: thread per (64-element tile, slot); C[q][e] is read
// once, coalesced over the tile's consecutive elements, and 16-byte chunks
// are written coalesced over slots.  The high word of each element's largest
// |C[q][e]| comes from the coefficient kernel.  Empty slots get zero slices.
// For groups whose coefficients the runtime-compiled slicing kernel
// (jit_slice_source) cannot evaluate.
struct ColSliceGroup {
    const double* C;  // [Q][nelem]
    const int32_t* elemtop;  // [nelem]; 0: no magnitude from 2^-1042 on
    const Tile* tiles;
    int nterms, ngp, Qpad;
    int64_t nelem, ntiles;
    int8_t* slices;   // [tile][kstep][2][S][64][16]
    double* colscale; // [ntiles][64]
    int64_t t0;       // first tile of the group in the launch
};

struct ColSliceParams {
    ColSliceGroup g[kSplitBatch];
    int ngroups;
    int64_t ntiles;   // sum over the groups
};

template <int B, int S>
__global__ void k_slice_cols(const __grid_constant__ ColSliceParams pb)
{
    const int64_t gt = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    const int64_t tg = gt / 64;
    const int slot = (int)(gt % 64);
    if (tg >= pb.ntiles)
        return;
    int gi = 0;
    while (gi + 1 < pb.ngroups && tg >= pb.g[gi + 1].t0) gi++;
    const ColSliceGroup& p = pb.g[gi];
    const int64_t t = tg - p.t0;
    const Tile tile = p.tiles[t];
    const bool valid = slot < tile.ne;
    const int64_t e = tile.e0 + slot;
    const double* col = p.C + e;
    const int top = valid ? p.elemtop[e] : 0;
    bool exact = B == 8 && top > 0;
    for (int64_t q = 0; exact && q < (int64_t)p.nterms * p.ngp; q++) exact = split_exact(col[q * p.nelem], top);
    double unit, pre;
    const double f = split_scale<B, S>(top, exact, &unit, &pre);
    p.colscale[t * 64 + slot] = unit;
    const int nchunk = p.Qpad / 16;
    uint4* out = reinterpret_cast<uint4*>(p.slices) + t * (int64_t)nchunk * S * kSplitNE + slot;
    for (int c = 0; c < nchunk; c++) {
        double x[16];
#pragma unroll
        for (int k = 0; k < 16; k++) {
            const int q = c * 16 + k, g = q / p.nterms, t = q - g * p.nterms;
            x[k] = valid && g < p.ngp ? col[((int64_t)t * p.ngp + g) * p.nelem] : 0.0;
        }
        uint32_t w[S][4];
#pragma unroll
        for (int k4 = 0; k4 < 4; k4++) {
            unsigned long long u[4];
#pragma unroll
            for (int k = 0; k < 4; k++) u[k] = split_digits<B, S>(pre == 1.0 ? x[4 * k4 + k] : x[4 * k4 + k] * pre, f);
            split_words<B, S>(u, w, k4);
        }
        // chunk c of K step c/2 lands at [kstep][c&1][s][slot]: (c*S + s) * NE.
#pragma unroll
        for (int s = 0; s < S; s++) out[((int64_t)c * S + s) * kSplitNE] = make_uint4(w[s][0], w[s][1], w[s][2], w[s][3]);
    }
}

// ---------------------------------------------------------------- PTX helpers

__device__ __forceinline__ uint32_t smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

__device__ __forceinline__ void mbar_init(uint64_t* bar, uint32_t count)
{
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count) : "memory");
}

__device__ __forceinline__ void mbar_expect_tx(uint64_t* bar, uint32_t bytes)
{
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes) : "memory");
}

__device__ __forceinline__ void mbar_arrive(uint64_t* bar)
{
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}

// Bounded wait for the phase with the given parity.  Gives up (false) after
// 2^22 polls, or early once another role of the CTA has recorded a failure.
__device__ __forceinline__ bool mbar_wait(uint64_t* bar, uint32_t parity, const volatile int* failed)
{
    const uint32_t a = smem_u32(bar);
    for (uint32_t it = 0; it < (1u << 22); it++) {
        uint32_t done;
        asm volatile(
            "{\n\t.reg .pred p;\n\t"
            "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
            "selp.u32 %0, 1, 0, p;\n\t}"
            : "=r"(done)
            : "r"(a), "r"(parity)
            : "memory");
        if (done)
            return true;
        if ((it & 255) == 255 && *failed)
            return false;
    }
    return false;
}

// Contiguous global -> shared copy completing on an mbarrier (16-byte
// aligned addresses, size a multiple of 16).
__device__ __forceinline__ void bulk_load(void* dst, const void* src, uint32_t bytes, uint64_t* bar)
{
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(smem_u32(dst)),
                 "l"(reinterpret_cast<uint64_t>(src)), "r"(bytes), "r"(smem_u32(bar))
                 : "memory");
}

// UMMA shared-memory descriptor, K-major, no swizzle (layout type 0), version 1.
__device__ __forceinline__ uint64_t umma_desc(uint32_t saddr, uint32_t lbo, uint32_t sbo)
{
    uint64_t d = 0;
    d |= (uint64_t)((saddr >> 4) & 0x3FFF);
    d |= (uint64_t)((lbo >> 4) & 0x3FFF) << 16;
    d |= (uint64_t)((sbo >> 4) & 0x3FFF) << 32;
    d |= (uint64_t)1 << 46;
    return d;
}

// Instruction descriptor for kind::i8: S32 accumulate, signed A and B,
// both K-major, N >> 3 at bits 17-22, M >> 4 at bits 24-28.
__host__ __device__ constexpr uint32_t umma_idesc_i8(int M, int N)
{
    return (2u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(N >> 3) << 17) | ((uint32_t)(M >> 4) << 24);
}

__device__ __forceinline__ void umma_i8(uint32_t tmem_d, uint64_t adesc, uint64_t bdesc, uint32_t idesc, uint32_t accumulate)
{
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::i8 [%0], %1, %2, %3, p;\n\t}" ::"r"(tmem_d),
        "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate)
        : "memory");
}

__device__ __forceinline__ void umma_commit(uint64_t* bar)
{
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_u32(bar)) : "memory");
}

// 8 consecutive 32-bit TMEM columns of this thread's lane (no wait).
__device__ __forceinline__ void tmem_ld8_nowait(uint32_t taddr, int32_t* r)
{
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
                 : "r"(taddr));
}

__device__ __forceinline__ void tmem_ld_wait() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }

// The NL levels r[l] of one output, most significant first, combined to
// T = sum_l r[l] 2^(B (NL - 1 - l)) with one rounding.  The last three levels
// make Lo, the others H; each is formed exactly in int64 on top of the bit
// pattern of C = 1.5 2^52, whose mantissa ulp is 1, so the patterns are the
// doubles C + H and C + Lo (no conversion instructions, which the outputs
// would saturate).  A level holds at most 6 pair products of at most
// K 2^14 each, with K <= 16384, so |r| < 2^30.6 and |H|, |Lo| < 2^47; then
// H 2^3B - C is exact, and adding C + Lo rounds once.
__device__ __forceinline__ long long mad_wide(int a, int b, long long c)
{
    long long d;
    asm("mad.wide.s32 %0, %1, %2, %3;" : "=l"(d) : "r"(a), "r"(b), "l"(c));
    return d;
}
template <int B, int NL>
__device__ __forceinline__ double split_combine(const int32_t (&r)[NL])
{
    constexpr double C = 0x1.8p52, W = (double)(1 << 3 * B);
    auto on_c = [](int32_t x) { return (long long)(((unsigned long long)(uint32_t)(0x43380000 + (x >> 31)) << 32) | (uint32_t)x); };
    const long long lo = mad_wide(r[NL - 3], 1 << 2 * B, mad_wide(r[NL - 2], 1 << B, on_c(r[NL - 1])));
    long long h = on_c(r[NL - 4]);
#pragma unroll
    for (int l = 0; l < NL - 4; l++) h = mad_wide(r[l], 1 << (B * (NL - 4 - l)), h);
    return fma(__longlong_as_double(h), W, -C * W - C) + __longlong_as_double(lo);
}

// One row's values of nj consecutive elements (es and em values apart) at
// its place and its mirror's (null: nowhere).
template <class V>
__device__ __forceinline__ void split_store(const double (&d)[16], V* out, int es, V* mirror, int em, int nj)
{
    if (out != nullptr) {
#pragma unroll
        for (int j = 0; j < 16; j++)
            if (j < nj)
                out[(int64_t)j * es] = (V)d[j];
    }
    if (mirror != nullptr) {
#pragma unroll
        for (int j = 0; j < 16; j++)
            if (j < nj)
                mirror[(int64_t)j * em] = (V)d[j];
    }
}

// ---------------------------------------------------------------- contraction

// Shared memory: pipeline stages, each one K step (32 bytes) of every A slice
// (128 rows) and every B slice (64 rows), plus barriers.
struct SplitSmem {
    alignas(1024) int8_t A[kSplitStages][kSplitMaxS * kSplitABytes];
    alignas(1024) int8_t B[kSplitStages][kSplitMaxS * kSplitBBytes];
    alignas(8) uint64_t full[kSplitStages];
    uint64_t empty[kSplitStages];
    uint64_t tmem_full, tmem_empty, drain;
    uint64_t item_full[kSplitItems], item_empty[kSplitItems];
    int64_t items[kSplitItems];
    double colscale[kSplitEpiWarps][16];  // each epilogue warp's columns of the tile at hand
    uint32_t tmem;
    int failed;
};
constexpr size_t split_smem_bytes() { return sizeof(SplitSmem) + 1024; }

// Persistent, warp-specialised kernel; one CTA per SM holds all 512 TMEM
// columns.  Work item w = (row tile w % ntp, element tile w / ntp).  Each
// CTA's first item is its index; later ones come from a global counter, so
// the items are taken in order and the CTAs working at the same time always
// hold neighbouring items: they share element tiles (B is read from L2 once
// per tile), and the 32-byte sectors that neighbouring row tiles' mirrored
// stores share are completed while they are still in L2.  (Handed out
// round-robin, the CTAs drift apart over a long launch.)  The producer
// passes each item to the MMA
// and epilogue roles through a ring of kSplitItems slots; -1 ends the CTA.
//   warp 0 (one thread): bulk copies of each K step into the stage ring;
//   warp 1 (one thread): MMAs; owns the TMEM allocation;
//   warps 2-17: epilogue; warp w reads TMEM lanes 32(w%4) .. 32(w%4)+31 and
//              16 of the 64 columns.
// Barriers: full/empty per stage (copies -> MMA -> copies), tmem_full (MMAs of a
// tile done -> epilogue) and tmem_empty (epilogue has read the accumulator ->
// MMAs of the next tile).  Every wait is bounded: on
// timeout the CTA records the failure, the roles stop, outstanding copies and
// MMAs are waited for (bounded), the TMEM is freed and the CTA returns.
template <int B, int S, int L>
__global__ void __launch_bounds__(kSplitThreads, 1) k_contract_split(const __grid_constant__ SplitParams p)
{
    constexpr int NL = L - 1;  // levels 2 .. L
    static_assert(S <= kSplitMaxS && NL <= S && NL >= 5 && NL <= 6, "level layout");
    constexpr int NE = kSplitNE, kSt = kSplitStages;
    static_assert(NL * NE <= 512, "the accumulator fits the 512 TMEM columns");
    extern __shared__ __align__(1024) unsigned char smem_raw[];
    SplitSmem& sm = *reinterpret_cast<SplitSmem*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    constexpr uint32_t kCols = 512;
    volatile int* failed = &sm.failed;

    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&sm.tmem)), "r"(kCols)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    if (tid == 0) {
        for (int s = 0; s < kSt; s++) {
            mbar_init(&sm.full[s], 1);
            mbar_init(&sm.empty[s], 1);
        }
        mbar_init(&sm.tmem_full, 1);
        mbar_init(&sm.tmem_empty, kSplitEpiWarps);
        for (int k = 0; k < kSplitItems; k++) {
            mbar_init(&sm.item_full[k], 1);
            mbar_init(&sm.item_empty[k], 1 + kSplitEpiWarps);  // MMA issuer and epilogue warps
        }
        mbar_init(&sm.drain, 1);
        sm.failed = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem = sm.tmem;
    constexpr uint32_t kABytes = S * kSplitABytes, kBBytes = S * kSplitBBytes;

    if (warp == 0 && lane == 0) {
        // ------------------------------------------------ producer
        int stage = 0;
        uint32_t phase = 0;
        uint32_t used = 0, last_parity = 0;  // per-stage bit sets
        bool ok = true;
        int gi = 0;
        int64_t w = blockIdx.x;
        for (uint32_t k = 0; ok; k++) {
            // The next work item, or -1 at the end.
            int64_t item = -1;
            if (w < p.nwork) {
                gi = split_group_of(p, gi, w);
                item = w;
            }
            const int slot = (int)(k % kSplitItems);
            if (!mbar_wait(&sm.item_empty[slot], ((k / kSplitItems) & 1) ^ 1, failed)) {
                ok = false;
                break;
            }
            sm.items[slot] = item;
            mbar_arrive(&sm.item_full[slot]);
            if (item < 0)
                break;
            w = (int64_t)atomicAdd(p.next, 1ull) + gridDim.x;  // in flight during this item's copies
            const SplitGroup& G = p.g[gi];
            const int64_t v = item - G.w0;
            const int pt = (int)(v % G.ntp);
            const int64_t u = v / G.ntp;
            const Tile unit = G.tiles[u];
            const int8_t* srcA = G.A + ((int64_t)unit.orient * G.ntp + pt) * G.nk * kABytes;
            const int8_t* srcB = G.B + u * G.nk * kBBytes;
            const int nk = G.nk;
            for (int ks = 0; ks < nk; ks++) {
                if (!mbar_wait(&sm.empty[stage], phase ^ 1, failed)) {
                    ok = false;
                    break;
                }
                mbar_expect_tx(&sm.full[stage], kABytes + kBBytes);
                bulk_load(sm.A[stage], srcA + (int64_t)ks * kABytes, kABytes, &sm.full[stage]);
                bulk_load(sm.B[stage], srcB + (int64_t)ks * kBBytes, kBBytes, &sm.full[stage]);
                used |= 1u << stage;
                last_parity = (last_parity & ~(1u << stage)) | (phase << stage);
                if (++stage == kSt) {
                    stage = 0;
                    phase ^= 1;
                }
            }
        }
        if (!ok) {
            *failed = 1;
            *(volatile unsigned int*)p.error = 1u;
        }
        // No copy may still be in flight when the CTA leaves.
        const int zero = 0;
        for (int s = 0; s < kSt; s++)
            if (used & (1u << s))
                if (!mbar_wait(&sm.full[s], (last_parity >> s) & 1, &zero))
                    *(volatile unsigned int*)p.error = 2u;
    } else if (warp == 1 && lane == 0) {
        // ------------------------------------------------ MMA issuer
        int stage = 0;
        uint32_t phase = 0;
        bool ok = true;
        int64_t i = 0;  // tiles processed by this CTA
        int gi = 0;
        for (uint32_t k = 0; ok; k++) {
            const int slot = (int)(k % kSplitItems);
            if (!mbar_wait(&sm.item_full[slot], (k / kSplitItems) & 1, failed)) {
                ok = false;
                break;
            }
            const int64_t w = sm.items[slot];
            mbar_arrive(&sm.item_empty[slot]);
            if (w < 0)
                break;
            gi = split_group_of(p, gi, w);
            const SplitGroup& G = p.g[gi];
            const int nk = G.nk;
            if (i > 0 && !mbar_wait(&sm.tmem_empty, (uint32_t)((i - 1) & 1), failed)) {
                ok = false;
                break;
            }
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            for (int ks = 0; ks < nk; ks++) {
                if (!mbar_wait(&sm.full[stage], phase, failed)) {
                    ok = false;
                    break;
                }
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                const uint32_t a_base = smem_u32(sm.A[stage]), b_base = smem_u32(sm.B[stage]);
#pragma unroll
                for (int a0 = 0; a0 < S; a0++) {
                    const int nbt = (S < L - 1 - a0) ? S : L - 1 - a0;  // b = 1 .. min(S, L - a)
                    const uint64_t ad = umma_desc(a_base + a0 * kSplitABytes, kSplitM * 16, 128);
#pragma unroll
                    for (int b0 = 0; b0 < nbt; b0 += kSplitGroupB) {
                        const int nb = (nbt - b0) < kSplitGroupB ? (nbt - b0) : kSplitGroupB;
                        const uint64_t bd = umma_desc(b_base + b0 * NE * 16, S * NE * 16, 128);
                        umma_i8(tmem + (uint32_t)(NE * (a0 + b0)), ad, bd, umma_idesc_i8(kSplitM, NE * nb),
                                (ks > 0 || a0 > 0) ? 1u : 0u);
                    }
                }
                umma_commit(&sm.empty[stage]);
                if (++stage == kSt) {
                    stage = 0;
                    phase ^= 1;
                }
            }
            if (!ok)
                break;
            umma_commit(&sm.tmem_full);
            i++;
        }
        if (!ok) {
            *failed = 1;
            *(volatile unsigned int*)p.error = 1u;
        }
        // Every MMA issued by this thread completes before the TMEM is freed.
        const int zero = 0;
        umma_commit(&sm.drain);
        if (!mbar_wait(&sm.drain, 0, &zero))
            *(volatile unsigned int*)p.error = 2u;
    } else if (warp >= 2) {
        // ------------------------------------------------ epilogue
        // Warp w reads TMEM lane quarter w % 4 and columns c0 .. c0+15 of
        // each level, 8 columns at a time; once they are in registers the
        // accumulator is released, and the rest of the recombination and the
        // stores overlap the next tile's MMAs.
        const int quarter = warp & 3;
        const int c0 = ((warp - 2) >> 2) * 16;
        const uint32_t lane_base = tmem + ((uint32_t)(quarter * 32) << 16);
        int64_t i = 0;
        int gi = 0;
        for (uint32_t k = 0;; k++) {
            const int slot = (int)(k % kSplitItems);
            if (!mbar_wait(&sm.item_full[slot], (k / kSplitItems) & 1, failed)) {
                *failed = 1;
                *(volatile unsigned int*)p.error = 1u;
                break;
            }
            const int64_t w = sm.items[slot];
            __syncwarp();
            if (lane == 0)
                mbar_arrive(&sm.item_empty[slot]);
            if (w < 0)
                break;
            gi = split_group_of(p, gi, w);
            const SplitGroup& G = p.g[gi];
            const int64_t v = w - G.w0;
            const int pt = (int)(v % G.ntp);
            const int64_t u = v / G.ntp;
            const Tile unit = G.tiles[u];
            // What the stores need from global memory is requested before the
            // accumulator is complete: a load issued after stores waits
            // behind them.
            const int pe = pt * kSplitM + quarter * 32 + lane;
            const bool live = pe < G.nrows;
            const double rsc = live ? __ldg(G.rowscale + (int64_t)unit.orient * G.Ppad + pe) : 0.0;
            const int2 m = !live ? make_int2(-1, -1) : G.rowmap != nullptr ? __ldg(G.rowmap + pe) : make_int2(pe, -1);
            if (lane < 16)
                sm.colscale[warp - 2][lane] = __ldg(G.colscale + u * NE + c0 + lane);
            __syncwarp();
            if (!mbar_wait(&sm.tmem_full, (uint32_t)(i & 1), failed)) {
                *failed = 1;
                *(volatile unsigned int*)p.error = 1u;
                break;
            }
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            const uint32_t col = lane_base + (uint32_t)c0;
            // V = R_p 2^(8 - B L) T Q_e 2^-8.
            double d[16];
#pragma unroll
            for (int h = 0; h < 16; h += 8) {
                int32_t r[NL][8];
#pragma unroll
                for (int l = 0; l < NL; l++) tmem_ld8_nowait(col + (uint32_t)(l * NE + h), r[l]);
                tmem_ld_wait();
                if (h == 8) {
                    // This warp's accumulators are in registers: release them.
                    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
                    __syncwarp();
                    if (lane == 0)
                        mbar_arrive(&sm.tmem_empty);
                }
#pragma unroll
                for (int j = 0; j < 8; j++) {
                    int32_t x[NL];
#pragma unroll
                    for (int l = 0; l < NL; l++) x[l] = r[l][j];
                    d[h + j] = split_combine<B, NL>(x) * rsc * sm.colscale[warp - 2][h + j];
                }
            }
            __syncwarp();  // every lane has read the scales before the next tile's
            const int64_t e = unit.e0 + c0;
            const int nj = min(16, unit.ne - c0);
            const int em = G.out2 != nullptr ? G.es2 : G.es;
            double* const out = m.x >= 0 ? G.out : nullptr;
            double* const mirror = m.y < 0 ? nullptr : G.out2 != nullptr ? G.out2 : G.out;
            if (p.f32) {
                // Value k of a float matrix is float k of the same buffer.
                split_store<float>(d, out != nullptr ? reinterpret_cast<float*>(out) + e * G.es + m.x : nullptr, G.es,
                                   mirror != nullptr ? reinterpret_cast<float*>(mirror) + e * em + m.y : nullptr, em, nj);
            } else {
                split_store<double>(d, out != nullptr ? out + e * G.es + m.x : nullptr, G.es,
                                    mirror != nullptr ? mirror + e * em + m.y : nullptr, em, nj);
            }
            i++;
        }
    }
    __syncthreads();
    if (warp == 1) {
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(kCols) : "memory");
    }
}

}  // namespace slgpu
