// FP64 element-matrix contraction on the FP64 tensor cores (DMMA).
//
// The element matrices of one group are K[e][p] = sum_q M[p][q] C[q][e]
// (src/formulation/contribution.cpp:200-210 with densemat::multiply,
// src/densemat.cpp:228-310), M[(i,j)][(t,g)] = T_t[o][i][g] * D_t[o][j][g].
// Here the product is computed as K^T = C^T M^T, element rows by entry
// columns, with mma.sync.m16n8k8.f64 (FP64 operands, FP64 accumulation; the
// FP64 tensor path of sm_100a -- tcgen05 has no FP64 kind).
//
//  * M^T of every orientation is built once per group and form
//    (k_build_mt, [norient][Qpad][rpad], zero outside Q x nrows) and stays
//    resident; its columns are the group's computed rows: every entry, or,
//    for the mirrored forms, the rows of a row map (upper triangle of a
//    symmetric group, or every entry of a group whose transposed partner is
//    written by the same launch).
//  * A block computes 64 elements x BP rows (BP = 128 or 64, picked per group
//    shape by timing); 8 warps of 32 elements x up to BP/32 MMA tiles of 8
//    rows.  The tiles of a row tile go round its four warps, starting at
//    another one in each block, and those behind the last row are left out:
//    the last row tile of 136 rows (order-3 quadrangles) has 8 of them, of
//    378 and 729 (order-2 hexahedra) 122 and 97.
//    K advances 16 at a time through a 3-stage cp.async ring of C^T and M^T
//    tiles in shared memory (rows padded to 68 and BP + 4 doubles so that the
//    fragment loads of a half-warp hit distinct banks).
//  * The finished tile is staged in shared memory and stored as whole 32-byte
//    sectors (one 4-value store per thread), at the entries and, for the
//    mirrored forms, at their mirrors (same matrix or the partner's), by a
//    list of stores per bin of rows.  Stored straight from the fragments, 8
//    bytes at a time, most sectors were written in parts, each part about as
//    dear as ten whole sectors (149 x 149 order-3 quadrangles: 50 -> 46 us).
#pragma once

#include "engine_internal.h"

#include <cstdint>

namespace slgpu {

constexpr int kMmaBE = 64;    // elements per block
constexpr int kMmaBPMax = 128;  // most rows (entries) per block; M^T rows are padded to it
constexpr int kMmaBQ = 16;    // (term, Gauss point) pairs per stage
constexpr int kMmaStages = 3;
constexpr int kMmaCS = kMmaBE + 4;  // C^T tile row stride (doubles)
constexpr int kMmaBin = 64;         // rows that stores take together

// One store: the values of 4 rows of a bin (-1: zero) at `place` .. place + 3
// of an element matrix of out, or of out2; where rows are not on sectors, one
// value.
struct StoreOp {
    int32_t place, mirror;
    int16_t src[4];
};
template <int BP>
struct MmaShape {
    static constexpr int MS = BP + 4;  // M^T tile row stride (doubles)
    static constexpr int StageDoubles = kMmaBQ * (kMmaCS + MS);
    static constexpr size_t Smem = (size_t)kMmaStages * StageDoubles * sizeof(double);
    static constexpr int NT = BP / 32;  // 8-row MMA tiles per warp
    static constexpr int OS = BP + 8;   // row stride of the staged tile [element][row]
    static_assert((size_t)kMmaBE * OS * sizeof(double) <= Smem, "the staged tile reuses the ring");
};

struct BuildMtParams {
    const double* tables;
    const int64_t* tab_off;
    const int32_t* term_tf;
    const int32_t* term_dof;
    const int32_t* rowentry;  // entry of each row (-1: a zero row); nullptr: row r is entry r
    int nterms, ngp, ntf, ndof, norient, nrows, Qpad, rpad;
    double* Mt;          // [norient][Qpad][rpad]
};

// M^T[o][q][r] = T_t[o][i][g] * D_t[o][j][g] for q = t*ngp + g < Q and
// r < nrows (entry p = i*ndof + j of row r), 0 elsewhere.
__global__ void k_build_mt(BuildMtParams p)
{
    const int64_t n = (int64_t)p.norient * p.Qpad * p.rpad;
    const int Q = p.nterms * p.ngp;
    for (int64_t idx = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; idx < n; idx += (int64_t)gridDim.x * blockDim.x) {
        const int r = (int)(idx % p.rpad);
        const int64_t oq = idx / p.rpad;
        const int q = (int)(oq % p.Qpad);
        const int o = (int)(oq / p.Qpad);
        double v = 0.0;
        const int pe = r >= p.nrows ? -1 : p.rowentry != nullptr ? p.rowentry[r] : r;
        if (q < Q && pe >= 0) {
            const int t = q / p.ngp, g = q - t * p.ngp;
            const int i = pe / p.ndof, j = pe - i * p.ndof;
            const double tv = p.tables[p.tab_off[p.term_tf[t]] + ((int64_t)o * p.ntf + i) * p.ngp + g];
            const int dt = p.term_dof[t];
            const double dv = dt >= 0 ? p.tables[p.tab_off[dt] + ((int64_t)o * p.ndof + j) * p.ngp + g] : 1.0;
            v = tv * dv;
        }
        p.Mt[idx] = v;
    }
}

// One group of a launch.
struct MmaGroup {
    const double* Mt;    // [norient][Qpad][rpad]
    const double* C;     // [Q][nelem]
    const Tile* tiles;   // orientation-uniform element runs of at most 64
    const StoreOp* ops;      // stores of each bin of kMmaBin rows
    const int32_t* opstart;  // [rpad / kMmaBin + 1]
    int sectors;             // stores of 4 values, on sectors
    int Q, Qpad, rpad;
    int es, es2;         // values per element matrix of out, of out2
    int nrt;             // row tiles of BP
    int rows;            // rows up to the last one that holds an entry
    int w0;              // first block of the group in the launch
    int64_t nelem;
    double* out;         // [nelem][es]
    double* out2;        // where the mirrors go, [nelem][es2]: out, or the transposed partner's matrices
};

// Groups of one launch, by value: one launch for every FP64 group of a step,
// whose last wave of blocks is then the only one that is not full (order-2
// elasticity, 27^3 hexahedra: six launches of 924 and 1848 blocks on 296
// places; the six contractions together 1.52 -> 1.35 ms).
constexpr int kMmaBatch = 24;
struct MmaParams {
    MmaGroup g[kMmaBatch];
    int ngroups;
};

__device__ __forceinline__ void cp_async8(double* dst, const double* src, bool valid)
{
    const unsigned d = (unsigned)__cvta_generic_to_shared(dst);
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;\n" ::"r"(d), "l"(src), "r"(valid ? 8 : 0) : "memory");
}

__device__ __forceinline__ void cp_async16(double* dst, const double* src)
{
    const unsigned d = (unsigned)__cvta_generic_to_shared(dst);
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(d), "l"(src) : "memory");
}

__device__ __forceinline__ void dmma_16x8x8(double (&c)[4], const double (&a)[4], const double (&b)[2])
{
    asm volatile(
        "mma.sync.aligned.m16n8k8.row.col.f64.f64.f64.f64 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};\n"
        : "+d"(c[0]), "+d"(c[1]), "+d"(c[2]), "+d"(c[3])
        : "d"(a[0]), "d"(a[1]), "d"(a[2]), "d"(a[3]), "d"(b[0]), "d"(b[1]));
}

template <int BP>
__global__ void __launch_bounds__(256, 2) k_contract_f64mma(const __grid_constant__ MmaParams pb)
{
    using Sh = MmaShape<BP>;
    constexpr int NT = Sh::NT;
    extern __shared__ double sm_mma[];
    int gi = 0;
    while (gi + 1 < pb.ngroups && (int)blockIdx.x >= pb.g[gi + 1].w0) gi++;
    const MmaGroup& p = pb.g[gi];
    const int rt = ((int)blockIdx.x - p.w0) % p.nrt;
    const Tile tile = p.tiles[((int)blockIdx.x - p.w0) / p.nrt];
    const int r0 = rt * BP;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int gid = lane >> 2, tig = lane & 3;
    // The warp's 32 elements, and its MMA tiles: rows 32 n + 8 wr .. + 7 for n < nt.
    const int we = warp >> 2, wr = (warp + (int)blockIdx.x) & 3;
    const int live = min(p.rows - r0, BP), nt = max(0, (live - 8 * wr + 31) >> 5);
    const double* Mt = p.Mt + (int64_t)tile.orient * p.Qpad * p.rpad + r0;
    const int nchunks = p.Qpad / kMmaBQ;

    auto stage_C = [&](int s) { return sm_mma + (int64_t)s * Sh::StageDoubles; };
    auto stage_M = [&](int s) { return sm_mma + (int64_t)s * Sh::StageDoubles + kMmaBQ * kMmaCS; };
    auto load = [&](int chunk, int s) {
        const int q0 = chunk * kMmaBQ;
        double* Cs = stage_C(s);
        double* Ms = stage_M(s);
#pragma unroll
        for (int k = 0; k < (kMmaBQ * kMmaBE) / 256; k++) {
            const int idx = tid + 256 * k;
            const int row = idx / kMmaBE, col = idx % kMmaBE;
            const bool valid = q0 + row < p.Q && col < tile.ne;
            const double* src = valid ? p.C + (int64_t)(q0 + row) * p.nelem + tile.e0 + col : p.C;
            cp_async8(Cs + row * kMmaCS + col, src, valid);
        }
#pragma unroll
        for (int k = 0; k < (kMmaBQ * BP) / (2 * 256); k++) {
            const int idx = tid + 256 * k;
            const int row = idx / (BP / 2), c2 = idx % (BP / 2);
            if (2 * c2 < ((live + 7) & ~7))
                cp_async16(Ms + row * Sh::MS + 2 * c2, Mt + (int64_t)(q0 + row) * p.rpad + 2 * c2);
        }
    };

    double acc[2][NT][4];
#pragma unroll
    for (int m = 0; m < 2; m++)
#pragma unroll
        for (int n = 0; n < NT; n++)
#pragma unroll
            for (int k = 0; k < 4; k++) acc[m][n][k] = 0.0;

    // Prologue: the first kMmaStages - 1 chunks in flight (one commit group each).
#pragma unroll
    for (int s = 0; s < kMmaStages - 1; s++) {
        if (s < nchunks)
            load(s, s);
        asm volatile("cp.async.commit_group;\n" ::: "memory");
    }
    for (int c = 0; c < nchunks; c++) {
        asm volatile("cp.async.wait_group %0;\n" ::"n"(kMmaStages - 2) : "memory");
        __syncthreads();  // chunk c landed for every thread; chunk c-1's stage is free
        const int nxt = c + kMmaStages - 1;
        if (nxt < nchunks)
            load(nxt, nxt % kMmaStages);
        asm volatile("cp.async.commit_group;\n" ::: "memory");
        const double* Cs = stage_C(c % kMmaStages);
        const double* Ms = stage_M(c % kMmaStages);
#pragma unroll
        for (int ks = 0; ks < kMmaBQ; ks += 8) {
            if (c * kMmaBQ + ks >= p.Q)
                break;  // the last chunk's second half holds padding alone
            double a[2][4], b[NT][2];
#pragma unroll
            for (int m = 0; m < 2; m++) {
                const int e = we * 32 + m * 16 + gid;
                a[m][0] = Cs[(ks + tig) * kMmaCS + e];
                a[m][1] = Cs[(ks + tig) * kMmaCS + e + 8];
                a[m][2] = Cs[(ks + tig + 4) * kMmaCS + e];
                a[m][3] = Cs[(ks + tig + 4) * kMmaCS + e + 8];
            }
            if (nt == NT) {
#pragma unroll
                for (int n = 0; n < NT; n++) {
                    const int r = n * 32 + wr * 8 + gid;
                    b[n][0] = Ms[(ks + tig) * Sh::MS + r];
                    b[n][1] = Ms[(ks + tig + 4) * Sh::MS + r];
                }
#pragma unroll
                for (int m = 0; m < 2; m++)
#pragma unroll
                    for (int n = 0; n < NT; n++) dmma_16x8x8(acc[m][n], a[m], b[n]);
            } else {
#pragma unroll
                for (int n = 0; n < NT - 1; n++) {
                    if (n >= nt)
                        break;
                    const int r = n * 32 + wr * 8 + gid;
                    b[n][0] = Ms[(ks + tig) * Sh::MS + r];
                    b[n][1] = Ms[(ks + tig + 4) * Sh::MS + r];
#pragma unroll
                    for (int m = 0; m < 2; m++) dmma_16x8x8(acc[m][n], a[m], b[n]);
                }
            }
        }
    }
    asm volatile("cp.async.wait_group 0;\n" ::: "memory");
    __syncthreads();  // the ring is free

    // Fragment (m, n): elements e = base + gid (+8), rows r = base + 2 tig (+1).
#pragma unroll
    for (int m = 0; m < 2; m++)
#pragma unroll
        for (int h = 0; h < 2; h++) {
            const int e = we * 32 + m * 16 + gid + 8 * h;
#pragma unroll
            for (int n = 0; n < NT; n++)
                *reinterpret_cast<double2*>(sm_mma + e * Sh::OS + n * 32 + wr * 8 + 2 * tig) =
                    make_double2(acc[m][n][2 * h], acc[m][n][2 * h + 1]);
        }
    __syncthreads();
    // Each warp stores every eighth element; a lane keeps its store for all
    // of them.
#pragma unroll
    for (int bin = 0; bin < BP / kMmaBin; bin++) {
        const int o1 = p.opstart[r0 / kMmaBin + bin + 1];
        const double* st = sm_mma + bin * kMmaBin;
        for (int o = p.opstart[r0 / kMmaBin + bin] + lane; o < o1; o += 32) {
            const StoreOp op = p.ops[o];
            const int es = op.mirror ? p.es2 : p.es;
            double* dst = (op.mirror ? p.out2 : p.out) + (int64_t)tile.e0 * es + op.place;
            if (p.sectors) {
                for (int e = warp; e < tile.ne; e += 8) {
                    double v[4];
#pragma unroll
                    for (int k = 0; k < 4; k++) v[k] = op.src[k] >= 0 ? st[e * Sh::OS + op.src[k]] : 0.0;
                    asm volatile("st.global.v4.f64 [%0], {%1, %2, %3, %4};" ::"l"(dst + (int64_t)e * es), "d"(v[0]), "d"(v[1]), "d"(v[2]),
                                 "d"(v[3])
                                 : "memory");
                }
            } else {
                for (int e = warp; e < tile.ne; e += 8) dst[(int64_t)e * es] = st[e * Sh::OS + op.src[0]];
            }
        }
    }
}

}  // namespace slgpu
