// Runtime-compiled geometry + coefficient kernels.
//
// The interpreter kernel (k_geometry_coef) walks a group's coefficient program
// instruction by instruction with its values in local memory.  Here the
// programs of all groups that share the same elements and Gauss points (the
// slices of one contribution) are turned into one straight-line CUDA kernel,
// compiled for sm_100a with NVRTC and cached by source text: the Jacobian is
// computed once per (element, Gauss point) and every program value lives in
// a register.  Results are written in the same [term][gp][element] layout.
#include "engine_internal.h"
#include "split_digits.cuh"

#include <nvrtc.h>

#include <cstdio>
#include <cstring>
#include <deque>
#include <map>
#include <mutex>
#include <sstream>
#include <stdexcept>
#include <algorithm>

namespace slgpu {

namespace {

const char* kPrelude = R"(
typedef long long i64;
struct JitGeom {
    const double* xyz;
    const int* conn;
    const int* elems;
    const int* orient;
    i64 nelem;
    const double* weights;
    const double* lagrange;
};
struct JitGroup {
    const double* tables;
    const double* elemdata;
    const double* fielddata;
    const double* term_scale;
    double* C;
    int* elemtop;
};
struct JitSlice {
    const double* tables;
    const double* elemdata;
    const double* fielddata;
    const double* term_scale;
    uint4* slices;
    double* colscale;
};
)";

std::string lit(double v)
{
    char buf[64];
    std::snprintf(buf, sizeof(buf), "(%a)", v);
    return buf;
}

}  // namespace

namespace {

// X, J, det J, the cofactor inverse I and wdet = w_g |det J| at element e,
// Gauss point g (as in src/field/jacobian.cpp:308-349, :396-504).
// Node coordinates come from the mesh, or, with `staged`, from
// xs[(3 k + c) * E + el].
void emit_geometry(std::ostringstream& s, int dim, int ncn, int ngp, const char* indent, bool staged = false)
{
    if (!staged)
        s << indent << "const int* cn = p.conn + (i64)p.elems[e] * " << ncn << ";\n";
    s << indent << "double X0 = 0, X1 = 0, X2 = 0;\n";
    for (int a = 0; a < dim; a++)
        for (int b = 0; b < dim; b++) s << indent << "double J" << a << b << " = 0;\n";
    s << indent << "#pragma unroll\n" << indent << "for (int k = 0; k < " << ncn << "; k++) {\n";
    if (staged) {
        s << indent << "  const double x0 = xs[3 * k * E + el], x1 = xs[(3 * k + 1) * E + el], x2 = xs[(3 * k + 2) * E + el];\n";
    } else {
        s << indent << "  const i64 nd = 3 * (i64)cn[k];\n";
        s << indent << "  const double x0 = p.xyz[nd], x1 = p.xyz[nd + 1], x2 = p.xyz[nd + 2];\n";
    }
    s << indent << "  const double nv = p.lagrange[k * " << ngp << " + g];\n";
    s << indent << "  X0 = fma(nv, x0, X0); X1 = fma(nv, x1, X1); X2 = fma(nv, x2, X2);\n";
    for (int a = 0; a < dim; a++) {
        s << indent << "  { const double dn = p.lagrange[(" << (1 + a) * ncn << " + k) * " << ngp << " + g];";
        for (int b = 0; b < dim; b++) s << " J" << a << b << " = fma(dn, x" << b << ", J" << a << b << ");";
        s << " }\n";
    }
    s << indent << "}\n";
    if (dim == 1) {
        s << indent << "const double det = J00;\n" << indent << "const double I00 = 1.0 / J00;\n";
    } else {
        // Cofactors by position; staged, they are divided by det J all together.
        std::vector<std::pair<std::string, std::string>> inv;
        if (dim == 2) {
            s << indent << "const double det = J00 * J11 - J01 * J10;\n";
            inv = {{"I00", "J11"}, {"I01", "-J01"}, {"I10", "-J10"}, {"I11", "J00"}};
        } else {
            s << indent << "const double det = J00 * (J11 * J22 - J21 * J12) - J01 * (J10 * J22 - J20 * J12) + J02 * (J10 * J21 - J20 * J11);\n";
            inv = {{"I00", "(J11 * J22 - J12 * J21)"}, {"I01", "(J02 * J21 - J01 * J22)"}, {"I02", "(J01 * J12 - J02 * J11)"},
                   {"I10", "(J12 * J20 - J10 * J22)"}, {"I11", "(J00 * J22 - J02 * J20)"}, {"I12", "(J02 * J10 - J00 * J12)"},
                   {"I20", "(J10 * J21 - J11 * J20)"}, {"I21", "(J01 * J20 - J00 * J21)"}, {"I22", "(J00 * J11 - J01 * J10)"}};
        }
        if (staged)
            s << indent << "const double rd = 1.0 / det;\n" << indent << "const bool odd = !(fabs(det) >= 0x1p-1022 && fabs(det) < 0x1p1021);\n";
        for (const auto& i : inv)
            if (staged)
                s << indent << "const double " << i.first << " = quotient(" << i.second << ", det, rd, odd);\n";
            else
                s << indent << "const double " << i.first << " = " << i.second << " / det;\n";
    }
    s << indent << "const double wdet = p.weights[g] * fabs(det);\n";
}

// Program nodes the given terms depend on.
std::vector<char> node_closure(const GroupDev& G, const std::vector<int>& terms)
{
    const int n = (int)G.nodes.size();
    std::vector<char> needed(n, 0);
    for (int t : terms) needed[G.term_node[t]] = 1;
    for (int i = n - 1; i >= 0; i--) {
        if (!needed[i])
            continue;
        const slgpu_node& nd = G.nodes[i];
        if (nd.op == SLGPU_OP_ADD || nd.op == SLGPU_OP_MUL || nd.op == SLGPU_OP_POW)
            needed[nd.a] = needed[nd.b] = 1;
        if (nd.op == SLGPU_OP_INV || nd.op == SLGPU_OP_NEG)
            needed[nd.a] = 1;
    }
    return needed;
}

// `const double v<i> = ...;` for the needed nodes (q: the group's descriptor;
// e, o, g, J.., I.., det, X.. in scope).
void emit_nodes(std::ostringstream& s, const GroupDev& G, const std::vector<char>& needed, int ngp, const char* indent)
{
    for (int i = 0; i < (int)G.nodes.size(); i++) {
        if (!needed[i])
            continue;
        const slgpu_node& nd = G.nodes[i];
        if (nd.op == SLGPU_OP_FIELD) {
            // sum_f coefficient[f][e] * form function f at (orientation, gp)
            const int rows = G.tab_rows[nd.b];
            s << indent << "double v" << i << " = 0;\n";
            s << indent << "for (int f = 0; f < " << rows << "; f++) v" << i << " = fma(q.fielddata[(i64)" << G.field_off[nd.a]
              << " + (i64)f * p.nelem + e], q.tables[(i64)" << G.tab_off[nd.b] << " + ((i64)o * " << rows << " + f) * " << ngp
              << " + g], v" << i << ");\n";
            continue;
        }
        s << indent << "const double v" << i << " = ";
        switch (nd.op) {
        case SLGPU_OP_CONST: s << lit(G.hconsts[nd.a]); break;
        case SLGPU_OP_JAC: s << "J" << nd.a << nd.b; break;
        case SLGPU_OP_INVJAC: s << "I" << nd.a << nd.b; break;
        case SLGPU_OP_DETJAC: s << "det"; break;
        case SLGPU_OP_ELEM: s << "q.elemdata[(i64)" << nd.a << " * p.nelem + e]"; break;
        case SLGPU_OP_COORD: s << "X" << nd.a; break;
        case SLGPU_OP_ADD: s << "v" << nd.a << " + v" << nd.b; break;
        case SLGPU_OP_MUL: s << "v" << nd.a << " * v" << nd.b; break;
        case SLGPU_OP_INV: s << "1.0 / v" << nd.a; break;
        case SLGPU_OP_NEG: s << "-v" << nd.a; break;
        case SLGPU_OP_POW: s << "pow(v" << nd.a << ", v" << nd.b << ")"; break;
        default: throw std::runtime_error("unknown coefficient op");
        }
        s << ";\n";
    }
}

std::vector<int> all_terms(const GroupDev& G)
{
    std::vector<int> t(G.nterms);
    for (int k = 0; k < G.nterms; k++) t[k] = k;
    return t;
}

}  // namespace

std::string jit_coef_source(const std::vector<const GroupDev*>& batch)
{
    const GroupDev& g0 = *batch[0];
    const int dim = g0.problemdim, ncn = g0.ncn, ngp = g0.ngp;
    std::ostringstream s;
    s << kPrelude;
    // The batch's group descriptors are passed by value (kernel parameter
    // space), so that a launch needs no argument upload.
    s << "struct JitGroups { JitGroup g[" << batch.size() << "]; };\n";
    s << "extern \"C\" __global__ void __launch_bounds__(128) slgpu_coef(JitGeom p, const JitGroups grp)\n{\n";
    s << "  const i64 n = blockIdx.x * (i64)blockDim.x + threadIdx.x;\n";
    s << "  if (n >= p.nelem * " << ngp << ") return;\n";
    s << "  const int g = (int)(n / p.nelem);\n  const i64 e = n - (i64)g * p.nelem;\n";
    s << "  const int o = p.orient[e];\n";
    emit_geometry(s, dim, ncn, ngp, "  ");
    s << "  (void)o; (void)X0; (void)X1; (void)X2;\n";
    for (size_t k = 0; k < batch.size(); k++) {
        const GroupDev& G = *batch[k];
        // A group whose coefficients are not needed in this launch (the
        // second group of a transposed pair) gets C = null.
        s << "  if (grp.g[" << k << "].C != nullptr) {\n    const JitGroup q = grp.g[" << k << "];\n";
        emit_nodes(s, G, node_closure(G, all_terms(G)), ngp, "    ");
        s << "    int top = 0;\n";
        for (int t = 0; t < G.nterms; t++) {
            const int c = G.term_node[t];
            s << "    { const double c = v" << c << " * q.term_scale[" << t << "] * wdet; q.C[((i64)" << t << " * " << ngp
              << " + g) * p.nelem + e] = c; top = max(top, __double2hiint(c) & 0x7fffffff); }\n";
        }
        // High word of the element's largest coefficient for split precision.
        s << "    if (q.elemtop != nullptr && top > 0) atomicMax(q.elemtop + e, top);\n";
        s << "  }\n";
    }
    s << "}\n";
    return s.str();
}

// Shape of the slicing kernel for a batch: elements per block, groups per
// round, and the shared memory of the values staged in a round (17/16 of them:
// see jit_slice_source).
//   Up to 64 points: a thread has one point of one element, so that it keeps
//   its Jacobian over the rounds; 256 threads at most.
//   More: 4 elements (the 16-byte stores of 4 neighbouring slots are two whole
//   sectors) and several points per thread.
// A round holds as many groups as leave room for four blocks per
// multiprocessor in shared memory.  (Order-2 elasticity, 9 groups of 243 values
// on 27 points, all staged at once: two blocks fit, and the kernel took 0.68
// instead of 0.49 ms at 48^3.  Its 80 registers then allow three blocks, those
// of the smaller kernels, 47 to 56, four or more.)
static size_t slice_staged(const GroupDev& g) { return ((size_t)g.nterms * g.ngp + 15) / 16 * 17; }

SliceShape slice_shape(const std::vector<const GroupDev*>& batch)
{
    const GroupDev& g0 = *batch[0];
    SliceShape sh;
    sh.E = 4;
    while (sh.E < 32 && 2 * sh.E * g0.ngp <= 256) sh.E *= 2;
    sh.single = sh.E * g0.ngp <= 256;
    size_t most = 0;
    for (const GroupDev* g : batch) most = std::max(most, slice_staged(*g));
    while (sh.E > 4 && 8 * most * sh.E > 50 * 1024) sh.E /= 2;
    sh.round = (int)std::max<size_t>(1, 50 * 1024 / (8 * most * sh.E));
    sh.round = std::min<int>(sh.round, (int)batch.size());
    sh.smem = 8 * most * sh.E * (size_t)sh.round;
    sh.threads = std::min(256, std::max(64, (g0.ngp * sh.E + 31) / 32 * 32));
    return sh;
}

// Coefficients straight to the column slices of the split contraction, for
// groups with one geometry and element tiles.  A block takes E elements (a
// part of a 64-element tile) and the batch's groups in rounds: it evaluates
// every coefficient of the round's groups into shared memory, finding each
// element's largest (the column scale), and then cuts them into slices, 16
// values along K per thread, stored 16 bytes at a time.  The coefficients
// never go to memory: per coefficient S bytes are written, where a kernel that
// writes them and one that slices them wrote 8, read 8 and wrote S; and an
// element's nodes are gathered once, not once per point.  Orders 1-5, 48,000
// tetrahedra: 0.42 -> 0.15 ms a step; order-2 elasticity, 48^3 hexahedra:
// 0.65 -> 0.47 ms.  (Evaluating twice instead of staging
// took 0.54 ms there.)
//
// Value q of element el of a group is at (q + q / 16) E + el of the group's
// place in the round: the extra E doubles per 16 values put the chunks that
// neighbouring threads read on other banks.  A group's descriptor without
// slices has no part in the launch.
std::string jit_slice_source(const std::vector<const GroupDev*>& batch, int tier)
{
    const GroupDev& g0 = *batch[0];
    const int dim = g0.problemdim, ncn = g0.ncn, ngp = g0.ngp;
    const int S = tier == 0 ? 6 : 5, B = tier == 0 ? 8 : 7;
    const size_t ng = batch.size();
    const SliceShape sh = slice_shape(batch);
    const size_t place = sh.smem / 8 / (size_t)sh.round;  // doubles per group of a round
    std::ostringstream s;
    s << kPrelude << "namespace slgpu { " << kSplitDigitSource << " }\n";
    s << "struct JitSlices { JitSlice g[" << ng << "]; };\n";
    // quotient: a / b, r = 1 / b correctly rounded.  The residual of a r corrects
    // it to the rounded quotient (P. Markstein, IBM J. Res. Dev. 34, 1990), in two
    // fma where a division takes its own reciprocal: with divisions the slices of
    // 48,000 tetrahedra of orders 1-5 took 37 us more than with a r alone, which
    // misses the last place; with this they take 151 us.  `odd` (b zero, no normal
    // double, or within 8 of the overflow): a r.  (A division there instead, by a
    // branch, held 64 registers instead of 47: 166 us.)
    s << "__device__ __forceinline__ double quotient(double a, double b, double r, bool odd)\n{\n"
      << "  const double q = a * r, c = fma(fma(-q, b, a), r, q);\n  return odd ? q : c;\n}\n";
    // One chunk: 16 staged values from `at` on, E apart, to the slices at out.
    // Not inlined: one copy for all rounds (compile time).  pr is 1 but for
    // magnitudes below 2^-900 (split_scale); a second copy without the product
    // took 50 ms more to compile and ran no faster.
    s << "extern __shared__ __align__(16) double st[];\n";
    s << "__device__ __noinline__ void cut(int at, double f, double pr, uint4* out)\n{\n";
    s << "  unsigned int wd[" << S << "][4];\n  #pragma unroll\n  for (int k4 = 0; k4 < 4; k4++) {\n    unsigned long long u[4];\n    #pragma unroll\n"
      << "    for (int i = 0; i < 4; i++) u[i] = slgpu::split_digits<" << B << ", " << S << ">(st[at + (4 * k4 + i) * " << sh.E
      << "] * pr, f);\n    slgpu::split_words<" << B << ", " << S << ">(u, wd, k4);\n  }\n";
    s << "  #pragma unroll\n  for (int i = 0; i < " << S << "; i++) out[i * 64] = make_uint4(wd[i][0], wd[i][1], wd[i][2], wd[i][3]);\n}\n";
    // Loops over the block's work, which take a few turns each, stay loops:
    // unrolled, nine groups of elasticity took 1.0 to 1.1 s to compile instead of
    // 0.5 to 0.65, and the calls in them cost 22 registers (48^3 hexahedra 0.66
    // instead of 0.49 ms, FP32 tetrahedra 101 instead of 87 us).
    const char* const kLoop = "#pragma unroll 1\n";
    s << "extern \"C\" __global__ void __launch_bounds__(" << sh.threads << ") slgpu_slices(JitGeom p, const JitSlices grp, const int4* tiles)\n{\n";
    s << "  constexpr int E = " << sh.E << ", NG = " << ng << ";\n";
    s << "  __shared__ double xs[" << 3 * ncn << " * E], fac[NG * E], pre[NG * E];\n  __shared__ int top[NG * E];\n";
    s << "  const i64 tile = blockIdx.x / (64 / E);\n  const int4 tl = tiles[tile];\n";
    s << "  const int base = (int)(blockIdx.x % (64 / E)) * E;\n  if (base >= tl.y) return;\n";
    s << "  const int o = tl.z;\n  (void)o;\n";
    // Slots past the end of a short tile repeat its last element.
    s << kLoop << "  for (int n = threadIdx.x; n < " << ncn << " * E; n += blockDim.x) { const int el = n % E, k = n / E;\n"
      << "    const i64 e = tl.x + (base + el < tl.y ? base + el : tl.y - 1);\n    const i64 nd = 3 * (i64)p.conn[(i64)p.elems[e] * " << ncn << " + k];\n"
      << "    xs[3 * k * E + el] = p.xyz[nd]; xs[(3 * k + 1) * E + el] = p.xyz[nd + 1]; xs[(3 * k + 2) * E + el] = p.xyz[nd + 2]; }\n";
    s << kLoop << "  for (int n = threadIdx.x; n < NG * E; n += blockDim.x) top[n] = 0;\n  __syncthreads();\n";
    auto point = [&](const char* indent) {
        s << indent << "const i64 e = tl.x + (base + el < tl.y ? base + el : tl.y - 1);\n";
        emit_geometry(s, dim, ncn, ngp, indent, true);
        s << indent << "(void)X0; (void)X1; (void)X2; (void)e;\n";
    };
    if (sh.single) {
        s << "  const bool live = threadIdx.x < " << ngp << " * E;\n";
        s << "  const int el = threadIdx.x % E, g = live ? threadIdx.x / E : " << ngp - 1 << ";\n";
        point("  ");
    }
    for (size_t r0 = 0; r0 < ng; r0 += (size_t)sh.round) {
        const size_t r1 = std::min(ng, r0 + (size_t)sh.round);
        s << (sh.single ? "" : kLoop) << (sh.single ? "  if (live) {\n" : "  for (int n = threadIdx.x; n < ");
        if (!sh.single) {
            s << ngp << " * E; n += blockDim.x) {\n    const int el = n % E, g = n / E;\n";
            point("    ");
        }
        for (size_t k = r0; k < r1; k++) {
            const GroupDev& G = *batch[k];
            s << "    if (grp.g[" << k << "].slices != nullptr) {\n      const JitSlice q = grp.g[" << k << "];\n";
            s << "      const int q0 = g * " << G.nterms << ";\n      double* out = st + " << (k - r0) * place << " + el;\n      int m = 0;\n";
            emit_nodes(s, G, node_closure(G, all_terms(G)), ngp, "      ");
            for (int t = 0; t < G.nterms; t++)
                s << "      { const double c = v" << G.term_node[t] << " * __ldg(q.term_scale + " << t << ") * wdet; out[(q0 + " << t << " + ((q0 + " << t
                  << ") >> 4)) * E] = c; m = max(m, __double2hiint(c) & 0x7fffffff); }\n";
            s << "      atomicMax(&top[" << k << " * E + el], m);\n    }\n";
        }
        s << "  }\n";
        for (size_t k = r0; k < r1; k++) {
            const int Q = batch[k]->nterms * ngp, Q16 = (Q + 15) / 16 * 16;
            if (Q16 > Q)
                s << kLoop << "  for (int n = threadIdx.x; n < " << Q16 - Q << " * E; n += blockDim.x) st[" << (k - r0) * place << " + " << Q + Q / 16
                  << " * E + n] = 0;\n";
        }
        bool same = true;
        for (size_t k = r0; k < r1; k++) same = same && batch[k]->nterms == batch[r0]->nterms;
        // Scales.  The values of a column are looked at until the first that a
        // scale by powers of two would not hold exactly, as a rule its first.
        s << "  __syncthreads();\n" << kLoop << "  for (int n = " << r0 << " * E + threadIdx.x; n < " << r1 << " * E; n += blockDim.x)\n"
          << "    if (grp.g[n / E].slices != nullptr) {\n";
        if (B == 8) {
            s << "      const int Q = ";
            for (size_t k = r0; !same && k + 1 < r1; k++) s << "n < " << k + 1 << " * E ? " << batch[k]->nterms * ngp << " : ";
            s << batch[r1 - 1]->nterms * ngp << ";\n      const double* v = st + (n / E - " << r0 << ") * " << place << " + n % E;\n"
              << "      bool exact = top[n] > 0;\n"
              << kLoop << "      for (int q = 0; exact && q < Q; q++) exact = slgpu::split_exact(v[(q + (q >> 4)) * E], top[n]);\n";
        } else {
            s << "      const bool exact = false;\n";
        }
        s << "      double unit;\n      fac[n] = slgpu::split_scale<" << B << ", " << S
          << ">(top[n], exact, &unit, &pre[n]);\n      grp.g[n / E].colscale[tile * 64 + base + n % E] = unit;\n    }\n  __syncthreads();\n";
        // Chunks of 16 values of the round's groups, the groups' chunks side by
        // side where they have equally many.
        auto chunks = [&](size_t a, size_t b) {
            const int Q = batch[a]->nterms * ngp, nc = (Q + 15) / 16, nchunk = (Q + 31) / 32 * 2;
            s << kLoop << "  for (int n = threadIdx.x; n < " << (b - a) * (size_t)nc << " * E; n += blockDim.x) {\n";
            s << "    const int el = n % E, gc = n / E, c = gc % " << nc << ", k = " << a << " + gc / " << nc << ";\n";
            s << "    uint4* out = grp.g[k].slices;\n    if (out == nullptr) continue;\n    out += ((tile * " << nchunk << " + c) * " << S
              << ") * 64 + base + el;\n";
            s << "    const double f = fac[k * E + el], pr = pre[k * E + el];\n    const int at = (k - " << r0 << ") * " << place
              << " + 17 * c * E + el;\n    cut(at, f, pr, out);\n  }\n";
        };
        if (same)
            chunks(r0, r1);
        else
            for (size_t k = r0; k < r1; k++) chunks(k, k + 1);
        if (r1 < ng)
            s << "  __syncthreads();\n";
    }
    s << "}\n";
    return s.str();
}

// Compiled kernels of the process by source, so that another context does not
// compile them again: the last kCubins compiled, under a lock.
namespace {
std::mutex cubin_mu;
constexpr size_t kCubins = 64;
std::deque<std::pair<std::string, std::vector<char>>> cubins;
}  // namespace

std::vector<char> jit_compile(const std::string& src)
{
    {
        std::lock_guard<std::mutex> lk(cubin_mu);
        for (const auto& c : cubins)
            if (c.first == src)
                return c.second;
    }
    nvrtcProgram prog;
    if (nvrtcCreateProgram(&prog, src.c_str(), "slgpu_coef.cu", 0, nullptr, nullptr) != NVRTC_SUCCESS)
        throw std::runtime_error("nvrtcCreateProgram failed");
    // No implicit multiply-add contraction: a coefficient program rounds the
    // same however the compiler schedules it; the sums of products (Jacobian,
    // coordinates, field values) are written as explicit fma.
    const char* opts[] = {"--gpu-architecture=sm_100a", "--std=c++17", "-default-device", "--fmad=false"};
    nvrtcResult r = nvrtcCompileProgram(prog, 4, opts);
    if (r != NVRTC_SUCCESS) {
        size_t n = 0;
        nvrtcGetProgramLogSize(prog, &n);
        std::string log(n, '\0');
        nvrtcGetProgramLog(prog, &log[0]);
        nvrtcDestroyProgram(&prog);
        throw std::runtime_error("NVRTC compile of a coefficient kernel failed: " + log.substr(0, 2000));
    }
    size_t n = 0;
    nvrtcGetCUBINSize(prog, &n);
    std::vector<char> cubin(n);
    nvrtcGetCUBIN(prog, cubin.data());
    nvrtcDestroyProgram(&prog);
    {
        std::lock_guard<std::mutex> lk(cubin_mu);
        cubins.emplace_back(src, cubin);
        if (cubins.size() > kCubins)
            cubins.pop_front();
    }
    return cubin;
}

cudaKernel_t jit_kernel(Ctx* ctx, const std::string& src, const char* name, int smem)
{
    auto it = ctx->jit_kernels.find(src);
    if (it != ctx->jit_kernels.end())
        return it->second;
    std::vector<char> cubin = jit_compile(src);
    cudaLibrary_t lib;
    cudaError_t e = cudaLibraryLoadData(&lib, cubin.data(), nullptr, nullptr, 0, nullptr, nullptr, 0);
    if (e != cudaSuccess)
        throw std::runtime_error(std::string("cudaLibraryLoadData: ") + cudaGetErrorString(e));
    cudaKernel_t k;
    e = cudaLibraryGetKernel(&k, lib, name);
    if (e != cudaSuccess)
        throw std::runtime_error(std::string("cudaLibraryGetKernel: ") + cudaGetErrorString(e));
    if (smem > 0) {
        e = cudaKernelSetAttributeForDevice(k, cudaFuncAttributeMaxDynamicSharedMemorySize, smem, ctx->device);
        if (e != cudaSuccess)
            throw std::runtime_error(std::string("shared memory of a runtime-compiled kernel: ") + cudaGetErrorString(e));
    }
    ctx->jit_libs.push_back(lib);
    ctx->jit_kernels[src] = k;
    return k;
}

}  // namespace slgpu
