// Source generator of the compiled executor: turns a unit's ComputeKernel
// templates into one CUDA C++ module for NVRTC (see codegen.hpp).
//
// Every template is emitted from the same linear code the interpreter's
// programs are bundled from (program.cpp: linearCode), one statement per
// operation, each with the same CUDA rounding intrinsic the interpreter
// executes (__dadd_rn, __fma_rn, the prelude's fast division ...).  The
// compiler is therefore free to schedule and allocate registers, but not to
// change any value: results are bit-identical to the interpreter's in both
// math modes, and in exact mode to the reference's generated code built
// without FP contraction.  Plan constants (instance counts, table offsets,
// output slots, value sets) are literals of the source, so index arithmetic
// folds at compile time.
//
// A thread takes 1, 2 or 4 work items, either tpb items apart (strided) or as
// consecutive instances of one value set whose index and constant entries it
// reads with vector loads from padded copies of the tables (grouped).  With
// one value set, output rows that no kernel reads may store their results
// straight at their final positions in the unit's result buffer (direct
// result rows, planned by the engine at init).
#include "codegen.hpp"

#include <algorithm>
#include <cmath>
#include <cstdio>
#include <map>
#include <set>
#include <cstring>
#include <sstream>
#include <stdexcept>

#include "program.hpp"

namespace symgb {
namespace engine {

namespace {

std::string u64(std::uint64_t v) { return std::to_string(v) + "ull"; }

std::string literal(std::uint64_t bits) {
    char buf[64];
    std::snprintf(buf, sizeof buf, "__longlong_as_double((long long)0x%016llxull)", (unsigned long long)bits);
    return buf;
}

const char* libName(int op) {
    switch (op) {
        case OP_SIN: return "sin";
        case OP_COS: return "cos";
        case OP_TAN: return "tan";
        case OP_ASIN: return "asin";
        case OP_ACOS: return "acos";
        case OP_ATAN: return "atan";
        case OP_EXP: return "exp";
        case OP_LOG: return "log";
        default: return nullptr;
    }
}

// Some of a template's output rows with the operations and loads they need
// (splitTemplate); a thread evaluates one piece of one work item.
struct Piece {
    std::vector<char> ops, loads;  // by linear operation, by load
    double cost = 0.0;             // FP64 instructions
};

// The device function of a piece, as the dispatch calls it.
struct Call {
    std::string body;  // symgbBody<k>, symgbMixed<k> or symgbPart<k>_<piece>
    std::size_t ops = 0;  // operations of the whole template
    bool mixed = false;
};

// Emits the device function evaluating kernel k.
//   Strided items (grouped == nullptr): symgbBody<k><L2, ORDER>(..., i, s)
//     evaluates one work item (instance i, value set s) and loads its own index
//     and constant entries; ORDER is what it does between these loads, which
//     no kernel writes, and its first read of x (emitPrologue).
//   Grouped items: symgbGroup<k><L2, IT, FULL>(..., g, s) evaluates the IT
//     consecutive instances g*IT .. g*IT+IT-1 of value set s; each index and
//     constant row is read with one vector load from the padded copies of the
//     tables (`grouped` gives their row bases), the instances' gathers,
//     arithmetic and stores follow, unrolled.  FULL = false guards the
//     instances past the kernel's end (the last group).
// Output rows with a start in `direct` (>= 0) store their results into
// res[dp[start + i]] (their final positions) instead of x.  L2 = 1 reads x
// through L2 only (values written earlier in the same launch, persistent
// schedule).  Returns the number of operations of the template.
//   With intMuls > 0: symgbMixed<k>, the strided body with that many of its
//     products, evenly spread, and the first products of its divisions and
//     square roots on the integer pipes (prelude: symgbMulInt), the same bits
//     as symgbBody<k>'s.  It returns whether an operand was outside what those
//     cover; the caller then evaluates symgbBody<k>, which stores the same
//     results again.  A product's range is checked at its factors that come
//     from loads or FP64 instructions, once each; products of up to four of
//     them need no check.
//   With `piece`: symgbPart<k>_<pieceIndex>, the strided body of those rows.
// `called`: emitted as a function of its own instead of into its callers.
std::size_t emitBody(std::ostringstream& os, int k, const symgb_kernel_desc& d, int math, unsigned S,
                     const GroupedTables* grouped, const std::vector<std::int64_t>* direct, bool called,
                     int intMuls = 0, const Piece* piece = nullptr, int pieceIndex = 0) {
    std::vector<std::uint64_t> loads;
    std::vector<LinOp> ops = linearCode(d, math, &loads);
    if (piece) {
        std::vector<std::uint64_t> l;
        std::vector<LinOp> o;
        for (std::size_t j = 0; j < loads.size(); ++j)
            if (piece->loads[j]) l.push_back(loads[j]);
        for (std::size_t j = 0; j < ops.size(); ++j)
            if (piece->ops[j]) o.push_back(ops[j]);
        loads.swap(l);
        ops.swap(o);
    }
    const std::uint64_t n = d.num_instances;
    const bool g = grouped != nullptr;
    const char* in = g ? "        " : "    ";
    const bool mixed = intMuls > 0;
    if (!mixed && !piece) os << "// kernel " << k << ": " << n << " instances, level " << d.level << ", " << loads.size() << " loads, "
       << ops.size() << " operations\n";
    if (called && !mixed && !piece) os << "#ifndef SYMGB_CALLED\n#define SYMGB_CALLED\n#endif\n";
    if (g)
        os << "template <int L2, int IT, bool FULL>\n__device__ __forceinline__ void symgbGroup" << k
           << "(const double* SYMGB_XR x, double* SYMGB_XR xw, const unsigned* __restrict__ p, "
              "const double* __restrict__ c, double* __restrict__ res, const unsigned* __restrict__ dp, "
              "unsigned long long g, unsigned s) {\n";
    else
        os << "template <int L2, int ORDER = 0>\n__device__ " << (called ? "SYMGB_CALLED " : "__forceinline__ ")
           << (mixed ? "bool symgbMixed" : piece ? "void symgbPart" : "void symgbBody") << k
           << (piece ? "_" + std::to_string(pieceIndex) : std::string())
           << "(const double* SYMGB_XR x, double* SYMGB_XR xw, const unsigned* __restrict__ p, "
              "const double* __restrict__ c, double* __restrict__ res, const unsigned* __restrict__ dp, "
              "unsigned long long i, unsigned s) {\n";
    std::vector<std::string> cur(256);
    int next = 0;
    // Integer products (mixed bodies): literals, factors of a value, values
    // whose range has been checked, values whose significand is at hand.
    std::map<std::string, std::uint64_t> literals;
    std::map<std::string, int> factors;
    std::set<std::string> checked, split;
    int mulsSeen = 0, mulsTaken = 0, mulCount = 0;
    for (const LinOp& L : ops) mulCount += L.op == OP_MUL;
    if (mixed) os << "    bool outside = false;\n";
    auto inWindow = [](std::uint64_t b) {
        const unsigned e = (unsigned)(b >> 52) & 0x7ffu;
        return e >= 768 && e < 1279;
    };
    auto check = [&](const std::string& v) {  // v's range, at run time: one factor from here on
        if (checked.insert(v).second && !literals.count(v)) os << in << "outside |= symgbOutside(" << v << ");\n";
        factors[v] = 1;
    };
    auto sig = [&](const std::string& v) {
        if (split.insert(v).second) os << in << "const unsigned s" << v << " = symgbSig(" << v << ");\n";
        return "s" + v;
    };
    // a * b on the integer pipes, or nothing where they do not cover it.
    auto intProduct = [&](std::string a, std::string b) -> std::string {
        if (literals.count(a)) std::swap(a, b);
        if (literals.count(a)) return std::string();
        const auto lit = literals.find(b);
        if (lit != literals.end()) {
            if (!inWindow(lit->second)) return std::string();
            const int K = (int)((lit->second >> 52) & 0x7ff) - 1023;
            if (!(lit->second & 0xfffffffffffffull) && K >= -64 && K <= 64) {
                if (!factors.count(a) || factors[a] > 3) check(a);
                factors["="] = factors[a] + 1;
                return "symgbMulPow2<" + std::to_string(K) + ", " + std::to_string((int)(lit->second >> 63)) + ">(" + a + ")";
            }
            factors[b] = 1;
        }
        if ((long long)mulsSeen * intMuls / std::max(1, mulCount) < mulsTaken) return std::string();
        if (!factors.count(a)) check(a);
        if (!factors.count(b)) check(b);
        if (factors[a] + factors[b] > 4) check(factors[a] > factors[b] ? a : b);
        if (factors[a] + factors[b] > 4) check(factors[a] > factors[b] ? a : b);
        ++mulsTaken;
        factors["="] = factors[a] + factors[b];
        const std::string sa = sig(a), sb = sig(b);
        return "symgbMulInt(" + a + ", " + b + ", " + sa + ", " + sb + ")";
    };
    auto fresh = [&](int reg) -> std::string {
        std::string v = "v" + std::to_string(next++);
        if (reg < 0 || reg >= (int)cur.size()) throw std::runtime_error("codegen: register out of range");
        cur[reg] = v;
        return v;
    };
    auto use = [&](int reg) -> const std::string& {
        if (reg < 0 || reg >= (int)cur.size() || cur[reg].empty())
            throw std::runtime_error("codegen: register read before written");
        return cur[reg];
    };
    const std::string xs = S == 1 ? std::string() : " * " + std::to_string(S) + "ull + s";
    // Index rows read by the gathers, each loaded once (correlated index
    // variables share a row and differ by their offsets); constant rows
    // likewise in the grouped layout.
    std::vector<int> rowVar(d.num_index_rows, -1);
    int rows = 0;
    for (std::uint64_t w : loads) {
        if ((int)(w & 0xff) != OP_LDX) continue;
        const std::uint64_t row = (w >> 16) & 0xffff;
        if (row >= d.num_index_rows) throw std::runtime_error("codegen: index row out of range");
        if (rowVar[row] >= 0) continue;
        rowVar[row] = rows++;
        if (g)
            os << "    unsigned q" << rowVar[row] << "[IT];\n    symgbLoadIdx<IT>(p + "
               << u64(grouped->indexBase[k] + row * grouped->stride[k]) << " + g * IT, q" << rowVar[row] << ");\n";
        else
            os << "    const unsigned q" << rowVar[row] << " = SYMGB_LD(p + " << u64(d.index_offset + row * n)
               << " + i);\n";
    }
    std::vector<int> constVar;
    if (!g) {
        constVar.assign(d.num_constant_rows, -1);
        int consts = 0;
        for (std::uint64_t w : loads) {
            if ((int)(w & 0xff) != OP_LDC) continue;
            const std::uint32_t row = (std::uint32_t)(w >> 32);
            if (row >= d.num_constant_rows) throw std::runtime_error("codegen: constant row out of range");
            if (constVar[row] >= 0) continue;
            constVar[row] = consts++;
            os << "    const double k" << constVar[row] << " = SYMGB_LD(c + "
               << u64(d.constants_offset + (std::uint64_t)row * n) << " + i);\n";
        }
        os << "#ifdef SYMGB_ORDERED\n    x = symgbOrder<ORDER>(x);\n#endif\n";
    } else {
        constVar.assign(d.num_constant_rows, -1);
        int consts = 0;
        for (std::uint64_t w : loads) {
            if ((int)(w & 0xff) != OP_LDC) continue;
            const std::uint32_t row = (std::uint32_t)(w >> 32);
            if (row >= d.num_constant_rows) throw std::runtime_error("codegen: constant row out of range");
            if (constVar[row] >= 0) continue;
            constVar[row] = consts++;
            os << "    double k" << constVar[row] << "[IT];\n    symgbLoadConst<IT>(c + "
               << u64(grouped->constBase[k] + row * grouped->stride[k]) << " + g * IT, k" << constVar[row] << ");\n";
        }
        os << "    #pragma unroll\n    for (int j = 0; j < IT; ++j) {\n"
           << "        const unsigned long long i = g * IT + j;\n"
           << "        if (!FULL && i >= " << u64(n) << ") break;\n";
    }
    const std::string qj = g ? "[j]" : "";
    for (std::uint64_t w : loads) {
        const int op = (int)(w & 0xff), dst = (int)((w >> 8) & 0xff);
        const std::uint32_t imm = (std::uint32_t)(w >> 32);
        if (op == OP_LDX) {
            const std::uint64_t row = (w >> 16) & 0xffff;
            const std::string v = fresh(dst);
            os << in << "const double " << v << " = symgbLoadX<L2>(x + (unsigned long long)(q" << rowVar[row] << qj
               << " + " << imm << "u)" << xs << ");\n";
        } else if (op == OP_LDC) {
            const std::string v = fresh(dst);
            os << in << "const double " << v << " = k" << constVar[imm] << (g ? "[j];\n" : ";\n");
        } else {
            throw std::runtime_error("codegen: unknown load word");
        }
    }
    for (const LinOp& L : ops) {
        std::string rhs;
        switch (L.op) {
            case OP_ST:
                if (direct && L.row < direct->size() && (*direct)[L.row] >= 0)
                    os << in << "res[SYMGB_LD(dp + " << u64((std::uint64_t)(*direct)[L.row]) << " + i)] = "
                       << use(L.src[0]) << ";\n";
                else
                    os << in << "xw[(" << u64(d.output_offset + (std::uint64_t)L.row * n) << " + i)" << xs
                       << "] = " << use(L.src[0]) << ";\n";
                continue;
            case OP_MOV: {
                const std::string src = use(L.src[0]);
                cur[L.d] = src;
                continue;
            }
            case OP_LDK: rhs = literal(L.lit); break;
            case OP_ADD: rhs = "__dadd_rn(" + use(L.src[0]) + ", " + use(L.src[1]) + ")"; break;
            case OP_SUB: rhs = "__dsub_rn(" + use(L.src[0]) + ", " + use(L.src[1]) + ")"; break;
            case OP_MUL:
                if (mixed) {
                    rhs = intProduct(use(L.src[0]), use(L.src[1]));
                    ++mulsSeen;
                    if (!rhs.empty()) break;
                }
                rhs = "__dmul_rn(" + use(L.src[0]) + ", " + use(L.src[1]) + ")";
                break;
            case OP_DIV: rhs = "__ddiv_rn(" + use(L.src[0]) + ", " + use(L.src[1]) + ")"; break;
            case OP_NEG: rhs = "symgbNegate(" + use(L.src[0]) + ")"; break;
            case OP_SQRT: rhs = "__dsqrt_rn(" + use(L.src[0]) + ")"; break;
            case OP_REC: rhs = "__ddiv_rn(1.0, " + use(L.src[0]) + ")"; break;
            case OP_FDIV:
                if (mixed && !literals.count(use(L.src[0]))) {
                    const std::string a = use(L.src[0]), b = use(L.src[1]);
                    if (!factors.count(a) || factors[a] > 1) check(a);  // the division's own range is narrower
                    rhs = "symgbFastDivInt(" + a + ", " + b + ", " + sig(a) + ", outside)";
                    break;
                }
                rhs = "symgbFastDiv(" + use(L.src[0]) + ", " + use(L.src[1]) + ")"; break;
            case OP_FSQRT:
                if (mixed && !literals.count(use(L.src[0]))) {
                    const std::string a = use(L.src[0]);
                    if (!factors.count(a) || factors[a] > 3) check(a);
                    rhs = "symgbFastSqrtInt(" + a + ", " + sig(a) + ", outside)";
                    break;
                }
                rhs = "symgbFastSqrt(" + use(L.src[0]) + ")"; break;
            case OP_FREC: rhs = "symgbFastRec(" + use(L.src[0]) + ")"; break;
            case OP_FMA: rhs = "__fma_rn(" + use(L.src[0]) + ", " + use(L.src[1]) + ", " + use(L.src[2]) + ")"; break;
            case OP_FMS:
                rhs = "__fma_rn(" + use(L.src[0]) + ", " + use(L.src[1]) + ", symgbNegate(" + use(L.src[2]) + "))";
                break;
            case OP_FNMA:
                rhs = "__fma_rn(symgbNegate(" + use(L.src[0]) + "), " + use(L.src[1]) + ", " + use(L.src[2]) + ")";
                break;
            case OP_FNMS:
                rhs = "__fma_rn(symgbNegate(" + use(L.src[0]) + "), " + use(L.src[1]) + ", symgbNegate(" +
                      use(L.src[2]) + "))";
                break;
            case OP_POW: rhs = "pow(" + use(L.src[0]) + ", " + use(L.src[1]) + ")"; break;
            default: {
                const char* f = libName(L.op);
                if (!f) throw std::runtime_error("codegen: operation " + std::to_string(L.op) + " not supported");
                rhs = std::string(f) + "(" + use(L.src[0]) + ")";
            }
        }
        const std::string v = fresh(L.d);
        os << in << "const double " << v << " = " << rhs << ";\n";
        if (mixed && L.op == OP_LDK) literals[v] = L.lit;
        if (mixed && factors.count("=")) {
            factors[v] = factors["="];
            factors.erase("=");
        }
    }
    if (mixed) os << "    return outside;\n";
    if (g) os << "    }\n";
    os << "}\n\n";
    return ops.size();
}

std::uint64_t blocksFor(std::uint64_t total, int tpb, int items) {
    const std::uint64_t per = (std::uint64_t)tpb * items;
    return (total + per - 1) / per;
}

// FP64 instructions of an operation.
int fp64Cost(int op) {
    switch (op) {
        case OP_LDK: case OP_ST: case OP_MOV: case OP_NEG: return 0;
        case OP_FDIV: return 5;
        case OP_FSQRT: return 6;
        case OP_FREC: return 4;
        case OP_DIV: case OP_SQRT: case OP_REC: return 9;
        default: return 1;
    }
}

// Products of every kernel that go to the integer pipes (symgbMixed), 0 for a
// kernel that stays on the FP64 pipe alone.  Results are the same bits.
//   * In levels of 16384 work items up.  Below, a launch leaves most schedulers
//     without a second warp to share the pipes with and pays for fetching the
//     longer code: Neo-Hookean 8^3, nine kernels of 10 k items, 41.1 us without
//     and 43.4 with, of 41 k 69.3 and 53.9; cloth 64 x 64, 7938 items, 41.1 and
//     40.9; eight small cloth patterns in one graph 206 and 220.
//   * Templates of 8 FP64 instructions up; lighter ones wait for memory.
//   * The share that keeps both pipes equally busy: an FP64 instruction of
//     three register operands holds a scheduler's pipe for 76 cycles (64 with two
//     of them constants), an integer product its issue slots and pipes for
//     about 44.
//   * As many as fit the instruction cache with the rest of the body (32
//     instructions each, 108 KB in all by this count; the cloth kernel it allows
//     is 125 KB): cloth 100 x 100 x 64 (plain, 64 x 4),
//     279 products, 1914 us with none, 1475 with 142 - 158, 1641 with 200, 1677 with
//     all but powers of two.
//   * At most 512 in a module, shared out by work: co-resident kernels share
//     the instruction cache (Neo-Hookean 8^3 x 16, 168 - 261 products in each of
//     nine templates: 69.3 us with none, 53.4 with 80 each, 63.1 with all), and
//     NVRTC takes about 7 ms per product.
std::vector<int> integerProducts(const std::vector<symgb_kernel_desc>& descs, int math, unsigned S) {
    constexpr std::uint64_t kLeastItems = 1024, kLeastLevelItems = 16384;
    constexpr int kLeastOps = 8, kCacheInstructions = 6912, kProductInstructions = 32, kModule = 512;
    constexpr int kFp64Cycles = 76, kProductCycles = 44;
    struct Count {
        int muls = 0, fp64 = 0, inner = 0, loads = 0;  // inner: first products of divisions and square roots
    };
    std::vector<Count> count(descs.size());
    std::map<int, std::uint64_t> levelItems;
    for (std::size_t k = 0; k < descs.size(); ++k) {
        std::vector<std::uint64_t> loads;
        Count& c = count[k];
        for (const LinOp& L : linearCode(descs[k], math, &loads)) {
            c.muls += L.op == OP_MUL;
            c.inner += L.op == OP_FDIV || L.op == OP_FSQRT;
            c.fp64 += fp64Cost(L.op);
        }
        c.loads = (int)loads.size();
        if (c.fp64 >= kLeastOps) levelItems[descs[k].level] += descs[k].num_instances * S;
    }
    std::vector<int> take(descs.size(), 0);
    std::vector<double> work(descs.size(), 0.0);
    double all = 0.0;
    int total = 0;
    for (std::size_t k = 0; k < descs.size(); ++k) {
        const Count& c = count[k];
        const std::uint64_t items = descs[k].num_instances * S;
        if (c.fp64 < kLeastOps || c.muls + c.inner == 0) continue;
        if (items < kLeastItems || levelItems[descs[k].level] < kLeastLevelItems) continue;
        const int share = (int)((long long)c.fp64 * kFp64Cycles / (kFp64Cycles + kProductCycles)) - c.inner;
        const int room = (kCacheInstructions - 3 * (c.fp64 - c.muls) - 6 * c.loads) / kProductInstructions - c.inner;
        take[k] = std::max(0, std::min({c.muls, share, room}));
        if (!take[k] && c.inner) take[k] = 1;  // a mixed body for its divisions and square roots
        total += take[k];
        work[k] = (double)items * c.fp64;
        all += work[k];
    }
    if (total > kModule)
        for (std::size_t k = 0; k < descs.size(); ++k)
            if (take[k]) take[k] = std::min(take[k], std::max(1, (int)(kModule * work[k] / all)));
    return take;
}

// A template's output rows with everything each of them needs.
struct Rows {
    int ops = 0, loads = 0;
    struct Row {
        std::vector<int> ops, loads;  // operations (its store among them) and loads it needs
        int cost = 0;
    };
    std::vector<Row> rows;   // in template order; empty where a row is stored twice
    std::vector<int> cost;   // by operation
};

Rows rowsOf(const symgb_kernel_desc& d, int math) {
    std::vector<std::uint64_t> loads;
    const std::vector<LinOp> ops = linearCode(d, math, &loads);
    Rows r;
    r.ops = (int)ops.size();
    r.loads = (int)loads.size();
    std::vector<int> def(256, -1);  // register -> load (0 .. loads - 1) or operation (loads + j) that wrote it
    for (int i = 0; i < r.loads; ++i) def[(loads[i] >> 8) & 0xff] = i;
    std::vector<std::vector<int>> needs(r.ops);
    std::vector<char> stored(d.num_output_rows, 0);
    for (int j = 0; j < r.ops; ++j) {
        for (int q = 0; q < ops[j].nsrc; ++q) needs[j].push_back(def[ops[j].src[q]]);
        if (ops[j].d >= 0) def[ops[j].d] = r.loads + j;
        r.cost.push_back(fp64Cost(ops[j].op));
    }
    std::vector<int> seen(r.ops + r.loads, -1);
    for (int j = 0; j < r.ops; ++j) {
        if (ops[j].op != OP_ST) continue;
        if (ops[j].row >= stored.size() || stored[ops[j].row]) return Rows();
        stored[ops[j].row] = 1;
        Rows::Row row;
        std::vector<int> todo{r.loads + j};
        while (!todo.empty()) {
            const int v = todo.back();
            todo.pop_back();
            if (v < 0 || seen[v] == j) continue;
            seen[v] = j;
            if (v < r.loads) {
                row.loads.push_back(v);
                continue;
            }
            row.ops.push_back(v - r.loads);
            row.cost += r.cost[v - r.loads];
            todo.insert(todo.end(), needs[v - r.loads].begin(), needs[v - r.loads].end());
        }
        r.rows.push_back(std::move(row));
    }
    return r;
}

// Cuts a template into `count` pieces: the cheapest piece so far takes the row
// that adds least to it (of equals the dearest), until all are taken.
std::vector<Piece> splitTemplate(const Rows& r, int count) {
    std::vector<Piece> ps(count, Piece{std::vector<char>(r.ops, 0), std::vector<char>(r.loads, 0), 0.0});
    std::vector<char> taken(r.rows.size(), 0);
    for (std::size_t left = r.rows.size(); left > 0; --left) {
        Piece* p = &ps[0];
        for (Piece& q : ps)
            if (q.cost < p->cost) p = &q;
        int row = -1, least = 0;
        for (std::size_t i = 0; i < r.rows.size(); ++i) {
            if (taken[i]) continue;
            int more = 0;
            for (int j : r.rows[i].ops)
                if (!p->ops[j]) more += r.cost[j];
            if (row < 0 || more < least || (more == least && r.rows[i].cost > r.rows[row].cost)) {
                row = (int)i;
                least = more;
            }
        }
        taken[row] = 1;
        p->cost += least;
        for (int j : r.rows[row].ops) p->ops[j] = 1;
        for (int j : r.rows[row].loads) p->loads[j] = 1;
    }
    return ps;
}

// Pieces of every kernel's template (empty: whole).  Heavy templates of
// launches that leave schedulers idle are cut, the pieces going to different
// blocks: an FP64 instruction takes a warp's scheduler 64 cycles whatever else
// the warp has ready, so a launch of few warps lasts as long as its longest
// template, and a shorter one helps although the pieces evaluate shared
// operations again.  Per level the number of pieces with the shortest estimate,
// where it is at least a tenth below that of fewer: the longest piece times the
// blocks that come to lie on one SM.  Blocks are dealt out evenly to GPCs of
// uneven size, so that from 117 blocks of four warps on (cloth 60 and 62, two
// pieces exact: 117 blocks and 118, 30.7 and 53.4 us), in a persistent grid of
// two blocks per SM from 59 on, some SM has two.  GB300, levels: cloth 64 x 64
// 33.8 -> 27.9 us (three pieces), cloth 20 x 20 31.3 -> 15.6 (six), Neo-Hookean
// 8^3 x 4 33.1 -> 27.6 (two), 4^3 exact 37.1 -> 12.8 (eight).
std::vector<std::vector<Piece>> templatePieces(const std::vector<symgb_kernel_desc>& descs, const JitConfig& cfg,
                                               const std::vector<int>& intMuls) {
    constexpr int kHeavy = 64;  // FP64 instructions
    constexpr double kRounds = 4.0, kAlone = 1.15;  // a warp alone on its scheduler also waits for its loads
    const double oneRound = cfg.kind == JIT_PERSISTENT ? 58.0 : 116.0;  // blocks of four warps
    std::vector<std::vector<Piece>> out(descs.size());
    std::map<int, std::vector<int>> heavy;  // by level
    std::vector<int> costs(descs.size(), 0);
    for (std::size_t k = 0; k < descs.size(); ++k) {
        if (!descs[k].num_instances || intMuls[k]) continue;
        if (!cfg.inPlace.empty() && cfg.inPlace[k]) continue;  // a piece would read what another has stored
        for (const LinOp& L : linearCode(descs[k], cfg.math, nullptr)) costs[k] += fp64Cost(L.op);
        if (costs[k] >= kHeavy) heavy[descs[k].level].push_back((int)k);
    }
    for (const auto& level : heavy) {
        // Blocks of four warps of kernel k's work items, per piece.
        auto blocks = [&](int k) {
            const int tpb = cfg.kind == JIT_PLAIN ? cfg.kernelTpb.at(k)
                                                  : cfg.levelTpb.at(cfg.kind == JIT_LEVELS ? level.first : 0);
            const int items = cfg.kind == JIT_PLAIN ? cfg.kernelItems.at(k)
                                                    : cfg.levelItems.at(cfg.kind == JIT_LEVELS ? level.first : 0);
            return (double)blocksFor(descs[k].num_instances * cfg.numSets, tpb, items) * tpb / 128.0;
        };
        auto estimate = [&](const std::vector<std::vector<Piece>>& ps) {
            double longest = 0.0, all = 0.0, count = 0.0;
            for (std::size_t i = 0; i < ps.size(); ++i) {
                const int k = level.second[i];
                double most = ps[i].empty() ? (double)costs[k] : 0.0, sum = most;
                for (const Piece& q : ps[i]) {
                    most = std::max(most, q.cost);
                    sum += q.cost;
                }
                longest = std::max(longest, most);
                all += sum * blocks(k);
                count += std::max<std::size_t>(1, ps[i].size()) * blocks(k);
            }
            const double rounds = std::ceil(count / oneRound);
            return rounds <= 1.0 ? kAlone * longest : longest + std::min(rounds - 1.0, count / oneRound) * all / count;
        };
        std::vector<std::vector<Piece>> best(level.second.size());
        double bound = estimate(best);
        double count = 0.0;
        for (int k : level.second) count += blocks(k);
        if (count > kRounds * oneRound) continue;  // the chip is full
        std::vector<Rows> rows;
        for (int k : level.second) rows.push_back(rowsOf(descs[k], cfg.math));
        for (int pieces : {2, 3, 4, 6, 8}) {
            std::vector<std::vector<Piece>> ps(rows.size());
            for (std::size_t i = 0; i < rows.size(); ++i)
                if (rows[i].rows.size() >= (std::size_t)pieces) ps[i] = splitTemplate(rows[i], pieces);
            const double t = estimate(ps);
            if (t > 0.9 * bound) continue;
            bound = t;
            best.swap(ps);
        }
        for (std::size_t i = 0; i < best.size(); ++i) out[level.second[i]].swap(best[i]);
    }
    return out;
}

// Templates of at most this many operations per thread (operations x items)
// get a second, unguarded copy of the items loop for threads whose items are
// all in range: without a bounds check per item the compiler can issue every
// item's index and gather loads before the first item's arithmetic, which is
// what a light, memory-bound template needs.  Heavier templates keep one
// guarded loop (their loads are hidden by arithmetic, and the copy would
// double their compile time).
constexpr std::size_t kSplitOps = 1024;

// Work items of kernel k for block `b0` (relative to the kernel's first
// block): `items` per thread, consecutive threads on consecutive items in
// each of the thread's rounds (coalesced), rounds unrolled so the items'
// loads are in flight together.  `split`: threads whose items are all in
// range take an unguarded copy of the loop (kSplitOps).
void emitItems(std::ostringstream& os, int k, const Call& call, std::uint64_t total, unsigned S, int tpb, int items,
               int l2, const std::string& b0, const char* indent, bool split, int order) {
    const bool mixed = call.mixed;
    const std::string body = (mixed ? "if (" : "") + call.body;
    const std::string tail = mixed ? ")) symgbRedo" + std::to_string(k) + "<" + std::to_string(l2) + ">(x, xw, p, c, res, dp, w / " +
                                         std::to_string(S) + "ull, (unsigned)(w % " + std::to_string(S) + "ull))"
                                   : ")";
    const std::string targs = "<" + std::to_string(l2) + (order ? ", " + std::to_string(order) : std::string()) + ">";
    os << indent << "const unsigned long long w0 = (" << b0 << ") * " << (std::uint64_t)tpb * items
       << "ull + threadIdx.x;\n";
    if (items > 1 && split) {
        os << indent << "if (w0 + " << u64((std::uint64_t)(items - 1) * tpb) << " < " << u64(total) << ") {\n"
           << indent << "    #pragma unroll\n" << indent << "    for (int j = 0; j < " << items << "; ++j) {\n"
           << indent << "        const unsigned long long w = w0 + (unsigned long long)j * " << tpb << "ull;\n"
           << indent << "        " << body << targs << "(x, xw, p, c, res, dp, w / " << S
           << "ull, (unsigned)(w % " << S << "ull)" << tail << ";\n"
           << indent << "    }\n" << indent << "} else {\n";
    }
    // A heavy mixed body is not unrolled: one copy of it nearly fills the
    // instruction cache.
    if (items > 1)
        os << indent << (mixed && !split ? "#pragma unroll 1\n" : "#pragma unroll\n") << indent << "for (int j = 0; j < " << items << "; ++j) {\n";
    else os << indent << "{\n" << indent << "    const int j = 0;\n";
    os << indent << "    const unsigned long long w = w0 + (unsigned long long)j * " << tpb << "ull;\n"
       << indent << "    if (w < " << u64(total) << ") {\n" << indent << "        " << body << targs << "(x, xw, p, c, res, dp, w / "
       << S << "ull, (unsigned)(w % " << S << "ull)" << tail << ";\n" << indent << "    }\n"
       << indent << "}\n";
    if (items > 1 && split) os << indent << "}\n";
}

// Blocks of kernel k: strided, n*S work items at tpb*items per block;
// grouped, ceil(n / items) groups per value set, one thread each.
std::uint64_t kernelBlocks(const symgb_kernel_desc& d, unsigned S, int tpb, int items, bool grouped) {
    if (!grouped) return blocksFor(d.num_instances * S, tpb, items);
    const std::uint64_t groups = (d.num_instances + items - 1) / items;
    return (groups * S + tpb - 1) / tpb;
}

// Grouped work of kernel k for block `b0` (relative to the kernel's first
// block): thread t takes group t / S of value set t % S (consecutive threads
// on consecutive sets, then groups).  Full groups run without per-instance
// guards when the template is light (`split`), as in emitItems.
void emitGroups(std::ostringstream& os, int k, const symgb_kernel_desc& d, unsigned S, int tpb, int items, int l2,
                const std::string& b0, const char* indent, bool split) {
    const std::uint64_t n = d.num_instances;
    const std::uint64_t groups = (n + items - 1) / items, full = n / items;
    os << indent << "const unsigned long long t = (" << b0 << ") * " << tpb << "ull + threadIdx.x;\n"
       << indent << "const unsigned long long g = t / " << S << "ull;\n"
       << indent << "const unsigned s = (unsigned)(t % " << S << "ull);\n";
    if (split && full)
        os << indent << "if (g < " << u64(full) << ") symgbGroup" << k << "<" << l2 << ", " << items
           << ", true>(x, xw, p, c, res, dp, g, s);\n"
           << indent << "else if (g < " << u64(groups) << ") symgbGroup" << k << "<" << l2 << ", " << items
           << ", false>(x, xw, p, c, res, dp, g, s);\n";
    else
        os << indent << "if (g < " << u64(groups) << ") symgbGroup" << k << "<" << l2 << ", " << items
           << ", false>(x, xw, p, c, res, dp, g, s);\n";
}

// The work of kernel k in either item layout.
void emitWork(std::ostringstream& os, int k, const symgb_kernel_desc& d, const Call& call, unsigned S, int tpb,
              int items, int l2, const std::string& b0, const char* indent, bool grouped, int order) {
    const bool split = call.ops * (std::size_t)items <= kSplitOps;
    if (grouped) emitGroups(os, k, d, S, tpb, items, l2, b0, indent, split);
    else emitItems(os, k, call, d.num_instances * S, S, tpb, items, l2, b0, indent, split, order);
}

// Dispatch of block `b` over the kernels of one launch (kernel-major block
// ranges, each piece's work items in consecutive blocks).
void emitDispatch(std::ostringstream& os, const std::vector<int>& ks, const std::vector<symgb_kernel_desc>& descs,
                  const std::vector<std::vector<Call>>& calls, unsigned S, int tpb, int items, int l2,
                  const char* indent, bool grouped, int order = 0) {
    std::uint64_t first = 0;
    const std::string inner = std::string(indent) + "    ";
    for (int k : ks) {
        const std::uint64_t blocks = kernelBlocks(descs[k], S, tpb, items, grouped);
        for (const Call& call : calls[k]) {
            os << indent << (first ? "else " : "") << "if (b < " << u64(first + blocks) << ") {\n";
            emitWork(os, k, descs[k], call, S, tpb, items, l2, "b - " + u64(first), inner.c_str(), grouped, order);
            os << indent << "}\n";
            first += blocks;
        }
    }
}

std::uint64_t blocksOf(const std::vector<int>& ks, const std::vector<symgb_kernel_desc>& descs,
                       const std::vector<std::vector<Call>>& calls, unsigned S, int tpb, int items, bool grouped) {
    std::uint64_t b = 0;
    for (int k : ks) b += kernelBlocks(descs[k], S, tpb, items, grouped) * calls[k].size();
    return b;
}

int checkedItems(int items) {
    if (items != 1 && items != 2 && items != 4) throw std::runtime_error("codegen: items per thread must be 1, 2 or 4");
    return items;
}

}  // namespace

extern const char* const kJitPrelude;

namespace {

// `__launch_bounds__(tpb)` or, with a minimum CTA count per SM that fits the
// SM's 2048 threads, `__launch_bounds__(tpb, minBlocks)`.
std::string launchBounds(int tpb, int minBlocks) {
    std::string s = "__launch_bounds__(" + std::to_string(tpb);
    const int fit = std::min(minBlocks, 2048 / std::max(1, tpb));
    if (fit > 0) s += ", " + std::to_string(fit);
    return s + ")";
}

// Every launch waits for its predecessor before its first read of x
// (programmatic dependent launch): only the wait of the reading grid itself makes
// earlier grids' writes visible to it.  It lets the next one in when its
// own work is done.  One work item per thread (strided): the wait goes behind
// the table loads of the body, which nothing writes (template argument ORDER),
// and the tables arrive while the predecessor drains.  Returns that argument.
int emitPrologue(std::ostringstream& os, bool inBody) {
    if (inBody) return 1;
    os << "    x = symgbOrder<1>(x);\n";
    return 0;
}

void emitEpilogue(std::ostringstream& os) { os << "    symgbLaunchDependents();\n"; }

}  // namespace

GroupedTables groupedTables(const std::vector<symgb_kernel_desc>& descs) {
    GroupedTables t;
    for (const auto& d : descs) {
        const std::uint64_t stride = (d.num_instances + 3) / 4 * 4;
        t.stride.push_back(stride);
        t.indexBase.push_back(t.indexSize);
        t.constBase.push_back(t.constSize);
        t.indexSize += stride * d.num_index_rows;
        t.constSize += stride * d.num_constant_rows;
    }
    return t;
}

namespace {

bool overlap(const SlotUse::Range& a, const SlotUse::Range& b) {
    return std::max(a.first, b.first) < std::min(a.second, b.second);
}

}  // namespace

SlotUse::Range SlotUse::writes(std::size_t k) const {
    const symgb_kernel_desc& d = descs[k];
    return Range(d.output_offset, d.output_offset + d.num_instances * d.num_output_rows);
}

// The bounds of a kernel's reads settle it for plans in memory order; the table
// is only searched where they reach into `r`.
bool SlotUse::reads(std::size_t k, const Range& r) const {
    if (readLo[k] > readHi[k] || !overlap(Range(readLo[k], readHi[k] + 1), r)) return false;
    const symgb_kernel_desc& d = descs[k];
    for (std::uint32_t a = 0; a < d.num_access; ++a) {
        const std::uint32_t* row = index + d.index_offset + (std::uint64_t)d.access[2 * a] * d.num_instances;
        const long long offset = d.access[2 * a + 1];
        for (std::uint64_t i = 0; i < d.num_instances; ++i) {
            const std::uint64_t slot = (std::uint64_t)((long long)row[i] + offset);
            if (slot >= r.first && slot < r.second) return true;
        }
    }
    return false;
}

std::vector<char> readsOwnRows(const SlotUse& use) {
    std::vector<char> own;
    for (std::size_t k = 0; k < use.descs.size(); ++k) own.push_back(use.reads(k, use.writes(k)));
    return own;
}

std::vector<char> besideEarlier(const SlotUse& use) {
    std::vector<char> beside(use.descs.size(), 0);
    std::vector<std::size_t> group;
    std::vector<SlotUse::Range> written;  // by the group, adjoining ranges merged
    for (std::size_t k = 0; k < use.descs.size(); ++k) {
        if (!use.descs[k].num_instances) continue;
        const SlotUse::Range w = use.writes(k);
        bool free = !group.empty();
        for (std::size_t j = 0; j < written.size() && free; ++j) free = !overlap(w, written[j]) && !use.reads(k, written[j]);
        for (std::size_t j = 0; j < group.size() && free; ++j) free = !use.reads(group[j], w);
        if (!free) {
            group.clear();
            written.clear();
        }
        beside[k] = free;
        group.push_back(k);
        if (!written.empty() && written.back().second == w.first) written.back().second = w.second;
        else written.push_back(w);
    }
    return beside;
}

JitSource generateModule(const std::vector<symgb_kernel_desc>& descs, int numLevels, const JitConfig& cfg) {
    JitSource out;
    std::ostringstream os;
    const unsigned S = cfg.numSets;
    if (cfg.itemLayout != SYMGB_ITEMS_STRIDED && cfg.itemLayout != SYMGB_ITEMS_GROUPED)
        throw std::runtime_error("codegen: unknown item layout");
    const bool grouped = cfg.itemLayout == SYMGB_ITEMS_GROUPED;
    out.grouped = grouped;
    GroupedTables gt;
    if (grouped) gt = groupedTables(descs);
    os << "// symgb compiled module: " << descs.size() << " kernels, " << numLevels << " levels, " << S
       << " value sets, math " << (cfg.math == SYMGB_MATH_FAST ? "fast" : "exact") << ", schedule " << cfg.kind
       << "\n";
    os << (cfg.kind == JIT_PERSISTENT ? "#define SYMGB_XR\n" : "#define SYMGB_XR __restrict__\n");
    os << kJitPrelude << "\n";
    // Loads of the tables and of x: the read-only data path (ld.global.nc),
    // cached in L1 (ld.global.ca) or in L2 only (ld.global.cg); values written
    // earlier in the same launch (L2 = 1) always come from L2.  The read-only
    // path is for the tables alone: a chained launch is resident, waiting, while the
    // one before it still writes x, and that path is for what does not change
    // while a kernel is resident.  GB300, x through it and without: cotan
    // 100 x 100 11.45 / 11.45 us, cloth 64 x 64 44.08 / 44.08, 300 x 300 x 64 12.64 / 12.68 ms;
    // of five others drawn at random two lost 1.2 and 1.4 %.
    static const char* const kLoad[] = {"__ldg", "__ldca", "__ldcg"};
    static const char* const kLoadX[] = {"__ldca", "__ldca", "__ldcg"};
    if (cfg.loadPath < 0 || cfg.loadPath > 2) throw std::runtime_error("codegen: load path must be 0, 1 or 2");
    os << "#define SYMGB_LD(a) " << kLoad[cfg.loadPath] << "(a)\n";
    os << "template <int L2>\n__device__ __forceinline__ double symgbLoadX(const double* a) {\n"
          "    return L2 ? __ldcg(a) : " << kLoadX[cfg.loadPath] << "(a);\n}\n\n";
    if (grouped)
        os << "// Entries of IT consecutive instances of one padded table row (aligned).\n"
              "template <int IT>\n__device__ __forceinline__ void symgbLoadIdx(const unsigned* a, unsigned (&q)[IT]) {\n"
              "    if constexpr (IT == 4) {\n"
              "        const uint4 v = SYMGB_LD(reinterpret_cast<const uint4*>(a));\n"
              "        q[0] = v.x; q[1] = v.y; q[2] = v.z; q[3] = v.w;\n"
              "    } else if constexpr (IT == 2) {\n"
              "        const uint2 v = SYMGB_LD(reinterpret_cast<const uint2*>(a));\n"
              "        q[0] = v.x; q[1] = v.y;\n"
              "    } else {\n"
              "        q[0] = SYMGB_LD(a);\n"
              "    }\n}\n"
              "template <int IT>\n__device__ __forceinline__ void symgbLoadConst(const double* a, double (&v)[IT]) {\n"
              "    if constexpr (IT >= 2) {\n"
              "        #pragma unroll\n"
              "        for (int h = 0; h < IT; h += 2) {\n"
              "            const double2 u = SYMGB_LD(reinterpret_cast<const double2*>(a + h));\n"
              "            v[h] = u.x; v[h + 1] = u.y;\n"
              "        }\n"
              "    } else {\n"
              "        v[0] = SYMGB_LD(a);\n"
              "    }\n}\n\n";
    // Heavy bodies of a kernel that dispatches over several are functions of
    // their own: in one, their compile time grows with its square (Neo-Hookean
    // levels, nine templates of 600 operations: 4.9 -> 1.3 s).
    constexpr std::size_t kHeavyOps = 200;
    std::vector<int> intMuls = grouped ? std::vector<int>(descs.size(), 0) : integerProducts(descs, cfg.math, S);
    for (std::size_t k = 0; k < cfg.inPlace.size(); ++k)
        if (cfg.inPlace[k]) intMuls[k] = 0;  // an item evaluated again would read what it has stored
    std::vector<std::vector<Piece>> pieces(descs.size());
    if (!grouped) pieces = templatePieces(descs, cfg, intMuls);
    std::vector<std::size_t> templateOps;
    std::size_t heavy = 0;
    for (std::size_t k = 0; k < descs.size(); ++k) {
        templateOps.push_back(linearCode(descs[k], cfg.math, nullptr).size());
        if (descs[k].num_instances && templateOps[k] > kHeavyOps) heavy += std::max<std::size_t>(1, pieces[k].size());
    }
    const bool dispatch = cfg.kind != JIT_PLAIN && !grouped && heavy > 1;
    if (!cfg.directBase.empty() && (cfg.directBase.size() != descs.size() || S != 1))
        throw std::runtime_error("codegen: direct result rows need one value set and a row table per kernel");
    std::vector<std::vector<Call>> calls(descs.size());
    for (std::size_t k = 0; k < descs.size(); ++k) {
        const std::vector<std::int64_t>* direct = cfg.directBase.empty() ? nullptr : &cfg.directBase[k];
        if (direct)
            for (std::int64_t b : *direct) out.direct |= b >= 0;
        const bool called = dispatch && templateOps[k] > kHeavyOps;
        const std::string id = std::to_string(k);
        const std::size_t ops =
            emitBody(os, (int)k, descs[k], cfg.math, S, grouped ? &gt : nullptr, direct, called);
        if (intMuls[k]) {
            os << "#ifdef SYMGB_ORDERED\n";
            emitBody(os, (int)k, descs[k], cfg.math, S, nullptr, direct, called, intMuls[k]);
            os << "template <int L2>\n__device__ __noinline__ void symgbRedo" << k
               << "(const double* x, double* xw, const unsigned* p, const double* c, double* res, const unsigned* dp, "
                  "unsigned long long i, unsigned s) {\n    symgbBody"
               << k << "<L2>(x, xw, p, c, res, dp, i, s);\n}\n#endif\n\n";
            calls[k].push_back({"symgbMixed" + id, ops, true});
        } else if (pieces[k].size() > 1) {
            os << "#ifdef SYMGB_ORDERED\n";
            for (std::size_t q = 0; q < pieces[k].size(); ++q) {
                emitBody(os, (int)k, descs[k], cfg.math, S, nullptr, direct, called, 0, &pieces[k][q], (int)q);
                calls[k].push_back({"symgbPart" + id + "_" + std::to_string(q), ops, false});
            }
            os << "#endif\n\n";
        } else {
            calls[k].push_back({"symgbBody" + id, ops, false});
        }
    }
    const char* params = "(const double* SYMGB_XR x, double* SYMGB_XR xw, const unsigned* __restrict__ p, "
                         "const double* __restrict__ c, double* __restrict__ res, const unsigned* __restrict__ dp";
    // Kernels of each level, heaviest first (their blocks are dispatched first).
    std::vector<std::vector<int>> byLevel(numLevels);
    for (std::size_t k = 0; k < descs.size(); ++k) {
        const int L = descs[k].level;
        if (L < 0 || L >= numLevels) throw std::runtime_error("codegen: kernel level out of range");
        if (descs[k].num_instances) byLevel[L].push_back((int)k);
    }
    if (cfg.kind == JIT_PLAIN) {
        for (int k = 0; k < (int)descs.size(); ++k) {
            if (!(descs[k].num_instances * S)) continue;
            const int tpb = cfg.kernelTpb.at(k);
            const int items = checkedItems(cfg.kernelItems.at(k));
            const std::string name = "symgb_k" + std::to_string(k);
            os << "extern \"C\" __global__ void " << launchBounds(tpb, cfg.minBlocks) << " " << name << params << ") {\n";
            const int order = emitPrologue(os, items == 1 && !grouped);
            os << "    const unsigned long long b = blockIdx.x;\n";
            emitDispatch(os, {k}, descs, calls, S, tpb, items, 0, "    ", grouped, order);
            emitEpilogue(os);
            os << "}\n\n";
            out.launches.push_back({name, k, -1, blocksOf({k}, descs, calls, S, tpb, items, grouped), tpb, items, false});
        }
    } else if (cfg.kind == JIT_LEVELS) {
        for (int L = 0; L < numLevels; ++L) {
            std::vector<int> ks = byLevel[L];
            if (ks.empty()) continue;
            std::stable_sort(ks.begin(), ks.end(), [&](int a, int b) {
                return descs[a].num_instances * (descs[a].num_nodes + 1) > descs[b].num_instances * (descs[b].num_nodes + 1);
            });
            const int tpb = cfg.levelTpb.at(L);
            const int items = checkedItems(cfg.levelItems.at(L));
            const std::string name = "symgb_l" + std::to_string(L);
            os << "extern \"C\" __global__ void " << launchBounds(tpb, cfg.minBlocks) << " " << name << params << ") {\n";
            const int order = emitPrologue(os, items == 1 && !grouped);
            os << "    const unsigned long long b = blockIdx.x;\n";
            emitDispatch(os, ks, descs, calls, S, tpb, items, 0, "    ", grouped, order);
            emitEpilogue(os);
            os << "}\n\n";
            out.launches.push_back({name, -1, L, blocksOf(ks, descs, calls, S, tpb, items, grouped), tpb, items, false});
        }
    } else if (cfg.kind == JIT_PERSISTENT) {
        const int tpb = cfg.levelTpb.at(0);
        const int items = checkedItems(cfg.levelItems.at(0));
        os << "struct SymgbBarrier { unsigned count; unsigned generation; int error; int pad; };\n";
        os << "extern \"C\" __global__ void " << launchBounds(tpb, cfg.minBlocks) << " symgb_persistent" << params
           << ", SymgbBarrier* bar, int* hostError, unsigned long long timeoutNs, unsigned extra) {\n"
           << "    symgbDependencyWait();\n";
        std::uint64_t most = 1;
        bool firstLevel = true;
        for (int L = 0; L < numLevels; ++L) {
            const std::vector<int>& ks = byLevel[L];
            if (ks.empty()) continue;
            if (!firstLevel)
                os << "    if (!symgbGridBarrier(bar, hostError, timeoutNs, gridDim.x + extra)) return;\n";
            const std::uint64_t nb = blocksOf(ks, descs, calls, S, tpb, items, grouped);
            most = std::max(most, nb);
            os << "    for (unsigned long long b = blockIdx.x; b < " << u64(nb) << "; b += gridDim.x) {\n";
            emitDispatch(os, ks, descs, calls, S, tpb, items, firstLevel ? 0 : 1, "        ", grouped);
            os << "    }\n";
            firstLevel = false;
        }
        os << "}\n\n";
        out.launches.push_back({"symgb_persistent", -1, -1, most, tpb, items, true});
    } else {
        throw std::runtime_error("codegen: unknown schedule");
    }
    out.source = os.str();
    return out;
}

}  // namespace engine
}  // namespace symgb
