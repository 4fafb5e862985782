// Compiled executor: source generation (codegen.cpp) and run-time compilation
// (jit.cu).  A unit's kernels are emitted as straight-line CUDA C++ - the
// form of the reference's generated kernels (ComputeUnit.cpp:409-421), with
// 1, 2 or 4 work items per thread - compiled for sm_103a by NVRTC at first use
// and cached by source text, and launched in one of three schedules.
#pragma once
#include <cstdint>
#include <memory>
#include <string>
#include <utility>
#include <vector>

#include "symgb.h"

namespace symgb {
namespace engine {

enum JitKind : int {
    JIT_PLAIN = 0,       // one kernel per ComputeKernel, launched in plan order
    JIT_LEVELS = 1,      // one kernel per dependency level, all its ComputeKernels
    JIT_PERSISTENT = 2,  // one cooperative kernel over all levels, grid barriers between them
};

struct JitConfig {
    int kind = JIT_LEVELS;
    int math = SYMGB_MATH_FAST;
    unsigned numSets = 1;
    std::vector<int> kernelTpb;    // per ComputeKernel (JIT_PLAIN)
    std::vector<int> levelTpb;     // per level (JIT_LEVELS); [0] for JIT_PERSISTENT
    std::vector<int> kernelItems;  // work items per thread, per ComputeKernel (JIT_PLAIN)
    std::vector<int> levelItems;   // per level (JIT_LEVELS); [0] for JIT_PERSISTENT
    int minBlocks = 0;  // > 0: __launch_bounds__ minimum CTAs per SM (caps registers)
    int loadPath = 0;   // SYMGB_LOAD_*: data path of the table and x loads
    int itemLayout = 0;  // SYMGB_ITEMS_*: which work items a thread takes
    // Direct result writes (one value set): per kernel and output row, the
    // row's start in the result-position table `dp` - the row's results go to
    // res[dp[start + i]] instead of x - or -1; empty when none is direct.
    std::vector<std::vector<std::int64_t>> directBase;
    // Per kernel: it reads slots of its own output rows (readsOwnRows), so that
    // a thread has to read everything before it stores anything, once; empty:
    // none does.
    std::vector<char> inPlace;
};

// Grouped item layout (SYMGB_ITEMS_GROUPED): copies of the index and constant
// tables whose rows are padded to a multiple of 4 entries (the row's last
// entry repeated), so that a thread reads the entries of 1, 2 or 4
// consecutive instances of a row with one aligned vector load.  Kernel k's
// row r starts at indexBase[k] + r * stride[k] (constBase[k] + r * stride[k]
// for constants); stride[k] = n_k rounded up to a multiple of 4.
struct GroupedTables {
    std::vector<std::uint64_t> indexBase, constBase, stride;
    std::uint64_t indexSize = 0, constSize = 0;  // entries of the padded copies
};
GroupedTables groupedTables(const std::vector<symgb_kernel_desc>& descs);

// One launch of a module: entry name, ComputeKernel (plain) or level (levels)
// it covers, blocks needed to cover its work items, block size.
struct JitLaunch {
    std::string name;
    int kernel;
    int level;
    std::uint64_t blocks;
    int tpb;
    int items;  // work items per thread
    bool cooperative;  // persistent: grid capped at the co-resident maximum
};

struct JitSource {
    std::string source;
    std::vector<JitLaunch> launches;  // in execution order
    bool grouped = false;             // reads the padded tables (GroupedTables)
    bool direct = false;              // writes some results straight into res
};

// Generates the module for a unit's kernels (host only; throws
// std::runtime_error for templates it cannot express).
JitSource generateModule(const std::vector<symgb_kernel_desc>& descs, int numLevels, const JitConfig& cfg);

// What the kernels of a plan read and write, from the tables.  readLo[k],
// readHi[k]: least and greatest slot kernel k reads (lo > hi: none).
struct SlotUse {
    const std::vector<symgb_kernel_desc>& descs;
    const std::uint32_t* index;
    const std::vector<std::uint64_t>&readLo, &readHi;
    using Range = std::pair<std::uint64_t, std::uint64_t>;  // [first, second)
    Range writes(std::size_t k) const;
    bool reads(std::size_t k, const Range& r) const;
};

// Which kernels read slots that they write themselves (JitConfig::inPlace).
std::vector<char> readsOwnRows(const SlotUse& use);

// Which kernels of a plan may run beside those in front of them, in plan order
// (JIT_PLAIN): [k] is true where kernel k and the kernels back to the last one
// with false neither read nor write a slot that another of them writes.
// From the tables alone, so that a plan's level numbers need not be right.
std::vector<char> besideEarlier(const SlotUse& use);

// A compiled and loaded module (jit.cu).  `kernels[j]` is the cudaKernel_t
// of launches[j], stored as void* (the form the runtime's launch calls take).
struct JitModule {
    std::vector<JitLaunch> launches;
    std::vector<const void*> kernels;
    std::vector<int> registers;  // per launch: registers per thread of the compiled kernel
    std::vector<int> blocksPerSm;  // cooperative launches: most resident blocks of an SM
    double compileSeconds = 0;
    bool grouped = false;        // launch with the padded tables (GroupedTables)
    bool direct = false;         // writes some results straight into res
};

// Compiles `source` with NVRTC without loading it (no device needed).
int compileOnly(const std::string& source, double* seconds, std::string* err);

// Compiles (or finds in the process-wide cache) the module for `src`.
// Returns 0 or a SYMGB_ERR_* code with the message in *err.
int loadModule(const JitSource& src, std::shared_ptr<const JitModule>* out, std::string* err);

}  // namespace engine
}  // namespace symgb
