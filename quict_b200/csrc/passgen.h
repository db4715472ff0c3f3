// Generated source, parameter block and launch shape of a planned register pass.
#pragma once

#include <cstdint>
#include <string>
#include <vector>

namespace qs {

struct JitPass {
    std::string src;
    std::vector<uint64_t> params;  // the kernel's parameter block (16-byte multiple)
    std::vector<uint8_t> classes;  // value class of every matrix entry (what the source depends on)
    int threads = 0;
    size_t smem = 0;
};

// Single-buffered generated kernels (see passgen.cu): QS_JIT_SINGLE_BUFFER=0 / 1,
// else every pass but plain complex64 ones (tables: per-instance tables or
// EXPECT ops).
bool jit_single_buffer(bool c128, bool tables);

// Generate the planned register pass `regargs` (a RegArgs filled by build_reg;
// the struct has the same layout in every file that includes regtile.cuh).
// mats_host: the host matrix table in the state's precision.  with_source:
// also the text, not only the parameter block, classes and launch shape.
// devfn: see passgen.cu.  False when the pass is not generated.
bool gen_pass(const void* regargs, int R, bool c128, const void* mats_host, JitPass& out, bool with_source,
              const char* devfn = nullptr);

}  // namespace qs
