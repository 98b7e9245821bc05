// The batched trait peel specialised to one problem at context creation
// (straight-line CUDA C++ compiled with NVRTC); see sl_jit.cc.
#pragma once
#include <cuda_runtime.h>

#include <cstddef>
#include <cstdint>
#include <memory>
#include <string>
#include <vector>

namespace sl {

// One compiled slot program and the sizes its source needs.
struct JitProgramIn {
    const int32_t* words;
    size_t n_words;
    const float* consts;
    int F, M, n, W, Nnf, slots;
    double marker_trans;
    int zero_ok;             // a zero trait likelihood is a zero term, not an error
};

// Threads per block of the scorer with its values in registers, and whether its
// warps go through the code together.  Every warp fetches the straight-line code,
// and from about 8,000 words of program on it no longer stays in the instruction
// cache: there a block's warps keep together (barriers), and with up to 192 slots
// the registers are limited so that four blocks share an SM.  Apart, with all
// registers | together, so limited, 1, 4 and 32 graphs of 2,000 SNPs: 66 members
// (9,002 words) 19, 20, 84 | 18, 20, 80 us; 90 members (10,808) 28, 58, 271 | 27, 29,
// 152; 130 members (184 slots) 38, 77, 363 | 38, 40, 203 (in blocks of 512 43, 41, 206:
// one has to wait for 16 warps).  A short program only loses: 30 members (4,154
// words) 11, 12, 35 | 10, 11, 39 (12, 13, 46), 54 members (5,141) 13, 14, 59 | 14, 14, 59.  With many
// slots the registers left are too few: 731 slots (400 members) 0.71 ms with all,
// 0.93 in blocks of 512; in between, 204 to 343 slots gain as much in large calls (32
// graphs 360 -> 207, 336 -> 221 in blocks of 512) as they lose in small ones (37 -> 42,
// 35 -> 43) and keep theirs.  The form in shared memory: 64 graphs of 120 members
// 0.67 | 0.48 ms.
constexpr int kJitLodThreads = 128;
inline bool jit_lod_together(const JitProgramIn& in, bool shared) {
    return in.n_words >= 8000 && (shared || in.slots <= 192);
}

struct JitLod {
    void* lib = nullptr;     // cudaLibrary_t
    void* kern = nullptr;    // cudaKernel_t
    int threads = 0;
    bool shared = false;     // values in a shared-memory arena (else registers)
    size_t smem = 0;
    int regs = 0;
    int local_bytes = 0;     // spill space per thread
    int blocks_per_sm = 0;
    double compile_ms = 0.0;
};

// One NVRTC compile of a source for sm_103a.
struct JitBinary {
    std::string source;
    std::vector<char> cubin;
    std::string log;
    int rc = -1;             // 0: cubin holds the binary
    double compile_ms = 0.0;
    bool done = false;
};

// The cubin of `src`, compiled on the calling thread (no CUDA context is
// needed) or taken from a process-wide cache of recent sources; a caller
// asking for a source another thread is compiling waits for that compile.
// At most a few compiles run at once.  Thread-safe.
std::shared_ptr<const JitBinary> jit_binary(const std::string& src, const char* file);

// Load `kernel` from a cubin into the current device's context (a
// cudaLibrary_t and a cudaKernel_t); 0 on success, else -1 with the reason.
int jit_load_kernel(const std::vector<char>& cubin, const char* kernel, void** lib, void** kern, std::string* log);

// jit_binary, then jit_load_kernel.
int jit_compile_kernel(const std::string& src, const char* file, const char* kernel, void** lib, void** kern,
                       std::string* log);

std::string jit_lod_source(const JitProgramIn& in, int threads, bool shared);
int jit_lod_compile(const JitProgramIn& in, int threads, bool shared, JitLod* out, std::string* log);
void jit_lod_release(JitLod* j);
cudaError_t jit_lod_launch(const JitLod& j, const uint32_t* graphs, int64_t graph_words, int G, double* vals,
                           int* status, const float* partial, const double* lt, const double* la, int64_t ntask,
                           int sms, cudaStream_t s);

}  // namespace sl
