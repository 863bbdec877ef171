// Launch parameters and lookup of the lean line passes (rk_lean.cuh).
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include <memory>
#include <vector>

namespace rk {

// n / d for n < 2^31 as (n * m) >> sh
struct FastDiv {
    uint32_t d, m;
    int32_t sh;
};
inline FastDiv fast_div(uint32_t d) {
    int s = 0;
    while ((1ull << s) < d) ++s;
    // m = ceil(2^(31 + s) / d): the error m d - 2^(31 + s) < d <= 2^s, times n < 2^31
    // stays below 2^(31 + s)
    const uint64_t m = ((1ull << (31 + s)) + d - 1) / d;
    return FastDiv{d, (uint32_t)m, 31 + s};
}

constexpr int LEAN_DIMS = 4;
struct LeanDim {
    FastDiv size;
    uint32_t stride;   // bytes
    uint32_t shift;    // index remap (r + shift) mod size
};
// Stage of a mixed-radix pass (rk_lean_mix.cuh): radix R after P = the product of the
// earlier ones, nb = L / R butterflies a line, J = nb / P twiddle groups
struct MixStage {
    uint32_t R, P, nb, J, tw;
    FastDiv bdiv, pdiv;   // by nb, by P
};
constexpr int MIX_STAGES = 4;
constexpr int MIX_SMEM = 200 * 1024;   // dynamic shared memory of a CTA at most
struct MixPlan {
    uint32_t n;
    int32_t ns;
    uint32_t nl, lsh;      // lines a tile (strided: a power of two, and its logarithm)
    uint32_t buf, pitch;   // elements of a buffer and of a line in it
    uint32_t pad;          // one pad word for each R0 positions (r0 divides by R0)
    uint32_t inplace;      // a thread has at most one butterfly a stage
    uint32_t bufs;         // buffers: one in place, or with nothing between first and last stage
    FastDiv r0;
    MixStage stage[MIX_STAGES];
};

// One side: a line index splits over the dims, innermost first; position j of the line is
// step bytes further for each j, after the remap (j + shift) mod L.
struct LeanSide {
    char* base;
    LeanDim dim[LEAN_DIMS];
    int32_t nd;
    uint32_t step;
    int32_t shift;
    int32_t flags;     // SF_SCALE, SF_PRE_CONJ
    double scale_re, scale_im;
};
struct LeanParams {
    LeanSide ld, st;
    const void* tw;
    const void* tw4_hi;
    const void* tw4_lo;
    FastDiv cI, cC;    // four-step co-index of a line: (line / I) mod C
    uint32_t nlines;
    int32_t rev;       // tiles in descending order
    uint32_t tw4_mask;
    int32_t tw4_sh;
    // Bluestein passes (rk_lean_blue.cuh): N, the element step of the axis index
    // a = c + j jB (columns of the three-pass form), chirp and kernel spectrum
    uint32_t blue_n, jB;
    const void* chirp;
    const void* blue_k;
    // real passes (rk_lean_real.cuh): w_k = exp(-i pi k / L), window pairs or null, bins
    // stored along the axis (Nyquist bin apart), LeanReal bits
    const void* rmix;
    const void* win;
    uint32_t bound;
    int32_t rflags;
    // mixed-radix passes: the plan on the device, lines and threads a CTA, shared memory
    const MixPlan* mix;
    uint32_t mix_nl, mix_nt, mix_smem;
    FastDiv mix_pairs;   // by n / 2 + 1, the bin pairs of a line (real transforms)
};
enum LeanReal : int32_t {
    LR_NYQ = 1,     // bin L is stored as well
    LR_PAIRS = 2,   // every line of the real array starts on a pair's boundary
    LR_NORM = 4,    // |X|^2 out, of the real type
    LR_SQRT = 8,    // its square root
};

struct StageSeg {      // one stage's twiddles of a table: W_Lp^(j1 m), 1 <= m < R, j1 < J
    int64_t off;
    int Lp, R, J;
};

struct LeanInfo {
    cudaError_t (*launch)(const LeanParams&, cudaStream_t);
    cudaError_t (*prepare)();
    void (*segments)(std::vector<StageSeg>&);
    int tw_elems;
    int nl;                // lines, threads and dynamic shared memory of a CTA
    int nt;
    size_t smem;
};
// What a plan keeps for a pass that a lean kernel takes
struct LeanPass {
    LeanInfo info;
    LeanParams prm;
    bool blue = false;        // a Bluestein body
    int real = 0;             // a real pass: its variant (4, 5, 6)
    // a plane pass: this is its rows, `second` its columns, mid the buffer between (null:
    // the output array)
    std::shared_ptr<const LeanPass> second;
    void* mid = nullptr;
    bool fuse_next = false;   // does the next pass' work as well (rows of the three-pass form)
    bool only = false;        // the pass' general parameters do not describe its whole work
};

// Mixed-radix passes: the kernel of a mode; real (contiguous lines): 1 RFFT, 2 IRFFT
void lean_mix_info_f32(int mode, int real, LeanInfo* out);
void lean_mix_info_f64(int mode, int real, LeanInfo* out);

// A plan's launches of one direction, but for the user's pointers
struct LeanChain {
    enum { FIXED = 0, INPUT = 1, OUTPUT = 2 };
    struct Item {
        cudaError_t (*launch)(const LeanParams&, cudaStream_t);
        LeanParams prm;           // sides of the user's arrays hold their offset from the pointer
        int32_t ld = FIXED, st = FIXED;
        uint32_t pair = 0;        // drop LR_PAIRS where the load's base is off this boundary
    };
    std::vector<Item> items;
};

// var 0 or 2 (transposed store); tw4: with four-step twiddles
bool lean_info_f32(int L, int mode, int var, bool tw4, LeanInfo* out);
bool lean_info_f64(int L, int mode, int var, bool tw4, LeanInfo* out);
// Bluestein bodies: var 1 whole lines (6 / 7: contiguous ones with the real-spectrum step
// after / before, RFFT and IRFFT), 3 rows and 4 / 5 first / last columns (strided
// lines) of the three-pass form
bool lean_blue_info_f32(int L, int mode, int var, LeanInfo* out);
bool lean_blue_info_f64(int L, int mode, int var, LeanInfo* out);
// real passes: var 6 bins or magnitudes, 5 magnitudes lane-fastest, 4 inverse
bool lean_real_info_f32(int L, int var, LeanInfo* out);
bool lean_real_info_f64(int L, int var, LeanInfo* out);

}  // namespace rk
