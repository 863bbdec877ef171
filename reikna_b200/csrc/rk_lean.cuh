// Lean line passes: a CTA transforms one tile of NL lines whose two sides are of the
// pass' own complex type with plain strides and byte offsets that fit 32 bits (plan
// temporaries and user arrays below 4 GB, the latter without cropping, additive terms or
// format conversions).  Others take line_body (rk_kernels.cuh).
//
// What bounds them is HBM (16 or 32 bytes an element against a few dozen instructions),
// as long as enough warps wait on loads at once, so they are built for occupancy and few
// instructions:
//  * one 64-bit base and 32-bit byte offsets (one multiply-add an address; the 64-bit
//    addresses of 16 strided rows took 32 registers and spilled), line indices split by
//    multiplication with reciprocals from the host;
//  * contiguous complex64 lines of up to 1024 points live in one warp or a part of it:
//    the exchange between two stages needs no block barrier;
//  * two stages where 32 elements a thread make that possible (512 = 32 x 16,
//    1024 = 32 x 32): one exchange instead of two.
// Measured on 16 Mi complex64 elements in three rotating buffer sets (a copy at the
// measured peak takes 41.6 us): contiguous lines of 64 / 256 / 1024 / 4096 points 42.7 /
// 43.1 / 44.9 / 49.2 us, strided ones of 32 / 128 / 256 / 512 points 43.2 / 47.0 / 49.2 /
// 51.6 us.  Whole calls against the kernels that ran before: 16384 x 1024 inverse 62.4 ->
// 47.6 us (persistent TMA-fed passes), 16 x 262144 84.2 -> 32.5 us (two strided passes with
// table twiddles), 2048 x 2048 67.4 -> 34.4 us.
#pragma once
#define RK_PACKED_F32   // packed complex64 sums (rk_dft.cuh)
#include "rk_internal.h"
#include "rk_kernels.cuh"
#include "rk_lean.h"

namespace rk {

// ------------------------------------------------------------------------------
// radix plans: RT elements a thread, stage radices R[] (each divides RT).  A plan whose
// first and last radix agree holds a line's output at the positions the next FFT of the
// same plan reads its input from: the two FFTs of a Bluestein pass then need no exchange
// between them.
// ------------------------------------------------------------------------------
template <int RT_, int... Rs> struct LeanRadix {
    static constexpr int RT = RT_;
    static constexpr int R[] = {Rs...};
    static constexpr int NS = sizeof...(Rs);
};
template <typename T, int L, int MODE, bool BLUE> struct LeanPlan;
#define RK_LP(TY, LL, MD, BL, ...) \
    template <> struct LeanPlan<TY, LL, MD, BL> : LeanRadix<__VA_ARGS__> {};
RK_LP(float, 16, MODE_POS, false, 4, 4, 4)
RK_LP(float, 32, MODE_POS, false, 8, 8, 4)
RK_LP(float, 64, MODE_POS, false, 8, 8, 8)
RK_LP(float, 128, MODE_POS, false, 16, 16, 8)
RK_LP(float, 256, MODE_POS, false, 16, 16, 16)
RK_LP(float, 512, MODE_POS, false, 32, 32, 16)
RK_LP(float, 1024, MODE_POS, false, 32, 32, 32)
RK_LP(float, 2048, MODE_POS, false, 16, 16, 16, 8)
RK_LP(float, 4096, MODE_POS, false, 16, 16, 16, 16)
RK_LP(float, 8192, MODE_POS, false, 32, 32, 16, 16)
RK_LP(float, 16384, MODE_POS, false, 32, 32, 32, 16)
RK_LP(float, 2, MODE_LANE, false, 2, 2)
RK_LP(float, 4, MODE_LANE, false, 4, 4)
RK_LP(float, 8, MODE_LANE, false, 8, 8)
RK_LP(float, 16, MODE_LANE, false, 16, 16)
RK_LP(float, 32, MODE_LANE, false, 8, 8, 4)
RK_LP(float, 64, MODE_LANE, false, 8, 8, 8)
RK_LP(float, 128, MODE_LANE, false, 16, 16, 8)
RK_LP(float, 256, MODE_LANE, false, 16, 16, 16)
RK_LP(float, 512, MODE_LANE, false, 32, 32, 16)
RK_LP(float, 1024, MODE_LANE, false, 32, 32, 32)
RK_LP(double, 16, MODE_POS, false, 4, 4, 4)
RK_LP(double, 32, MODE_POS, false, 8, 8, 4)
RK_LP(double, 64, MODE_POS, false, 8, 8, 8)
RK_LP(double, 128, MODE_POS, false, 16, 16, 8)
RK_LP(double, 256, MODE_POS, false, 16, 16, 16)
RK_LP(double, 512, MODE_POS, false, 8, 8, 8, 8)
RK_LP(double, 1024, MODE_POS, false, 16, 16, 16, 4)
RK_LP(double, 2048, MODE_POS, false, 16, 16, 16, 8)
RK_LP(double, 4096, MODE_POS, false, 16, 16, 16, 16)
RK_LP(double, 8192, MODE_POS, false, 16, 16, 16, 16, 2)
RK_LP(double, 2, MODE_LANE, false, 2, 2)
RK_LP(double, 4, MODE_LANE, false, 4, 4)
RK_LP(double, 8, MODE_LANE, false, 8, 8)
RK_LP(double, 16, MODE_LANE, false, 16, 16)
RK_LP(double, 32, MODE_LANE, false, 8, 8, 4)
RK_LP(double, 64, MODE_LANE, false, 8, 8, 8)
RK_LP(double, 128, MODE_LANE, false, 16, 16, 8)
RK_LP(double, 256, MODE_LANE, false, 16, 16, 16)
RK_LP(double, 512, MODE_LANE, false, 16, 16, 16, 2)
// Bluestein passes (padded length M = L)
RK_LP(float, 16, MODE_POS, true, 4, 4, 4)
RK_LP(float, 32, MODE_POS, true, 8, 8, 4)
RK_LP(float, 64, MODE_POS, true, 8, 8, 8)
RK_LP(float, 128, MODE_POS, true, 16, 16, 8)
RK_LP(float, 256, MODE_POS, true, 16, 16, 16)
RK_LP(float, 512, MODE_POS, true, 32, 32, 16)
RK_LP(float, 1024, MODE_POS, true, 32, 32, 32)
RK_LP(float, 2048, MODE_POS, true, 16, 16, 8, 16)
RK_LP(float, 4096, MODE_POS, true, 16, 16, 16, 16)
RK_LP(float, 8192, MODE_POS, true, 32, 16, 32, 16)
RK_LP(float, 16384, MODE_POS, true, 32, 32, 16, 32)
RK_LP(float, 16, MODE_LANE, true, 4, 4, 4)
RK_LP(float, 32, MODE_LANE, true, 8, 8, 4)
RK_LP(float, 64, MODE_LANE, true, 8, 8, 8)
RK_LP(float, 128, MODE_LANE, true, 16, 16, 8)
RK_LP(float, 256, MODE_LANE, true, 16, 16, 16)
RK_LP(float, 512, MODE_LANE, true, 32, 32, 16)
RK_LP(float, 1024, MODE_LANE, true, 32, 32, 32)
RK_LP(float, 2048, MODE_LANE, true, 32, 32, 2, 32)
RK_LP(double, 16, MODE_POS, true, 4, 4, 4)
RK_LP(double, 32, MODE_POS, true, 8, 8, 4)
RK_LP(double, 64, MODE_POS, true, 8, 8, 8)
RK_LP(double, 128, MODE_POS, true, 16, 16, 8)
RK_LP(double, 256, MODE_POS, true, 16, 16, 16)
RK_LP(double, 512, MODE_POS, true, 8, 8, 8, 8)
RK_LP(double, 1024, MODE_POS, true, 16, 16, 4, 16)
RK_LP(double, 2048, MODE_POS, true, 16, 16, 8, 16)
RK_LP(double, 4096, MODE_POS, true, 16, 16, 16, 16)
RK_LP(double, 8192, MODE_POS, true, 16, 16, 2, 16, 16)
RK_LP(double, 16, MODE_LANE, true, 4, 4, 4)
RK_LP(double, 32, MODE_LANE, true, 8, 8, 4)
RK_LP(double, 64, MODE_LANE, true, 8, 8, 8)
RK_LP(double, 128, MODE_LANE, true, 16, 16, 8)
RK_LP(double, 256, MODE_LANE, true, 16, 16, 16)
RK_LP(double, 512, MODE_LANE, true, 16, 16, 2, 16)
RK_LP(double, 1024, MODE_LANE, true, 16, 16, 4, 16)
#undef RK_LP

// Plan of a few complex128 lines' four-step first pass (VAR 8): 512-point columns on 8 elements
// a thread, whose twice as many threads hide its chain of table twiddle loads while
// they do not fill the GPU.  2^18 points, 8 against 16 elements: 1 line 14.7 us against 19.7, 2
// 15.3 against 21.5, 4 24.3 against 23.8, but 8 lines 48.6 against 46.9 and 64 328 against 285;
// 2^19 points: 1 line 19.7 against 20.7, 2 30.9 both.
template <typename T, int L, int MODE, int VAR> struct LeanPick {
    using P = LeanPlan<T, L, MODE, VAR == 1>;
};
template <> struct LeanPick<double, 512, MODE_LANE, 8> {
    using P = LeanRadix<8, 8, 8, 8>;
};

// stage twiddle table of a plan: [m - 1][j1] of stage s after the earlier stages'
template <int L, class P> struct LeanTw {
    static constexpr int size_of(int s) {
        int p = 1;
        for (int i = 0; i < s; ++i) p *= P::R[i];
        return (P::R[s] - 1) * (L / (p * P::R[s]));
    }
    static constexpr int offset(int s) {
        int o = 0;
        for (int i = 0; i < s; ++i) o += size_of(i);
        return o;
    }
    static constexpr int total() { return P::NS > 1 ? offset(P::NS - 1) : 0; }
};

// VAR 0: plain; 1: Bluestein bodies (rk_lean_blue.cuh: two FFTs of the line with the
// kernel spectrum between); 2: contiguous lines stored lane-fastest (transposed) through
// shared memory; 5: the same for magnitudes (rk_lean_real.cuh); 8: plain, a few lines'
// four-step first pass (LeanPick)
template <typename T, int L, int MODE, int VAR> struct LeanCfg {
    using P = typename LeanPick<T, L, MODE, VAR>::P;
    using V = cplx<T>;
    static constexpr int RT = P::RT, TPL = L / RT, ESZ = sizeof(V);
    static constexpr int SEG = 128 / ESZ;   // elements of a 128-byte segment
    // contiguous lines: 128 threads a CTA for the bodies of 16 and more elements a thread
    // (finer tiles than 256 threads at the same occupancy), whole lines
    static constexpr int NT_POS = RT >= 16 ? 128 : 256;
    static constexpr int NL_POS = TPL >= NT_POS ? 1 : NT_POS / TPL;
    // transposed store: segments of 64 bytes and more a position
    static constexpr int NL_T0 = NL_POS < SEG / 2 ? SEG / 2 : NL_POS;
    // (magnitudes are half as wide: as many lines as 256 threads hold)
    static constexpr int NL_T1 = NL_T0 * TPL < 256 && NL_T0 < SEG ? 2 * NL_T0 : NL_T0;
    static constexpr int NL_T = VAR == 5 ? NL_T1 : NL_T0;
    // strided lines: one 128-byte segment of adjacent lines a position, or half of one
    // where a tile would pass 64 KB
    static constexpr int NL_L0 = TPL >= 128 ? 1 : 128 / TPL;
    static constexpr int NL_L1 = NL_L0 < SEG ? SEG : NL_L0;
    static constexpr int NL_L2 = NL_L1 * L * ESZ > 65536 && NL_L1 > SEG / 2 ? SEG / 2 : NL_L1;
    static constexpr int NL_LANE = NL_L2 * L * ESZ > 65536 ? NL_L2 / 2 : NL_L2;
    static constexpr int NL = MODE == MODE_LANE ? NL_LANE : VAR == 2 || VAR == 5 ? NL_T : NL_POS;
    static constexpr int NT = NL * TPL;
    // every line inside one warp: exchanges need only a warp barrier
    static constexpr bool WARP = MODE == MODE_POS && TPL <= 32;
    // one pad word for each R0 positions: both stage orders then meet every bank once
    // (a half-warp of 8-byte words, a quarter-warp of 16-byte words)
    static constexpr int LS = L + L / P::R[0];
    static constexpr bool LPAD = MODE == MODE_LANE && NL < SEG && P::NS > 1;
    // transposed read-back: a half-warp takes 16 / NL positions of NL lines (16-byte
    // words: 8 / NL)
    static constexpr int D = (SEG > NL) ? SEG / NL : 1;
    static constexpr int EX = MODE == MODE_POS ? NL * LS : L * NL + (LPAD ? L / P::R[0] * NL : 0);
    static constexpr int TLS = L + (2 * D > 1 ? 2 * D : 2);   // magnitudes, Nyquist bin included
    static constexpr int TR = VAR == 2 ? NL * (L + D) : VAR == 5 ? (NL * TLS + 1) / 2 : 0;
    static constexpr size_t SMEM = (P::NS > 1 || VAR != 0) ? (size_t)(EX > TR ? EX : TR) * ESZ : 0;
    // threads an SM the register budget is sized for: 32 complex64 (or 16 complex128)
    // elements a thread need 128 registers, 16 need 80, 8 and fewer 48
    static constexpr int WORDS = RT * ESZ / 4;
    static constexpr int TSM = WORDS >= 64 ? 512 : WORDS >= 32 ? 768 : WORDS >= 16 ? 1280 : 1536;
    static constexpr int MINB = TSM / NT > 0 ? TSM / NT : 1;
};

// The R-point DFT of a[0 .. R/2) followed by zeros
template <int R, typename V> __device__ __forceinline__ void dft_half(V* a) {
    if constexpr (R == 1) {
        return;
    } else if constexpr (R == 2) {
        a[1] = a[0];
    } else if constexpr (R == 4) {
        const V x = a[0], y = a[1], r = cmk<V>(y.y, -y.x);
        a[0] = x + y;
        a[2] = x - y;
        a[1] = x + r;
        a[3] = x - r;
    } else {
        using DF = Dft<R, 1, V>;
        constexpr int A = DF::A, B = DF::B;
#pragma unroll
        for (int n = 0; n < B; ++n) {
            if constexpr (A == 2) {
                a[B + n] = a[n];
            } else {
                const V x = a[n], y = a[B + n], r = cmk<V>(y.y, -y.x);
                a[n] = x + y;
                a[2 * B + n] = x - y;
                a[B + n] = x + r;
                a[3 * B + n] = x - r;
            }
        }
        DF::template step2<0>(a);
        DF::template step3<0>(a);
        // slot B k1 + k2 holds X[k1 + A k2]
        V t[R];
#pragma unroll
        for (int k = 0; k < R; ++k) t[k % B * A + k / B] = a[k];
#pragma unroll
        for (int k = 0; k < R; ++k) a[k] = t[k];
    }
}

// Programmatic dependent launch: a kernel's CTAs may be placed while the last CTAs of the
// kernel before it in the stream still run; they touch memory only after that kernel has
// completed and its writes are visible.  Between two kernels of one stream a full launch
// dependency costs 2 to 4 us (256 KB strided 64-point lines 4.1 -> 2.4 us a pass, 8.4 MB
// 6.2 -> 4.0, 134 MB 43.7 -> 41.6).
__device__ __forceinline__ void lean_begin() {
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    asm volatile("griddepcontrol.wait;" ::: "memory");
}
inline cudaError_t lean_launch(void (*k)(LeanParams), unsigned nb, int nt, size_t smem, const LeanParams& p, cudaStream_t st) {
    if (nb == 0) return cudaSuccess;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(nb, 1, 1);
    cfg.blockDim = dim3(nt, 1, 1);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute a[1];
    a[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    a[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = a;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, k, p);
}

// First line of the CTA's tile.  Every second launch of a chain takes its tiles in
// descending order: it then starts with the lines the launch before wrote last, which L2
// still holds (three passes over 134 MB 133.7 -> 129.4 us, two over 101 MB 67.4 -> 62.8;
// nothing where the whole array stays in L2).
__device__ __forceinline__ uint32_t lean_tile(const LeanParams& p) {
    return p.rev ? gridDim.x - 1 - blockIdx.x : blockIdx.x;
}

template <bool WARP> __device__ __forceinline__ void lean_sync() {
    if constexpr (WARP)
        __syncwarp();
    else
        __syncthreads();
}

template <typename T, int L, int MODE, int VAR> struct LeanEngine {
    using V = cplx<T>;
    using C = LeanCfg<T, L, MODE, VAR>;
    using P = typename C::P;
    using TwT = LeanTw<L, P>;
    static constexpr int RT = P::RT, TPL = C::TPL, NS = P::NS, NL = C::NL;
    static constexpr int R0 = P::R[0], RL = P::R[NS - 1];

    // shared-memory index of a position, line offset excluded.  Every position below is a
    // thread's base plus a compile-time constant whose remainders by R0 never carry, so
    // spos(base + k) = spos(base) + spos(k): one register addresses a whole stage (left to
    // the compiler, the pads cost an address register an element, and the passes with two
    // FFTs kept them all: 896 bytes of spills at 8192 points)
    static __host__ __device__ constexpr int spos(int pos) {
        return MODE == MODE_POS ? pos + pos / R0 : pos * NL + (C::LPAD ? pos / R0 * NL : 0);
    }
    static __device__ __forceinline__ int sline(int ln) { return MODE == MODE_POS ? ln * C::LS : ln; }
    // position of element i: thread's b plus a compile-time offset
    static constexpr int ik(int i) { return TPL * (i / R0) + (L / R0) * (i % R0); }
    static constexpr int ok(int i) { return TPL * (i / RL) + (L / RL) * (i % RL); }

    // Bluestein passes take plain loads, not the read-only path: those the compiler would
    // take to be the same in the second FFT, and keep and spill them
    static __device__ __forceinline__ V twiddle(const V* p) {
        if constexpr (VAR == 1) return *p;
        else return __ldg(p);
    }
    // HALF: the upper half of the line's inputs is zero (and v's slots for it are unset)
    template <int S, int PP, bool HALF> static __device__ __forceinline__ void stages(V* v, V* sm, int ln, int tb, const V* tw) {
        constexpr int R = P::R[S], NB = RT / R;
        if constexpr (S + 1 < NS) {
            constexpr int J = L / (PP * R);
            // butterfly b = tb + TPL z: l = b % PP and j1 = b / PP split the same way.
            const V* tws = tw + TwT::offset(S) + tb / PP;
            V* wr = sm + sline(ln) + spos(tb % PP + PP * R * (tb / PP));
            if constexpr (S > 0) lean_sync<C::WARP>();
#pragma unroll
            for (int z = 0; z < NB; ++z) {
                if constexpr (HALF) dft_half<R>(v + z * R);
                else dft<R>(v + z * R);
#pragma unroll
                for (int m = 1; m < R; ++m) v[z * R + m] = cmul(v[z * R + m], twiddle(tws + ((m - 1) * J + TPL * z / PP)));
#pragma unroll
                for (int m = 0; m < R; ++m) wr[spos(TPL * z % PP + PP * R * (TPL * z / PP) + PP * m)] = v[z * R + m];
            }
            lean_sync<C::WARP>();
            constexpr int R2 = P::R[S + 1], NB2 = RT / R2;
            const V* rd = sm + sline(ln) + spos(tb);
#pragma unroll
            for (int z = 0; z < NB2; ++z)
#pragma unroll
                for (int m = 0; m < R2; ++m) v[z * R2 + m] = rd[spos(TPL * z + (L / R2) * m)];
            stages<S + 1, PP * R, false>(v, sm, ln, tb, tw);
        } else {
#pragma unroll
            for (int z = 0; z < NB; ++z) {
                if constexpr (HALF) dft_half<R>(v + z * R);
                else dft<R>(v + z * R);
            }
        }
    }
    template <bool HALF = false> static __device__ __forceinline__ void run(V* v, V* sm, int ln, int tb, const V* tw) {
        stages<0, 1, HALF>(v, sm, ln, tb, tw);
    }
};

__device__ __forceinline__ uint32_t fd_div(const FastDiv& f, uint32_t n) {
    return (uint32_t)(((uint64_t)n * f.m) >> f.sh);
}

// byte offset of a line on one side
__device__ __forceinline__ uint32_t lean_offset(const LeanSide& s, uint32_t line) {
    uint32_t off = 0;
#pragma unroll
    for (int d = 0; d < LEAN_DIMS; ++d) {
        if (d < s.nd) {
            const uint32_t q = fd_div(s.dim[d].size, line);
            uint32_t r = line - q * s.dim[d].size.d + s.dim[d].shift;
            if (r >= s.dim[d].size.d) r -= s.dim[d].size.d;
            off += r * s.dim[d].stride;
            line = q;
        }
    }
    return off;
}

// W_{tw4N}^e from the two-level FP64 table
__device__ __forceinline__ double2 lean_tw4(const LeanParams& p, uint32_t e) {
    const uint32_t k = (e & p.tw4_mask) << p.tw4_sh;
    const double2 hi = __ldg(reinterpret_cast<const double2*>(p.tw4_hi) + (k >> 12));
    const double2 lo = __ldg(reinterpret_cast<const double2*>(p.tw4_lo) + (k & (TW4_HALF - 1)));
    return cmul(hi, lo);
}

// Four-step twiddles W^(c k) on a thread's outputs (positions tb + ok(i)).  complex64:
// the powers of one step in FP64, rounded once each (one FP64 product an element; two
// 16-byte table reads an element, scattered over c, made the pass wait on L1: 262144-point
// lines 61.9 us a pass, 20.5 with the products and the lean tile).  complex128 reads the
// tables for every element, whose error the products would exceed.
template <typename T, class E> __device__ __forceinline__ void lean_tw4_block(const LeanParams& p, uint32_t c, int tb, cplx<T>* v) {
    constexpr int RT = E::RT, RL = E::RL, TPL = E::TPL;
    if constexpr (sizeof(T) == 4) {
        const double2 st = lean_tw4(p, c * (uint32_t)E::ok(1 % RL));
#pragma unroll
        for (int z = 0; z < RT / RL; ++z) {
            double2 w = lean_tw4(p, c * (uint32_t)(tb + TPL * z));
#pragma unroll
            for (int m = 0; m < RL; ++m) {
                v[z * RL + m] = cmul(v[z * RL + m], make_float2((float)w.x, (float)w.y));
                if (m + 1 < RL) w = cmul(w, st);
            }
        }
    } else {
#pragma unroll
        for (int i = 0; i < RT; ++i) v[i] = cmul(v[i], lean_tw4(p, c * (uint32_t)(tb + E::ok(i))));
    }
}

template <typename T, int N> __device__ __forceinline__ void lean_conj(cplx<T>* v) {
#pragma unroll
    for (int i = 0; i < N; ++i) v[i].y = -v[i].y;
}
template <typename T, int N> __device__ __forceinline__ void lean_scale(const LeanSide& s, cplx<T>* v) {
    const T re = (T)s.scale_re, im = (T)s.scale_im;
    if (im == T(0)) {
#pragma unroll
        for (int i = 0; i < N; ++i) v[i] = cscale(v[i], re);
    } else {
        const cplx<T> c = cmk<cplx<T>>(re, im);
#pragma unroll
        for (int i = 0; i < N; ++i) v[i] = cmul(v[i], c);
    }
}

// Loads of element i at position tb + K(i); UNIT: positions are adjacent in memory.
template <typename T, int L, int N, bool UNIT, class KF>
__device__ __forceinline__ void lean_load(const LeanSide& s, uint32_t off, int tb, KF K, cplx<T>* v) {
    using V = cplx<T>;
    if (s.shift == 0) {
        if constexpr (UNIT) {
            const V* lp = reinterpret_cast<const V*>(s.base + off) + tb;
#pragma unroll
            for (int i = 0; i < N; ++i) v[i] = lp[K(i)];
        } else {
            const uint32_t o0 = off + (uint32_t)tb * s.step;
#pragma unroll
            for (int i = 0; i < N; ++i) v[i] = *reinterpret_cast<const V*>(s.base + (o0 + (uint32_t)K(i) * s.step));
        }
    } else {
#pragma unroll
        for (int i = 0; i < N; ++i)
            v[i] = *reinterpret_cast<const V*>(s.base + (off + (uint32_t)((tb + K(i) + s.shift) & (L - 1)) * s.step));
    }
    if (s.flags & SF_SCALE) lean_scale<T, N>(s, v);
    if (s.flags & SF_PRE_CONJ) lean_conj<T, N>(v);
}

// Stores, after the conjugation and the scale.  HALF: element i and i ^ HALF sit half
// the axis apart (a remap by half the axis is then a register swap).
template <typename T, int L, int N, bool UNIT, int HALF, class KF>
__device__ __forceinline__ void lean_store(const LeanSide& s, uint32_t off, int tb, bool ok, KF K, cplx<T>* v) {
    using V = cplx<T>;
    if (s.flags & SF_PRE_CONJ) lean_conj<T, N>(v);
    if (s.flags & SF_SCALE) lean_scale<T, N>(s, v);
    if (!ok) return;
    int shift = s.shift;
    if (HALF > 0 && shift == L / 2) {
#pragma unroll
        for (int i = 0; i < N; ++i)
            if (!(i & HALF)) {
                const V t = v[i];
                v[i] = v[i | HALF];
                v[i | HALF] = t;
            }
        shift = 0;
    }
    if (shift == 0) {
        if constexpr (UNIT) {
            V* lp = reinterpret_cast<V*>(s.base + off) + tb;
#pragma unroll
            for (int i = 0; i < N; ++i) lp[K(i)] = v[i];
        } else {
            const uint32_t o0 = off + (uint32_t)tb * s.step;
#pragma unroll
            for (int i = 0; i < N; ++i) *reinterpret_cast<V*>(s.base + (o0 + (uint32_t)K(i) * s.step)) = v[i];
        }
    } else {
#pragma unroll
        for (int i = 0; i < N; ++i)
            *reinterpret_cast<V*>(s.base + (off + (uint32_t)((tb + K(i) + shift) & (L - 1)) * s.step)) = v[i];
    }
}

// Plain pass of contiguous (POS) or strided (LANE) lines; VAR 2: contiguous lines stored
// lane-fastest; TW4: four-step twiddles W^(c k) on the outputs.
template <typename T, int L, int MODE, int VAR, bool TW4>
__global__ void __launch_bounds__((LeanCfg<T, L, MODE, VAR>::NT), (LeanCfg<T, L, MODE, VAR>::MINB))
    k_lean(const __grid_constant__ LeanParams p) {
    using V = cplx<T>;
    using C = LeanCfg<T, L, MODE, VAR>;
    using E = LeanEngine<T, L, MODE, VAR>;
    constexpr int RT = E::RT, TPL = E::TPL, NL = E::NL;
    extern __shared__ __align__(16) unsigned char rk_smem[];
    V* sm = reinterpret_cast<V*>(rk_smem);
    lean_begin();
    const int tid = threadIdx.x;
    const int ln = MODE == MODE_POS ? tid / TPL : tid % NL;
    const int tb = MODE == MODE_POS ? tid % TPL : tid / NL;
    // lines past the end repeat the last one and store nothing
    const uint32_t line0 = lean_tile(p) * NL;
    const uint32_t line = min(line0 + ln, p.nlines - 1);
    V v[RT];
    lean_load<T, L, RT, MODE == MODE_POS>(p.ld, lean_offset(p.ld, line), tb, [](int i) { return E::ik(i); }, v);
    E::run(v, sm, ln, tb, reinterpret_cast<const V*>(p.tw));
    if constexpr (TW4) {
        const uint32_t q = fd_div(p.cI, line);
        lean_tw4_block<T, E>(p, q - fd_div(p.cC, q) * p.cC.d, tb, v);
    }
    if constexpr (VAR == 2) {
        __syncthreads();
#pragma unroll
        for (int i = 0; i < RT; ++i) sm[ln * (L + C::D) + tb + E::ok(i)] = v[i];
        __syncthreads();
        const int lane = tid % NL, p0 = tid / NL;
#pragma unroll
        for (int q = 0; q < RT; ++q) v[q] = sm[lane * (L + C::D) + p0 + TPL * q];
        const uint32_t sline = line0 + lane;
        lean_store<T, L, RT, false, (RT >= 2 ? RT / 2 : 0)>(p.st, lean_offset(p.st, min(sline, p.nlines - 1)), p0, sline < p.nlines,
                                           [](int q) { return TPL * q; }, v);
    } else {
        lean_store<T, L, RT, MODE == MODE_POS, E::RL / 2>(p.st, lean_offset(p.st, line), tb, line0 + ln < p.nlines,
                                                [](int i) { return E::ok(i); }, v);
    }
}

template <class C, int L> void lean_segments(std::vector<StageSeg>& out) {
    int pp = 1;
    for (int s = 0; s + 1 < C::P::NS; ++s) {
        const int R = C::P::R[s];
        out.push_back(StageSeg{LeanTw<L, typename C::P>::offset(s), L / pp, R, L / (pp * R)});
        pp *= R;
    }
}

template <typename T, int L, int MODE, int VAR, bool TW4> struct LeanLauncher {
    using C = LeanCfg<T, L, MODE, VAR>;
    static cudaError_t launch(const LeanParams& p, cudaStream_t st) {
        return lean_launch(k_lean<T, L, MODE, VAR, TW4>, (p.nlines + C::NL - 1) / C::NL, C::NT, C::SMEM, p, st);
    }
    // launch attributes (not allowed during stream capture, so set when a plan is made)
    static cudaError_t prepare() {
        if (C::SMEM <= 48 * 1024) return cudaSuccess;
        return cudaFuncSetAttribute(k_lean<T, L, MODE, VAR, TW4>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)C::SMEM);
    }
    static LeanInfo info() {
        LeanInfo r{};
        r.launch = &launch;
        r.prepare = &prepare;
        r.segments = &lean_segments<C, L>;
        r.tw_elems = LeanTw<L, typename C::P>::total();
        r.nl = C::NL;
        r.nt = C::NT;
        r.smem = C::SMEM;
        return r;
    }
};

}  // namespace rk
