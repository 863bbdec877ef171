// Lean Bluestein passes.  With chirp[a] = exp(-i pi a^2 / N) and K the padded kernel's
// spectrum over M, y[a] = chirp[a] (IFFT_M(FFT_M(x chirp) K))[a]; the inverse FFT runs as
// the conjugate of a forward FFT of the conjugate.
//
//  * k_lean_blue: a whole line of M points a CTA.  N <= M / 2 always, so the upper half of
//    the first FFT's inputs is zero (its first butterflies are halved) and only the lower
//    half of the second one's outputs is computed.  The radix plans read the second FFT's
//    inputs from the positions where the first leaves its outputs (first radix = last
//    radix), so the multiplication by K happens in registers, without an exchange.
//  * k_lean_mid and the chirp forms of the strided pass: M = N1 N2 in three passes.
//    Columns of x chirp (length N1, four-step twiddles on the way out); then, row by row,
//    FFT_N2, times K, conjugate, FFT_N2, times the same twiddles; then columns again.
//    The spectrum is only multiplied element by element, so it may stay in the order the
//    rows leave it in (K is laid out the same way): no transposition, and the two middle
//    passes of the four-pass form are one.
//
// What bounds them is instruction issue and the barriers between stages (two FFTs of M > 2N
// points for each line of N), so they hold 128 registers a thread at 32 elements (two
// 256-thread CTAs an SM at M = 8192; the general kernel's paths took 255 and one CTA).
// Measured, whole calls, against the general fused and four-pass kernels: 1000 x 3001
// 85.9 -> 42.7 us, 64 x 65521 279.4 -> 80.9 us (under ncu columns of 128 points 28 and 22 us,
// rows of 1024 points 41 us: issue slots 53 to 54% used, 15 to 22 of 64 warps active, the L1
// data path 49 to 55%).
#pragma once
#include "rk_lean.cuh"

namespace rk {

// v (elements i with i % R0 < R0/2 of a line; a = a0 + (tb + K(i)) jB) = x[a] chirp[a]
// for a < N, else 0.  off excludes the position.
template <typename T, class E, bool UNIT>
__device__ __forceinline__ void blue_load(const LeanParams& p, uint32_t off, int tb, int a0, cplx<T>* v) {
    using V = cplx<T>;
    const LeanSide& s = p.ld;
    const V* ch = reinterpret_cast<const V*>(p.chirp);
    const int n = (int)p.blue_n, jb = UNIT ? 1 : (int)p.jB;
    const int at = a0 + tb * jb;
    constexpr int H = E::R0 / 2;
    if (s.shift == 0) {
        if constexpr (UNIT) {
            const V* lp = reinterpret_cast<const V*>(s.base + off) + tb;
#pragma unroll
            for (int i = 0; i < E::RT; ++i)
                if (i % E::R0 < H) v[i] = at + E::ik(i) < n ? lp[E::ik(i)] : cmk<V>(T(0), T(0));
        } else {
            const uint32_t o0 = off + (uint32_t)at * s.step, st = (uint32_t)jb * s.step;
#pragma unroll
            for (int i = 0; i < E::RT; ++i)
                if (i % E::R0 < H)
                    v[i] = at + E::ik(i) * jb < n ? *reinterpret_cast<const V*>(s.base + (o0 + (uint32_t)E::ik(i) * st))
                                                  : cmk<V>(T(0), T(0));
        }
    } else {
#pragma unroll
        for (int i = 0; i < E::RT; ++i)
            if (i % E::R0 < H) {
                const int a = at + E::ik(i) * jb;
                int u = a + s.shift;
                if (u >= n) u -= n;
                v[i] = a < n ? *reinterpret_cast<const V*>(s.base + (off + (uint32_t)u * s.step)) : cmk<V>(T(0), T(0));
            }
    }
    if (s.flags & SF_SCALE) lean_scale<T, E::RT>(s, v);
    if (s.flags & SF_PRE_CONJ) lean_conj<T, E::RT>(v);
#pragma unroll
    for (int i = 0; i < E::RT; ++i)
        if (i % E::R0 < H) {
            const int a = at + E::ik(i) * jb;
            if (a < n) v[i] = cmul(v[i], ch[a]);
        }
}

// Outputs i with i % RL < RL/2: chirp[a] conj(v), the inverse transform's conjugation and
// the scale, stored for a < N.
template <typename T, class E, bool UNIT>
__device__ __forceinline__ void blue_store(const LeanParams& p, uint32_t off, int tb, int a0, bool ok, cplx<T>* v) {
    using V = cplx<T>;
    const LeanSide& s = p.st;
    const V* ch = reinterpret_cast<const V*>(p.chirp);
    const int n = (int)p.blue_n, jb = UNIT ? 1 : (int)p.jB;
    const int at = a0 + tb * jb;
    constexpr int H = E::RL / 2;
#pragma unroll
    for (int i = 0; i < E::RT; ++i)
        if (i % E::RL < H) {
            const int a = at + E::ok(i) * jb;
            if (a < n) v[i] = cmulc(ch[a], v[i]);
        }
    if (s.flags & SF_PRE_CONJ) {
#pragma unroll
        for (int i = 0; i < E::RT; ++i)
            if (i % E::RL < H) v[i].y = -v[i].y;
    }
    if (s.flags & SF_SCALE) {
        const T re = (T)s.scale_re, im = (T)s.scale_im;
#pragma unroll
        for (int i = 0; i < E::RT; ++i)
            if (i % E::RL < H) v[i] = im == T(0) ? cscale(v[i], re) : cmul(v[i], cmk<V>(re, im));
    }
    if (!ok) return;
    if (s.shift == 0) {
        if constexpr (UNIT) {
            V* lp = reinterpret_cast<V*>(s.base + off) + tb;
#pragma unroll
            for (int i = 0; i < E::RT; ++i)
                if (i % E::RL < H && at + E::ok(i) < n) lp[E::ok(i)] = v[i];
        } else {
            const uint32_t o0 = off + (uint32_t)at * s.step, st = (uint32_t)jb * s.step;
#pragma unroll
            for (int i = 0; i < E::RT; ++i)
                if (i % E::RL < H && at + E::ok(i) * jb < n)
                    *reinterpret_cast<V*>(s.base + (o0 + (uint32_t)E::ok(i) * st)) = v[i];
        }
    } else {
#pragma unroll
        for (int i = 0; i < E::RT; ++i)
            if (i % E::RL < H) {
                const int a = at + E::ok(i) * jb;
                int u = a + s.shift;
                if (u >= n) u -= n;
                if (a < n) *reinterpret_cast<V*>(s.base + (off + (uint32_t)u * s.step)) = v[i];
            }
    }
}

// FFT, times K, conjugate, FFT.  kp: the line's kernel spectrum.
template <typename T, class E, bool HALF>
__device__ __forceinline__ void blue_core(const LeanParams& p, const cplx<T>* kp, cplx<T>* v, cplx<T>* sm, int ln, int tb) {
    using V = cplx<T>;
    using C = typename E::C;
    const V* tw = reinterpret_cast<const V*>(p.tw);
    E::template run<HALF>(v, sm, ln, tb, tw);
    kp += tb;
#pragma unroll
    for (int i = 0; i < E::RT; ++i) {
        const V k = kp[E::ok(i)];
        v[i] = cmk<V>(v[i].x * k.x - v[i].y * k.y, -v[i].x * k.y - v[i].y * k.x);
    }
    if constexpr (E::NS > 1) lean_sync<C::WARP>();
    if constexpr (E::R0 != E::RL) {
        V* ex = sm + E::sline(ln) + E::spos(tb);
#pragma unroll
        for (int i = 0; i < E::RT; ++i) ex[E::spos(E::ok(i))] = v[i];
        lean_sync<C::WARP>();
#pragma unroll
        for (int i = 0; i < E::RT; ++i) v[i] = ex[E::spos(E::ik(i))];
        lean_sync<C::WARP>();
    }
    E::run(v, sm, ln, tb, tw);
}

// The real-spectrum step of a line (RFFT): outputs chirp[a] conj(v) to shared memory, then
// bins in pairs k, N - k.
template <typename T, class E>
__device__ __forceinline__ void blue_bins_out(const LeanParams& p, uint32_t off, int ln, int tb, bool ok, cplx<T>* sm, cplx<T>* v) {
    using V = cplx<T>;
    using C = typename E::C;
    const V* ch = reinterpret_cast<const V*>(p.chirp);
    const int n = (int)p.blue_n;
    V* z = sm + ln * C::LS;
    lean_sync<C::WARP>();
#pragma unroll
    for (int i = 0; i < E::RT; ++i)
        if (i % E::RL < E::RL / 2 && tb + E::ok(i) < n) z[tb + E::ok(i)] = cmulc(ch[tb + E::ok(i)], v[i]);
    lean_sync<C::WARP>();
    if (!ok) return;
    const V* wk = reinterpret_cast<const V*>(p.rmix);
    V* out = reinterpret_cast<V*>(p.st.base + off);
#pragma unroll 1
    for (int k = tb; 2 * k <= n; k += E::TPL) {
        V o[2];
        real_pair<T>(z[k], z[k == 0 ? 0 : n - k], __ldg(wk + k), T(0.5), o[0], o[1]);
        if (p.st.flags & SF_PRE_CONJ) lean_conj<T, 2>(o);
        if (p.st.flags & SF_SCALE) lean_scale<T, 2>(p.st, o);
        out[k] = o[0];
        if (k == 0 ? (p.rflags & LR_NYQ) != 0 : 2 * k < n) out[n - k] = o[1];
    }
}

// The inverse step (IRFFT): bins to the half-length spectrum in shared memory, then times
// the chirp into v.
template <typename T, class E>
__device__ __forceinline__ void blue_bins_in(const LeanParams& p, uint32_t off, int ln, int tb, cplx<T>* sm, cplx<T>* v) {
    using V = cplx<T>;
    using C = typename E::C;
    const V* ch = reinterpret_cast<const V*>(p.chirp);
    const V* wk = reinterpret_cast<const V*>(p.rmix);
    const int n = (int)p.blue_n;
    const V* in = reinterpret_cast<const V*>(p.ld.base + off);
    V* z = sm + ln * C::LS;
#pragma unroll 2
    for (int k = tb; 2 * k <= n; k += E::TPL) {
        V y[2] = {in[k], in[n - k]}, a, b;
        if (p.ld.flags & SF_SCALE) lean_scale<T, 2>(p.ld, y);
        if (p.ld.flags & SF_PRE_CONJ) lean_conj<T, 2>(y);
        if (k == 0) {
            // bins 0 and N of a real signal are real
            y[0].y = T(0);
            y[1].y = T(0);
        }
        real_pair<T>(y[0], y[1], __ldg(wk + k), T(0.5), a, b);
        z[k] = a;
        if (k > 0 && 2 * k < n) z[n - k] = b;
    }
    lean_sync<C::WARP>();
#pragma unroll
    for (int i = 0; i < E::RT; ++i)
        if (i % E::R0 < E::R0 / 2) {
            const int a = tb + E::ik(i);
            v[i] = a < n ? cmul(z[a], ch[a]) : cmk<V>(T(0), T(0));
        }
    lean_sync<C::WARP>();
}

template <typename T, int L, int MODE, int REAL>
__global__ void __launch_bounds__((LeanCfg<T, L, MODE, 1>::NT), (LeanCfg<T, L, MODE, 1>::MINB))
    k_lean_blue(const __grid_constant__ LeanParams p) {
    using V = cplx<T>;
    using E = LeanEngine<T, L, MODE, 1>;
    constexpr int TPL = E::TPL, NL = E::NL;
    extern __shared__ __align__(16) unsigned char rk_smem[];
    V* sm = reinterpret_cast<V*>(rk_smem);
    lean_begin();
    const int tid = threadIdx.x;
    const int ln = MODE == MODE_POS ? tid / TPL : tid % NL;
    const int tb = MODE == MODE_POS ? tid % TPL : tid / NL;
    const uint32_t lt = lean_tile(p) * NL + ln, line = min(lt, p.nlines - 1);
    V v[E::RT];
    if constexpr (REAL == 2) blue_bins_in<T, E>(p, lean_offset(p.ld, line), ln, tb, sm, v);
    else blue_load<T, E, MODE == MODE_POS>(p, lean_offset(p.ld, line), tb, 0, v);
    blue_core<T, E, true>(p, reinterpret_cast<const V*>(p.blue_k), v, sm, ln, tb);
    if constexpr (REAL == 1) blue_bins_out<T, E>(p, lean_offset(p.st, line), ln, tb, lt < p.nlines, sm, v);
    else blue_store<T, E, MODE == MODE_POS>(p, lean_offset(p.st, line), tb, 0, lt < p.nlines, v);
}

// Rows of the three-pass form: line (o, c, i) of N2 = L points; K and the twiddles of row c.
template <typename T, int L, int MODE>
__global__ void __launch_bounds__((LeanCfg<T, L, MODE, 1>::NT), (LeanCfg<T, L, MODE, 1>::MINB))
    k_lean_mid(const __grid_constant__ LeanParams p) {
    using V = cplx<T>;
    using E = LeanEngine<T, L, MODE, 1>;
    constexpr int TPL = E::TPL, NL = E::NL;
    extern __shared__ __align__(16) unsigned char rk_smem[];
    V* sm = reinterpret_cast<V*>(rk_smem);
    lean_begin();
    const int tid = threadIdx.x;
    const int ln = MODE == MODE_POS ? tid / TPL : tid % NL;
    const int tb = MODE == MODE_POS ? tid % TPL : tid / NL;
    const uint32_t lt = lean_tile(p) * NL + ln, line = min(lt, p.nlines - 1);
    const uint32_t q = fd_div(p.cI, line), c = q - fd_div(p.cC, q) * p.cC.d;
    V v[E::RT];
    lean_load<T, L, E::RT, MODE == MODE_POS>(p.ld, lean_offset(p.ld, line), tb, [](int i) { return E::ik(i); }, v);
    blue_core<T, E, false>(p, reinterpret_cast<const V*>(p.blue_k) + c * (uint32_t)L, v, sm, ln, tb);
    lean_tw4_block<T, E>(p, c, tb, v);
    lean_store<T, L, E::RT, MODE == MODE_POS, 0>(p.st, lean_offset(p.st, line), tb, lt < p.nlines,
                                                 [](int i) { return E::ok(i); }, v);
}

// Columns of the three-pass form.  OUT false: the first pass (chirp and zero padding on
// the load, twiddles on the store); true: the last one (chirp on the store, a < N only).
template <typename T, int L, bool OUT>
__global__ void __launch_bounds__((LeanCfg<T, L, MODE_LANE, 0>::NT), (LeanCfg<T, L, MODE_LANE, 0>::MINB))
    k_lean_cols(const __grid_constant__ LeanParams p) {
    using V = cplx<T>;
    using E = LeanEngine<T, L, MODE_LANE, 0>;
    constexpr int NL = E::NL;
    extern __shared__ __align__(16) unsigned char rk_smem[];
    V* sm = reinterpret_cast<V*>(rk_smem);
    lean_begin();
    const int ln = threadIdx.x % NL, tb = threadIdx.x / NL;
    const uint32_t lt = lean_tile(p) * NL + ln, line = min(lt, p.nlines - 1);
    const uint32_t q = fd_div(p.cI, line), c = q - fd_div(p.cC, q) * p.cC.d;
    V v[E::RT];
    if constexpr (!OUT) {
        blue_load<T, E, false>(p, lean_offset(p.ld, line), tb, (int)c, v);
        E::template run<true>(v, sm, ln, tb, reinterpret_cast<const V*>(p.tw));
        lean_tw4_block<T, E>(p, c, tb, v);
        lean_store<T, L, E::RT, false, 0>(p.st, lean_offset(p.st, line), tb, lt < p.nlines, [](int i) { return E::ok(i); }, v);
    } else {
        lean_load<T, L, E::RT, false>(p.ld, lean_offset(p.ld, line), tb, [](int i) { return E::ik(i); }, v);
        E::run(v, sm, ln, tb, reinterpret_cast<const V*>(p.tw));
        blue_store<T, E, false>(p, lean_offset(p.st, line), tb, (int)c, lt < p.nlines, v);
    }
}

// VAR 1: whole lines (6 / 7: with the real-spectrum step after / before); 3: rows of the
// three-pass form; 4 / 5: its first / last columns
template <typename T, int L, int MODE, int VAR> struct LeanBlueLauncher {
    using C = LeanCfg<T, L, MODE, (VAR == 4 || VAR == 5 ? 0 : 1)>;
    static constexpr auto kernel() {
        if constexpr (VAR == 1 || VAR >= 6) return &k_lean_blue<T, L, MODE, (VAR >= 6 ? VAR - 5 : 0)>;
        else if constexpr (VAR == 3) return &k_lean_mid<T, L, MODE>;
        else return &k_lean_cols<T, L, VAR == 5>;
    }
    static cudaError_t launch(const LeanParams& p, cudaStream_t st) {
        return lean_launch(kernel(), (p.nlines + C::NL - 1) / C::NL, C::NT, C::SMEM, p, st);
    }
    static cudaError_t prepare() {
        if (C::SMEM <= 48 * 1024) return cudaSuccess;
        return cudaFuncSetAttribute(kernel(), cudaFuncAttributeMaxDynamicSharedMemorySize, (int)C::SMEM);
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
