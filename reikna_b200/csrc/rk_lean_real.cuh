// Lean passes of the real transforms: a line of L = N / 2 points holds the sample pairs
// x[2u] + i x[2u+1] of a real line of N samples (or of a frame of a signal).
//
//  * k_lean_rpost (RFFT, spectrogram): pairs in, times the window, FFT_L, the real-spectrum
//    step, bins or magnitudes out (VAR 5: lane-fastest through shared memory);
//  * k_lean_rpre (IRFFT): bins in, the inverse step, FFT_L, pairs out.
//
// The step needs bin k and its mirror L - k at once.  A thread holds the bins tb + TPL j of
// its line, so the mirror of its bin j sits in thread TPL - tb at RT - 1 - j (thread 0: in
// itself at RT - j): one shuffle moves it, where lines live inside a warp.  The general
// kernel wrote the whole line to shared memory and read it back between two block
// barriers, at 64 registers with spills; what bounds both is instruction issue.
// Measured, whole calls: spectrogram of 2^22 samples (1024 / 256) 41.0 -> 25.5 us, IRFFT of
// 16384 x 513 bins 46.5 -> 27.9 us (a copy of its bytes 20.8 us), RFFT of 16384 x 1024 (pass
// time) 41 -> 31 us, transposed spectrogram (pass time) 48 -> 37 us.
#pragma once
#include "rk_lean.cuh"

namespace rk {

// element held for position index j (bin tb + TPL j) after the FFT / before it
template <class E> constexpr int out_slot(int j) { return j % (E::RT / E::RL) * E::RL + j / (E::RT / E::RL); }
template <class E> constexpr int in_slot(int j) { return j % (E::RT / E::R0) * E::R0 + j / (E::RT / E::R0); }

template <int TPL, typename V> __device__ __forceinline__ V mirror_shfl(V v, int tb) {
    const int src = (TPL - tb) & (TPL - 1);
    V r;
    r.x = __shfl_sync(0xffffffffu, v.x, src, TPL);
    r.y = __shfl_sync(0xffffffffu, v.y, src, TPL);
    return r;
}
template <typename V> __device__ __forceinline__ V pick(bool c, V a, V b) {
    return cmk<V>(c ? a.x : b.x, c ? a.y : b.y);
}

// bin positions of o[]: slot j < RT/2 is bin tb + TPL j, slot RT/2 + j its mirror L - k
// (thread 0: slot RT/2 is bin L/2, and bin L is kept apart)
template <int L, int RT, int TPL> __device__ __forceinline__ int mirror_pos(int tb, int j) {
    return j == 0 && tb == 0 ? L / 2 : L - tb - TPL * j;
}

template <typename T, int L, int VAR>
__global__ void __launch_bounds__((LeanCfg<T, L, MODE_POS, VAR>::NT), (LeanCfg<T, L, MODE_POS, VAR>::MINB))
    k_lean_rpost(const __grid_constant__ LeanParams p) {
    using V = cplx<T>;
    using C = LeanCfg<T, L, MODE_POS, VAR>;
    using E = LeanEngine<T, L, MODE_POS, VAR>;
    constexpr int RT = E::RT, TPL = E::TPL, NL = E::NL, H = RT / 2;
    extern __shared__ __align__(16) unsigned char rk_smem[];
    V* sm = reinterpret_cast<V*>(rk_smem);
    lean_begin();
    const int tid = threadIdx.x, ln = tid / TPL, tb = tid % TPL;
    const uint32_t line0 = blockIdx.x * NL, lt = line0 + ln, line = min(lt, p.nlines - 1);
    V v[RT];
    {
        const T* lp = reinterpret_cast<const T*>(p.ld.base + lean_offset(p.ld, line)) + 2 * tb;
        if (p.rflags & LR_PAIRS) {
#pragma unroll
            for (int i = 0; i < RT; ++i) v[i] = *reinterpret_cast<const V*>(lp + 2 * E::ik(i));
        } else {
#pragma unroll
            for (int i = 0; i < RT; ++i) v[i] = cmk<V>(lp[2 * E::ik(i)], lp[2 * E::ik(i) + 1]);
        }
        if (p.win) {
            const V* w = reinterpret_cast<const V*>(p.win) + tb;
#pragma unroll
            for (int i = 0; i < RT; ++i) {
                const V f = __ldg(w + E::ik(i));
                v[i].x *= f.x;
                v[i].y *= f.y;
            }
        }
    }
    E::run(v, sm, ln, tb, reinterpret_cast<const V*>(p.tw));
    const V* wk = reinterpret_cast<const V*>(p.rmix) + tb;
    V o[RT], nyq;
    if constexpr (!C::WARP) {
        lean_sync<false>();
        V* z = sm + E::sline(ln) + E::spos(tb);
#pragma unroll
        for (int j = 0; j < RT; ++j) z[E::spos(TPL * j)] = v[out_slot<E>(j)];
        lean_sync<false>();
    }
#pragma unroll
    for (int j = 0; j < H; ++j) {
        V q;
        if constexpr (C::WARP) {
            q = mirror_shfl<TPL>(pick(tb == 0, v[out_slot<E>((RT - j) % RT)], v[out_slot<E>(RT - 1 - j)]), tb);
        } else {
            const int m = (L - tb - TPL * j) & (L - 1);
            q = sm[E::sline(ln) + E::spos(m)];
        }
        real_pair<T>(v[out_slot<E>(j)], q, __ldg(wk + TPL * j), T(0.5), o[j], o[H + j]);
    }
    nyq = o[H];
    if (tb == 0) {
        // bin L/2 is its own mirror and w there is -i: X = conj(Z)
        o[H] = cconj(v[out_slot<E>(H)]);
    }
    if (p.st.flags & SF_PRE_CONJ) {
        lean_conj<T, RT>(o);
        nyq.y = -nyq.y;
    }
    if (p.st.flags & SF_SCALE) {
        lean_scale<T, RT>(p.st, o);
        lean_scale<T, 1>(p.st, &nyq);
    }
    const bool ok = lt < p.nlines, last = tb == 0 && (p.rflags & LR_NYQ);
    const int bound = (int)p.bound;
    if constexpr (VAR == 5) {
        // magnitudes, staged line by line and stored lane-fastest
        T* ts = reinterpret_cast<T*>(rk_smem);
        constexpr int LS = C::TLS;
        auto mag = [&](V x) {
            const T r = x.x * x.x + x.y * x.y;
            return (p.rflags & LR_SQRT) ? mag_sqrt<T>(r) : r;
        };
        __syncthreads();
        T* tl = ts + ln * LS;
#pragma unroll
        for (int j = 0; j < H; ++j) {
            tl[tb + TPL * j] = mag(o[j]);
            tl[mirror_pos<L, RT, TPL>(tb, j)] = mag(o[H + j]);
        }
        if (last) tl[L] = mag(nyq);
        __syncthreads();
        const int lane = tid % NL, p0 = tid / NL;
        const uint32_t sl = line0 + lane;
        if (sl >= p.nlines) return;
        char* dst = p.st.base + lean_offset(p.st, sl);
        const uint32_t o0 = (uint32_t)p0 * p.st.step;
        const T* tr = ts + lane * LS + p0;
#pragma unroll
        for (int q = 0; q < RT; ++q)
            if (p0 + TPL * q < bound) *reinterpret_cast<T*>(dst + (o0 + (uint32_t)(TPL * q) * p.st.step)) = tr[TPL * q];
        if (p0 == 0 && (p.rflags & LR_NYQ)) *reinterpret_cast<T*>(dst + (uint32_t)L * p.st.step) = ts[lane * LS + L];
    } else {
        if (!ok) return;
        if (p.rflags & LR_NORM) {
            T* lp = reinterpret_cast<T*>(p.st.base + lean_offset(p.st, line));
            auto put = [&](int at, V x) {
                const T r = x.x * x.x + x.y * x.y;
                if (at < bound) lp[at] = (p.rflags & LR_SQRT) ? mag_sqrt<T>(r) : r;
            };
#pragma unroll
            for (int j = 0; j < H; ++j) put(tb + TPL * j, o[j]);
#pragma unroll
            for (int j = 0; j < H; ++j) put(mirror_pos<L, RT, TPL>(tb, j), o[H + j]);
            if (last) {
                const T r = nyq.x * nyq.x + nyq.y * nyq.y;
                lp[L] = (p.rflags & LR_SQRT) ? mag_sqrt<T>(r) : r;
            }
        } else {
            V* lp = reinterpret_cast<V*>(p.st.base + lean_offset(p.st, line));
            if (bound == L) {
#pragma unroll
                for (int j = 0; j < H; ++j) lp[tb + TPL * j] = o[j];
#pragma unroll
                for (int j = 0; j < H; ++j) lp[mirror_pos<L, RT, TPL>(tb, j)] = o[H + j];
            } else {
#pragma unroll
                for (int j = 0; j < H; ++j)
                    if (tb + TPL * j < bound) lp[tb + TPL * j] = o[j];
#pragma unroll
                for (int j = 0; j < H; ++j)
                    if (mirror_pos<L, RT, TPL>(tb, j) < bound) lp[mirror_pos<L, RT, TPL>(tb, j)] = o[H + j];
            }
            if (last) lp[L] = nyq;
        }
    }
}

template <typename T, int L>
__global__ void __launch_bounds__((LeanCfg<T, L, MODE_POS, 0>::NT), (LeanCfg<T, L, MODE_POS, 0>::MINB))
    k_lean_rpre(const __grid_constant__ LeanParams p) {
    using V = cplx<T>;
    using C = LeanCfg<T, L, MODE_POS, 0>;
    using E = LeanEngine<T, L, MODE_POS, 0>;
    constexpr int RT = E::RT, TPL = E::TPL, NL = E::NL, H = RT / 2;
    extern __shared__ __align__(16) unsigned char rk_smem[];
    V* sm = reinterpret_cast<V*>(rk_smem);
    lean_begin();
    const int tid = threadIdx.x, ln = tid / TPL, tb = tid % TPL;
    const uint32_t lt = blockIdx.x * NL + ln, line = min(lt, p.nlines - 1);
    V y[RT], yh;   // bins tb + TPL j and their mirrors L - k; thread 0: bin L/2 apart
    {
        const V* lp = reinterpret_cast<const V*>(p.ld.base + lean_offset(p.ld, line));
#pragma unroll
        for (int j = 0; j < H; ++j) y[j] = lp[tb + TPL * j];
#pragma unroll
        for (int j = 0; j < H; ++j) y[H + j] = lp[L - tb - TPL * j];
        yh = tb == 0 ? lp[L / 2] : y[0];
    }
    if (p.ld.flags & SF_SCALE) {
        lean_scale<T, RT>(p.ld, y);
        lean_scale<T, 1>(p.ld, &yh);
    }
    if (p.ld.flags & SF_PRE_CONJ) {
        lean_conj<T, RT>(y);
        yh.y = -yh.y;
    }
    if (tb == 0) {
        // bins 0 and L of a real signal are real
        y[0].y = T(0);
        y[H].y = T(0);
    }
    const V* wk = reinterpret_cast<const V*>(p.rmix) + tb;
#pragma unroll
    for (int j = 0; j < H; ++j) real_pair<T>(y[j], y[H + j], __ldg(wk + TPL * j), T(0.5), y[j], y[H + j]);
    // y[j] goes to position tb + TPL j, y[H + j] to its mirror, bin L/2 becomes its conjugate
    yh = cconj(yh);
    V v[RT];
    if constexpr (C::WARP) {
#pragma unroll
        for (int j = 0; j < H; ++j) v[in_slot<E>(j)] = y[j];
#pragma unroll
        for (int j = H; j < RT; ++j)
            v[in_slot<E>(j)] = mirror_shfl<TPL>(pick(tb == 0, j == H ? yh : y[H + (RT - j) % RT], y[H + RT - 1 - j]), tb);
    } else {
        V* z = sm + E::sline(ln);
#pragma unroll
        for (int j = 0; j < H; ++j) {
            z[E::spos(tb) + E::spos(TPL * j)] = y[j];
            if (j > 0 || tb > 0) z[E::spos(L - tb - TPL * j)] = y[H + j];
            else z[E::spos(L / 2)] = yh;
        }
        lean_sync<false>();
#pragma unroll
        for (int j = 0; j < RT; ++j) v[in_slot<E>(j)] = z[E::spos(tb) + E::spos(TPL * j)];
        lean_sync<false>();
    }
    E::run(v, sm, ln, tb, reinterpret_cast<const V*>(p.tw));
    lean_store<T, L, RT, true, 0>(p.st, lean_offset(p.st, line), tb, lt < p.nlines, [](int i) { return E::ok(i); }, v);
}

// VAR 6: bins or magnitudes along the line; 5: magnitudes lane-fastest; 4: the inverse
template <typename T, int L, int VAR> struct LeanRealLauncher {
    using C = LeanCfg<T, L, MODE_POS, (VAR == 5 ? 5 : 0)>;
    static constexpr auto kernel() {
        if constexpr (VAR == 4) return &k_lean_rpre<T, L>;
        else return &k_lean_rpost<T, L, (VAR == 5 ? 5 : 0)>;
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
