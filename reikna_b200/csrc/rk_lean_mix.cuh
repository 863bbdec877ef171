// Lean passes of lengths with small prime factors (up to 13) that are not powers of two:
// the FFT of the length itself, by a Stockham plan of two to four radices of at most 16,
// instead of Bluestein's two transforms of more than twice the length.
//
// One kernel takes every length: the radices come with the plan, and a stage is one of the
// register DFTs below for every butterfly of the tile.  The first stage reads global memory
// and the last writes it; between, the tile stays in shared memory, in place where a thread
// has one butterfly a stage, else from one buffer to another.  With one pad word for each
// R0 positions where the first radix R0 is even, the first stage's stride-R0 writes meet
// different banks, and since R0 divides every later stride a butterfly's addresses are a
// base plus m times a stride.
//
// What bounds it: the latency of a tile's chain of stages and instruction issue (two to four
// stages of about 30 instructions an element), at a quarter to a half of the copy rate.
// 2 Mi complex64 elements (33.5 MB, copied in 5.2 us), against the general Bluestein
// kernels, rows: 96 points 30.8 -> 8.4 us, 360 43.0 -> 13.4, 1000 35.3 -> 14.3, 5460 (13 x 14 x 10 x 3)
// 43.9 (lean Bluestein) -> 21.2; for columns: 100 points 34.9 -> 10.5, 1000 47.1 -> 19.3, 1920
// 90.1 -> 22.9.
#pragma once
#include "rk_lean.cuh"

namespace rk {

// cos(2 pi k / n) and sin(2 pi k / n) by their power series after reduction to an octant
constexpr double mix_pi = 3.14159265358979323846264338327950288;
constexpr double mix_series(double x, bool sine) {
    double term = sine ? x : 1.0, sum = term;
    for (int i = sine ? 1 : 0; i < 24; i += 2) {
        term *= -x * x / ((i + 1.0) * (i + 2.0));
        sum += term;
    }
    return sum;
}
constexpr double mix_cos(int k, int n) {
    k = ((k % n) + n) % n;
    if (2 * k > n) k = n - k;                      // cos is even
    if (4 * k > n) return -mix_cos(n - 2 * k, 2 * n);   // cos(pi - x) = -cos x
    return 8 * k > n ? mix_series(2.0 * mix_pi * (n - 4.0 * k) / (4.0 * n), true) : mix_series(2.0 * mix_pi * k / n, false);
}
constexpr double mix_sin(int k, int n) { return mix_cos(4 * k - n, 4 * n); }   // sin x = cos(x - pi/2)

constexpr int mix_inv(int a, int n) {
    for (int i = 1; i < n; ++i)
        if (a * i % n == 1) return i;
    return 1;
}

// the constants as compile-time values (an indexed table would live in local memory)
template <int K, int N> struct MixW {
    static constexpr double c = mix_cos(K, N), s = mix_sin(K, N);
};

// c += sum_j cos(2 pi j K / R) t_j and d = sum_j sin(2 pi j K / R) s_j, j = 1 .. (R - 1) / 2
template <int R, int K, int J, typename V> __device__ __forceinline__ void mix_row(const V* t, const V* s, V& c, V& d) {
    if constexpr (J <= (R - 1) / 2) {
        using T = decltype(c.x);
        constexpr T cs = (T)MixW<J * K, R>::c, sn = (T)MixW<J * K, R>::s;
        c.x += cs * t[J - 1].x;
        c.y += cs * t[J - 1].y;
        d.x = J == 1 ? sn * s[0].x : d.x + sn * s[J - 1].x;
        d.y = J == 1 ? sn * s[0].y : d.y + sn * s[J - 1].y;
        mix_row<R, K, J + 1>(t, s, c, d);
    }
}
template <int R, int K, typename V> __device__ __forceinline__ void mix_rows(V a0, const V* t, const V* s, V* a) {
    if constexpr (K <= (R - 1) / 2) {
        V c = a0, d;
        mix_row<R, K, 1>(t, s, c, d);
        // X[K] = c - i d, X[R - K] = c + i d
        a[K] = cmk<V>(c.x + d.y, c.y - d.x);
        a[R - K] = cmk<V>(c.x - d.y, c.y + d.x);
        mix_rows<R, K + 1>(a0, t, s, a);
    }
}
template <int N, int K, typename V> __device__ __forceinline__ V mix_mul(V v) {
    if constexpr (K == 0) {
        return v;
    } else {
        using T = decltype(v.x);
        constexpr T c = (T)MixW<K, N>::c, s = (T)MixW<K, N>::s;
        return cmk<V>(v.x * c + v.y * s, v.y * c - v.x * s);
    }
}

// R-point DFT in place, natural order.  Odd primes by the symmetric sums a_j +- a_{R-j};
// products of coprime factors by the Chinese remainder index maps (no twiddles); 9 as 3 x 3.
template <int R, typename V> __device__ __forceinline__ void mix_dft(V* a) {
    using T = decltype(a[0].x);
    if constexpr (R == 2 || R == 4 || R == 8 || R == 16) {
        dft<R>(a);
    } else if constexpr (R == 9) {
        // columns n2, twiddles W_9^(n2 k1), rows
#pragma unroll
        for (int n2 = 0; n2 < 3; ++n2) {
            V c[3] = {a[n2], a[n2 + 3], a[n2 + 6]};
            mix_dft<3>(c);
#pragma unroll
            for (int k = 0; k < 3; ++k) a[n2 + 3 * k] = c[k];
        }
        a[4] = mix_mul<9, 1>(a[4]);
        a[5] = mix_mul<9, 2>(a[5]);
        a[7] = mix_mul<9, 2>(a[7]);
        a[8] = mix_mul<9, 4>(a[8]);
        V b[9];
#pragma unroll
        for (int k1 = 0; k1 < 3; ++k1) {
            mix_dft<3>(a + 3 * k1);
#pragma unroll
            for (int k2 = 0; k2 < 3; ++k2) b[k1 + 3 * k2] = a[3 * k1 + k2];
        }
#pragma unroll
        for (int k = 0; k < 9; ++k) a[k] = b[k];
    } else if constexpr (R == 6 || R == 10 || R == 12 || R == 14 || R == 15) {
        constexpr int A = R == 12 ? 4 : R == 15 ? 3 : 2, B = R / A;
        constexpr int ea = B * mix_inv(B % A, A), eb = A * mix_inv(A % B, B);   // 1 mod A / 0 mod B, and the other
        V b[R];
#pragma unroll
        for (int n2 = 0; n2 < B; ++n2) {
            V c[A];
#pragma unroll
            for (int n1 = 0; n1 < A; ++n1) c[n1] = a[(B * n1 + A * n2) % R];
            mix_dft<A>(c);
#pragma unroll
            for (int k1 = 0; k1 < A; ++k1) b[k1 * B + n2] = c[k1];
        }
#pragma unroll
        for (int k1 = 0; k1 < A; ++k1) {
            mix_dft<B>(b + k1 * B);
#pragma unroll
            for (int k2 = 0; k2 < B; ++k2) a[(ea * k1 + eb * k2) % R] = b[k1 * B + k2];
        }
    } else {
        static_assert(R == 3 || R == 5 || R == 7 || R == 11 || R == 13, "no DFT of this radix");
        constexpr int H = (R - 1) / 2;
        V t[H], s[H], x0 = a[0];
        const V a0 = a[0];
#pragma unroll
        for (int j = 1; j <= H; ++j) {
            t[j - 1] = a[j] + a[R - j];
            s[j - 1] = a[j] - a[R - j];
            x0 = x0 + t[j - 1];
        }
        a[0] = x0;
        mix_rows<R, 1>(a0, t, s, a);
    }
}

template <typename T> struct MixCfg {
    // threads of a CTA at most, and the CTAs an SM the registers are sized for
    static constexpr int NT = sizeof(T) == 4 ? 384 : 256, MINB = 2;
};

// Where a stage reads from and writes to: global memory (first stage, last stage), the
// tile's buffers, or the tile's buffers at both ends of a real transform (first stage from
// lines without pads, last stage to whole lines, before the real-spectrum step).
enum MixEnd { MIX_GLOBAL, MIX_TILE, MIX_LINES };

// One stage of radix R over the tile's butterflies.
template <typename T, int R, int MODE, int SRC, int DST>
__device__ __forceinline__ void mix_stage(const LeanParams& p, const MixPlan& x, const MixStage& g, const cplx<T>* src,
                                          cplx<T>* dst, const uint32_t* off_ld, const uint32_t* off_st, uint32_t valid) {
    using V = cplx<T>;
    constexpr bool FIRST = SRC != MIX_TILE, LAST = DST != MIX_TILE;
    const uint32_t nb = g.nb, total = nb * x.nl, nll = x.nl;
    const V* tw = reinterpret_cast<const V*>(p.tw) + g.tw;
    auto pad = [&](uint32_t at) { return x.pad ? fd_div(x.r0, at) : 0u; };
    // distance between a butterfly's inputs and between its outputs
    const uint32_t rd = FIRST ? nb : MODE == MODE_LANE ? nb * nll : nb + pad(nb);
    const uint32_t wr = DST == MIX_GLOBAL ? g.P : MODE == MODE_LANE ? g.P * nll : FIRST ? 1 : g.P + pad(g.P);
    uint32_t i = threadIdx.x;
    do {
        const bool act = i < total;
        uint32_t ln, b;
        if constexpr (MODE == MODE_LANE) {
            ln = i & (nll - 1);
            b = i >> x.lsh;
        } else {
            ln = fd_div(g.bdiv, i);
            b = i - ln * nb;
        }
        V v[R];
        if (act) {
            if constexpr (SRC == MIX_LINES) {
                const V* q = src + ln * x.n + b;
#pragma unroll
                for (int m = 0; m < R; ++m) v[m] = q[m * nb];
            } else if constexpr (FIRST) {
                if constexpr (MODE == MODE_POS) {
                    const V* lp = reinterpret_cast<const V*>(p.ld.base + off_ld[ln]) + b;
#pragma unroll
                    for (int m = 0; m < R; ++m) v[m] = lp[m * rd];
                } else {
                    const uint32_t o0 = off_ld[ln] + b * p.ld.step, st = rd * p.ld.step;
#pragma unroll
                    for (int m = 0; m < R; ++m) v[m] = *reinterpret_cast<const V*>(p.ld.base + (o0 + m * st));
                }
                if (p.ld.flags & SF_SCALE) lean_scale<T, R>(p.ld, v);
                if (p.ld.flags & SF_PRE_CONJ) lean_conj<T, R>(v);
            } else {
                const V* q = src + (MODE == MODE_LANE ? b * nll + ln : ln * x.pitch + b + pad(b));
#pragma unroll
                for (int m = 0; m < R; ++m) v[m] = q[m * rd];
            }
            mix_dft<R>(v);
        }
        // P = L / R in the last stage: j1 = 0, output m at b + P m
        const uint32_t j1 = FIRST ? b : LAST ? 0 : fd_div(g.pdiv, b), l = FIRST ? 0 : b - j1 * g.P;
        if constexpr (DST != MIX_GLOBAL) {
            if (!LAST && act) {
#pragma unroll
                for (int m = 1; m < R; ++m) v[m] = cmul(v[m], __ldg(tw + ((m - 1) * g.J + j1)));
            }
            // in place: every butterfly of the stage is in registers before one is written
            if (SRC != MIX_GLOBAL && x.inplace) __syncthreads();
            if (act) {
                const uint32_t at = LAST ? b : l + g.P * R * j1;
                V* q = dst + (MODE == MODE_LANE ? at * nll + ln : ln * x.pitch + at + pad(at));
#pragma unroll
                for (int m = 0; m < R; ++m) q[m * wr] = v[m];
            }
        } else if (act && ln < valid) {
            if (p.st.flags & SF_PRE_CONJ) lean_conj<T, R>(v);
            if (p.st.flags & SF_SCALE) lean_scale<T, R>(p.st, v);
            if (p.st.shift == 0) {
                if constexpr (MODE == MODE_POS) {
                    V* lp = reinterpret_cast<V*>(p.st.base + off_st[ln]) + b;
#pragma unroll
                    for (int m = 0; m < R; ++m) lp[m * wr] = v[m];
                } else {
                    const uint32_t o0 = off_st[ln] + b * p.st.step, st = wr * p.st.step;
#pragma unroll
                    for (int m = 0; m < R; ++m) *reinterpret_cast<V*>(p.st.base + (o0 + m * st)) = v[m];
                }
            } else {
#pragma unroll
                for (int m = 0; m < R; ++m) {
                    uint32_t u = b + m * wr + (uint32_t)p.st.shift;
                    if (u >= x.n) u -= x.n;
                    *reinterpret_cast<V*>(p.st.base + (off_st[ln] + u * p.st.step)) = v[m];
                }
            }
        }
        i += blockDim.x;
    } while (i < total);
}

template <typename T, int MODE, int SRC, int DST>
__device__ __forceinline__ void mix_radix(const LeanParams& p, const MixPlan& x, int s, const cplx<T>* src, cplx<T>* dst,
                                          const uint32_t* off_ld, const uint32_t* off_st, uint32_t valid) {
    const MixStage& g = x.stage[s];
#define RK_MIX(R) \
    case R: mix_stage<T, R, MODE, SRC, DST>(p, x, g, src, dst, off_ld, off_st, valid); break;
    switch (g.R) {
        RK_MIX(2) RK_MIX(3) RK_MIX(4) RK_MIX(5) RK_MIX(6) RK_MIX(7) RK_MIX(8) RK_MIX(9)
        RK_MIX(10) RK_MIX(11) RK_MIX(12) RK_MIX(13) RK_MIX(14) RK_MIX(15) RK_MIX(16)
    }
#undef RK_MIX
}

// A bin pair k, n - k (k <= n / 2) of a line of the tile
template <typename V> struct MixPair {
    const V* src;
    V* dst;
    uint32_t k;
    V y[2];
};

// The bin pairs of the tile's lines, one after another over the CTA's threads, U of a thread
// loaded before the first is used; line(ln) gives a line's pointers.  MANY: tiles of several lines.
// Line by line, 26 of 384 threads had work at 50 samples: 41943 lines of them, float32, RFFT
// 23.6 -> 6.6 us and IRFFT 26.5 -> 6.6, 116508 lines of 18 samples 52.3 -> 7.1 and 63.5 -> 7.0.
template <bool MANY, int U, typename V, class Line, class Load, class Use>
__device__ __forceinline__ void mix_pairs(const LeanParams& p, uint32_t lines, Line line, Load load, Use use) {
    const uint32_t pairs = p.mix_pairs.d, total = MANY ? lines * pairs : pairs;
    MixPair<V> q[U];
    if constexpr (!MANY) {
#pragma unroll
        for (int u = 0; u < U; ++u) line(q[u], 0u);
    }
    for (uint32_t i = threadIdx.x; i < total; i += U * blockDim.x) {
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const uint32_t at = i + u * blockDim.x;
            if (at < total) {
                q[u].k = at;
                if constexpr (MANY) {
                    const uint32_t ln = fd_div(p.mix_pairs, at);
                    line(q[u], ln);
                    q[u].k = at - ln * pairs;
                }
                load(q[u]);
            }
        }
#pragma unroll
        for (int u = 0; u < U; ++u)
            if (i + u * blockDim.x < total) use(q[u]);
    }
}

// The real-spectrum step of the tile's lines: z (pitch and pads of the tile) to bins
// X[0 .. n) and, where stored, X[n].  w_k = exp(-i pi k / n) in rmix.
template <typename T, bool MANY>
__device__ __forceinline__ void mix_bins_out(const LeanParams& p, const MixPlan& x, const cplx<T>* z, const uint32_t* off_st,
                                             uint32_t valid) {
    using V = cplx<T>;
    const V* wk = reinterpret_cast<const V*>(p.rmix);
    const uint32_t n = x.n;
    auto at = [&](uint32_t k) { return k + (x.pad ? fd_div(x.r0, k) : 0u); };
    mix_pairs<MANY, 1, V>(
        p, valid,
        [&](MixPair<V>& q, uint32_t ln) {
            q.src = z + ln * x.pitch;
            q.dst = reinterpret_cast<V*>(p.st.base + off_st[ln]);
        },
        [&](MixPair<V>& q) {
            q.y[0] = q.src[at(q.k)];
            q.y[1] = q.src[at(q.k == 0 ? 0 : n - q.k)];
        },
        [&](MixPair<V>& q) {
            V o[2];
            real_pair<T>(q.y[0], q.y[1], __ldg(wk + q.k), T(0.5), o[0], o[1]);
            if (p.st.flags & SF_PRE_CONJ) lean_conj<T, 2>(o);
            if (p.st.flags & SF_SCALE) lean_scale<T, 2>(p.st, o);
            q.dst[q.k] = o[0];
            if (q.k == 0 ? (p.rflags & LR_NYQ) != 0 : 2 * q.k < n) q.dst[n - q.k] = o[1];
        });
}

// The inverse step: bins of the tile's lines to the half-length spectrum, lines of n points.
template <typename T, bool MANY>
__device__ __forceinline__ void mix_bins_in(const LeanParams& p, const MixPlan& x, cplx<T>* z, const uint32_t* off_ld) {
    using V = cplx<T>;
    const V* wk = reinterpret_cast<const V*>(p.rmix);
    const uint32_t n = x.n;
    mix_pairs<MANY, 2, V>(
        p, x.nl,
        [&](MixPair<V>& q, uint32_t ln) {
            q.src = reinterpret_cast<const V*>(p.ld.base + off_ld[ln]);
            q.dst = z + ln * n;
        },
        [&](MixPair<V>& q) {
            q.y[0] = q.src[q.k];
            q.y[1] = q.src[n - q.k];
        },
        [&](MixPair<V>& q) {
            V a, b;
            if (p.ld.flags & SF_SCALE) lean_scale<T, 2>(p.ld, q.y);
            if (p.ld.flags & SF_PRE_CONJ) lean_conj<T, 2>(q.y);
            if (q.k == 0) {
                // bins 0 and n of a real signal are real
                q.y[0].y = T(0);
                q.y[1].y = T(0);
            }
            real_pair<T>(q.y[0], q.y[1], __ldg(wk + q.k), T(0.5), a, b);
            q.dst[q.k] = a;
            if (q.k > 0 && 2 * q.k < n) q.dst[n - q.k] = b;
        });
}

// REAL 1: the real-spectrum step after the FFT (RFFT: sample pairs in, bins out); 2: the
// inverse step before it (IRFFT).  The mirror of bin k is bin n - k of the same line, both
// in shared memory.
template <typename T, int MODE, int REAL, bool MANY>
__global__ void __launch_bounds__(MixCfg<T>::NT, MixCfg<T>::MINB) k_lean_mix(const __grid_constant__ LeanParams p) {
    using V = cplx<T>;
    extern __shared__ __align__(16) unsigned char rk_smem[];
    __shared__ MixPlan x;
    // (the plan is constant: read before the wait for the kernel before)
    for (uint32_t i = threadIdx.x; i < sizeof(MixPlan) / 4; i += blockDim.x)
        reinterpret_cast<uint32_t*>(&x)[i] = reinterpret_cast<const uint32_t*>(p.mix)[i];
    lean_begin();
    __syncthreads();
    V* buf0 = reinterpret_cast<V*>(rk_smem);
    V* buf1 = x.bufs == 1 ? buf0 : buf0 + x.buf;
    uint32_t* off_ld = reinterpret_cast<uint32_t*>(buf1 + x.buf);
    uint32_t* off_st = off_ld + x.nl;
    const uint32_t line0 = lean_tile(p) * x.nl;
    for (uint32_t i = threadIdx.x; i < x.nl; i += blockDim.x) {
        const uint32_t line = min(line0 + i, p.nlines - 1);
        off_ld[i] = lean_offset(p.ld, line);
        off_st[i] = lean_offset(p.st, line);
    }
    __syncthreads();
    const uint32_t valid = min(x.nl, p.nlines - line0);
    if constexpr (REAL == 2) {
        mix_bins_in<T, MANY>(p, x, buf0, off_ld);
        __syncthreads();
        mix_radix<T, MODE, MIX_LINES, MIX_TILE>(p, x, 0, buf0, buf1, off_ld, off_st, valid);
        V* t = buf0;
        buf0 = buf1;
        buf1 = t;
    } else {
        mix_radix<T, MODE, MIX_GLOBAL, MIX_TILE>(p, x, 0, nullptr, buf0, off_ld, off_st, valid);
    }
    // (not a loop: hoisting what its bodies share out of it spilled 900 bytes a thread)
    V *last = buf0, *other = buf1;
    if (x.ns > 2) {
        __syncthreads();
        mix_radix<T, MODE, MIX_TILE, MIX_TILE>(p, x, 1, buf0, buf1, off_ld, off_st, valid);
        last = buf1;
        other = buf0;
    }
    if (x.ns > 3) {
        __syncthreads();
        mix_radix<T, MODE, MIX_TILE, MIX_TILE>(p, x, 2, buf1, buf0, off_ld, off_st, valid);
        last = buf0;
        other = buf1;
    }
    __syncthreads();
    if constexpr (REAL == 1) {
        mix_radix<T, MODE, MIX_TILE, MIX_LINES>(p, x, x.ns - 1, last, other, off_ld, off_st, valid);
        __syncthreads();
        mix_bins_out<T, MANY>(p, x, other, off_st, valid);
    } else {
        mix_radix<T, MODE, MIX_TILE, MIX_GLOBAL>(p, x, x.ns - 1, last, nullptr, off_ld, off_st, valid);
    }
}

template <typename T, int MODE, int REAL> struct LeanMixLauncher {
    static cudaError_t launch(const LeanParams& p, cudaStream_t st) {
        return lean_launch(REAL && p.mix_nl > 1 ? k_lean_mix<T, MODE, REAL, (REAL > 0)> : k_lean_mix<T, MODE, REAL, false>,
                           (p.nlines + p.mix_nl - 1) / p.mix_nl, p.mix_nt, p.mix_smem, p, st);
    }
    static cudaError_t prepare() {
        const cudaError_t e =
            cudaFuncSetAttribute(k_lean_mix<T, MODE, REAL, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, MIX_SMEM);
        if (e != cudaSuccess || !REAL) return e;
        return cudaFuncSetAttribute(k_lean_mix<T, MODE, REAL, (REAL > 0)>, cudaFuncAttributeMaxDynamicSharedMemorySize, MIX_SMEM);
    }
};

}  // namespace rk
