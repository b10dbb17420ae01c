// Transforms of any line length with prime factors up to 61 (the axes the
// power-of-two register passes do not take): the five passes of the spectral
// Stokes solve
//
//   x r2c  ->  y fwd  ->  [z fwd, projector, z inv]  ->  y inv  ->  x c2r
//
// Reference: src/stokes_solve.jl:21-42 (unnormalised FFTW r2c / c2r; the
// 1/M normalisation folded into the projector) and :200-240 (the projector
// f <- (inv_M/mu)(1/k^2)(f - k (k.f)/k^2), k = 0 -> 0). The c2r follows the
// FFTW / pocketfft convention for the halved x axis: complex inverse DFTs over
// y and z first, then the 1-D c2r along x, which ignores the imaginary parts
// of the x DC and Nyquist bins.
//
// Spectrum layout: spec[c][z][y][kx], kx fastest, row pitch hxp >= Mx/2+1
// complex values (rows start on 128-byte boundaries).
//
// Stockham autosort stages, each butterfly in registers with compile-time
// twiddles inside it, so that a line of a few hundred points is two stages with
// one shared-memory exchange between them (the host picks the radices,
// mix_plan). A block takes B neighbouring lines; element i of line b sits at
// i * pitch + b, so that a warp's accesses are B-wide runs whatever the
// stage's stride. The y and z passes read their first stage from global memory
// and write their last one back to it; the z pass keeps the three components of
// the modes its last forward stage produced in registers, applies the projector
// there and goes on with the first inverse stage of the same radix, which reads
// exactly those modes. A stage between shared-memory buffers writes to a second
// one; the projector stage works in place when every thread has one butterfly
// at most (all reads, a barrier, all writes). Inverse transforms run the forward code
// and write element i to place (n - i) mod n.
//
// What bounds it: the issue of the butterflies' and address instructions at the
// few warps their registers leave (ncu at 240 x 200 x 160, Float32: 40-48% of
// issue slots, shared-memory conflicts negligible, DRAM at 0.8-1.6 TB/s).
// Measured there, against runtime-radix stages of radix 2, 4, 8 and odd primes
// with every stage through shared memory: y 312 -> 58 us, z and projector
// 818 -> 84 us, x r2c 155 -> 79 us, x c2r 140 -> 86 us (93 MB spectrum; the x
// passes at 104 and 113 us with their rows loaded through registers, which left
// too few loads in flight).
#pragma once

#include "common.cuh"
#include "fft.cuh"

namespace ffcm {

constexpr int MIX_MAX_STAGES = 14;
// Whether a radix has a register butterfly: all up to 16 and, in Float32 (whose
// values take half the registers), the composites that make most lines of up
// to 400 points two stages.
// LONG: lines so long that their twiddle table does not fit in shared memory
// beside the values and is read from global memory; few radices, since such
// lines are rare and every radix is code in each kernel.
template <typename T, bool LONG>
__host__ __device__ constexpr bool mix_has_radix(int R) {
    if (LONG) return R == 2 || R == 3 || R == 4 || R == 5 || R == 7 || R == 8;
    return (R >= 2 && R <= 16) || (sizeof(T) == 4 && (R == 18 || R == 20 || R == 25));
}
constexpr int MIX_MAX_PRIME = 61;    // largest prime factor of a line length

#define FFCM_MIX_RADICES                                                                                        \
    FFCM_MIX(2) FFCM_MIX(3) FFCM_MIX(4) FFCM_MIX(5) FFCM_MIX(6) FFCM_MIX(7) FFCM_MIX(8) FFCM_MIX(9) FFCM_MIX(10) \
    FFCM_MIX(11) FFCM_MIX(12) FFCM_MIX(13) FFCM_MIX(14) FFCM_MIX(15) FFCM_MIX(16) FFCM_MIX(18) FFCM_MIX(20)      \
    FFCM_MIX(25)

struct MixPlan {
    int n;                        // line length
    int nst;
    int tw_stride;                // W_n^e = table[e * tw_stride]
    int radix[MIX_MAX_STAGES];
    int m[MIX_MAX_STAGES];            // n / radix: butterflies of a line
    int step[MIX_MAX_STAGES];         // twiddle W_(Ns radix)^1 = table[step] (span Ns before the stage)
    unsigned magic[MIX_MAX_STAGES];   // ceil(2^32 / Ns)
};

// cos and sin of 2 pi k / P by their Taylor series on [0, pi/4], evaluated by
// the compiler.
__host__ __device__ constexpr double mix_series(double x, bool sine) {
    double term = sine ? x : 1.0, sum = term;
    for (int i = sine ? 2 : 1; i < 30; i += 2) {
        term *= -x * x / (i * (i + 1.0));
        sum += term;
    }
    return sum;
}
__host__ __device__ constexpr double mix_cos(int k, int P) {
    k %= P;
    if (2 * k > P) k = P - k;
    if (4 * k > P) return -mix_cos(P - 2 * k, 2 * P);
    const double tau = 6.283185307179586476925286766559;
    if (8 * k > P) return mix_series(tau * (P - 4 * k) / (4.0 * P), true);
    return mix_series(tau * k / P, false);
}
__host__ __device__ constexpr double mix_sin(int k, int P) { return mix_cos(4 * k + 3 * P, 4 * P); }

template <int P>
struct MixTable {
    double c[P], s[P];
};
template <int P>
__host__ __device__ constexpr MixTable<P> mix_table() {
    MixTable<P> t{};
    for (int k = 0; k < P; ++k) {
        t.c[k] = mix_cos(k, P);
        t.s[k] = mix_sin(k, P);
    }
    return t;
}

// a W_R^e, e < R a constant after unrolling.
template <typename T, int R>
__device__ __forceinline__ cplx<T> mul_root(cplx<T> a, int e) {
    constexpr MixTable<R> t = mix_table<R>();
    if (e == 0) return a;
    if (4 * e == R) return mul_mi(a);
    if (2 * e == R) return cplx<T>{-a.x, -a.y};
    if (4 * e == 3 * R) return mul_pi(a);
    return cmul(a, cplx<T>{T(t.c[e]), T(-t.s[e])});
}

// The split of a composite radix: R = first * second.
__host__ __device__ constexpr int mix_split(int R) {
    if (R % 4 == 0 && R > 4) return 4;
    for (int q = 2; q * q <= R; ++q)
        if (R % q == 0) return q;
    return R;
}

// Forward DFT of R values in registers, natural order in and out.
template <typename T, int R>
struct MixDft {
    __device__ __forceinline__ static void run(cplx<T> (&v)[R]) {
        if constexpr (R == 2 || R == 4 || R == 8) {
            SmallDft<T, R>::run(v, false);
        } else if constexpr (mix_split(R) == R) {
            // odd prime: pairs (k, R - k) share their cosine and sine products
            constexpr MixTable<R> t = mix_table<R>();
            constexpr int H = (R - 1) / 2;
            cplx<T> s[H], d[H];
            cplx<T> sum = v[0];
#pragma unroll
            for (int k = 1; k <= H; ++k) {
                s[k - 1] = cadd(v[k], v[R - k]);
                d[k - 1] = csub(v[k], v[R - k]);
                sum = cadd(sum, s[k - 1]);
            }
            const cplx<T> v0 = v[0];
            v[0] = sum;
#pragma unroll
            for (int q = 1; q <= H; ++q) {
                cplx<T> a = v0, b{T(0), T(0)};
#pragma unroll
                for (int k = 1; k <= H; ++k) {
                    const T c = T(t.c[(k * q) % R]), n = T(t.s[(k * q) % R]);
                    a.x += c * s[k - 1].x;
                    a.y += c * s[k - 1].y;
                    b.x += n * d[k - 1].x;
                    b.y += n * d[k - 1].y;
                }
                v[q] = cplx<T>{a.x + b.y, a.y - b.x};
                v[R - q] = cplx<T>{a.x - b.y, a.y + b.x};
            }
        } else {
            constexpr int R1 = mix_split(R), R2 = R / R1;
            cplx<T> w[R1][R2];
#pragma unroll
            for (int a = 0; a < R1; ++a) {
#pragma unroll
                for (int b = 0; b < R2; ++b) w[a][b] = v[a + R1 * b];
                MixDft<T, R2>::run(w[a]);
#pragma unroll
                for (int b = 1; b < R2; ++b) w[a][b] = mul_root<T, R>(w[a][b], a * b);
            }
#pragma unroll
            for (int b = 0; b < R2; ++b) {
                cplx<T> u[R1];
#pragma unroll
                for (int a = 0; a < R1; ++a) u[a] = w[a][b];
                MixDft<T, R1>::run(u);
#pragma unroll
                for (int a = 0; a < R1; ++a) v[b + R2 * a] = u[a];
            }
        }
    }
};

// Where a stage reads or writes: element i of line b of component c at
// p[c * cs + i * es + b].
template <typename T>
struct MixSpan {
    cplx<T>* p;
    int64_t es, cs;
};
// The same in shared memory (32-bit strides).
template <typename T>
struct MixBuf {
    cplx<T>* p;
    int es, cs;
};

enum { MIX_FIRST, MIX_MID, MIX_LAST };   // Ns = 1 | between buffers | Ns = n / radix

// One stage over NC components of the block's lines: butterfly t is (component
// c, j < m, line b). inv (MIX_LAST): element i goes to (n - i) mod n. src and
// dst differ, or every butterfly's reads are over (MIX_LAST to the array
// MIX_FIRST read). No barrier.
template <typename T, int R, int NC, int KIND, typename S, typename D>
__device__ __forceinline__ void mix_stage(const MixPlan& p, int s, int Ns, int lb, const cplx<T>* tw, S src, D dst,
                                          bool inv) {
    const int m = p.m[s], per = m << lb, total = NC * per, mask = (1 << lb) - 1;
    for (int t = threadIdx.x; t < total; t += blockDim.x) {
        int u = t, c = 0, q = 0;
        if (NC == 3) {
            if (u >= per) { u -= per; c = 1; }
            if (u >= per) { u -= per; c = 2; }
        }
        int k = u >> lb;
        cplx<T> v[R];
        {
            const cplx<T>* a = src.p + c * src.cs + k * src.es + (u & mask);
            const auto as = m * src.es;
#pragma unroll
            for (int r = 0; r < R; ++r) {
                v[r] = *a;
                a += as;
            }
        }
        if (KIND == MIX_MID && Ns == 1) {
            q = k;
            k = 0;
        } else if (KIND != MIX_FIRST) {
            if (KIND == MIX_MID) {
                q = (int)__umulhi((unsigned)k, p.magic[s]);
                k -= q * Ns;
            }
            const int e = k * p.step[s];
            const cplx<T>* w = tw;
#pragma unroll
            for (int r = 1; r < R; ++r) {
                w += e;
                v[r] = cmul(v[r], *w);
            }
        }
        MixDft<T, R>::run(v);
        cplx<T>* a = dst.p + c * dst.cs + (u & mask);
        if (KIND == MIX_LAST) {
            const auto as = inv ? -(m * dst.es) : m * dst.es;
            a[inv && k > 0 ? (p.n - k) * dst.es : k * dst.es] = v[0];
            a += (inv ? p.n - k : k) * dst.es;
#pragma unroll
            for (int r = 1; r < R; ++r) {
                a += as;
                *a = v[r];
            }
        } else {
            const auto as = KIND == MIX_FIRST ? dst.es : Ns * dst.es;
            a += (KIND == MIX_FIRST ? k * R : q * Ns * R + k) * dst.es;
#pragma unroll
            for (int r = 0; r < R; ++r) {
                *a = v[r];
                a += as;
            }
        }
    }
}

// A stage of a prime radix above the register butterflies (up to 61): O(R^2),
// every output sums over the inputs again. Outputs u > 0 of a butterfly without
// twiddles sum the differences from its first value (the roots add up to zero):
// a line's mean then drops out exactly, instead of leaving the rounding of R
// table entries times the mean in the lowest modes, which the projector weighs
// most (60 x 190 x 24, noise of deviation 1 about 0.3, Float64: 80 rounding
// units of the velocities without, 4 with it).
template <typename T, int NC, int KIND, typename S, typename D>
__device__ __forceinline__ void mix_stage_prime(const MixPlan& p, int R, int s, int Ns, int lb, const cplx<T>* tw,
                                                S src, D dst, bool inv) {
    const int m = p.m[s], per = m << lb, total = NC * per * R, mask = (1 << lb) - 1;
    const int root = m * p.tw_stride, size = p.n * p.tw_stride;
    for (int t = threadIdx.x; t < total; t += blockDim.x) {
        const int u = t / (NC * per);   // output of the butterfly
        int w = t - u * NC * per, c = 0;
        if (NC == 3) {
            if (w >= per) { w -= per; c = 1; }
            if (w >= per) { w -= per; c = 2; }
        }
        const int b = w & mask, j = w >> lb;
        const int q = Ns > 1 ? (int)__umulhi((unsigned)j, p.magic[s]) : j, k = j - q * Ns;
        const cplx<T>* a = src.p + c * src.cs + j * src.es + b;
        const auto as = m * src.es;
        const int de = (int)(((int64_t)u * root + (int64_t)k * p.step[s]) % size);
        const cplx<T> base = k == 0 && u > 0 ? *a : cplx<T>{T(0), T(0)};
        cplx<T> acc{T(0), T(0)};
        int e = 0;
        for (int r = 0; r < R; ++r) {
            acc = cadd(acc, cmul(csub(*a, base), tw[e]));
            a += as;
            e += de;
            if (e >= size) e -= size;
        }
        int o = q * Ns * R + k + u * Ns;
        if (inv && o > 0) o = p.n - o;
        dst.p[c * dst.cs + o * dst.es + b] = acc;
    }
}

template <typename T, bool LONG, int NC, int KIND, typename S, typename D>
__device__ __forceinline__ void mix_run_stage(const MixPlan& p, int s, int Ns, int lb, const cplx<T>* tw, S src, D dst,
                                              bool inv = false) {
    switch (p.radix[s]) {
#define FFCM_MIX(RR) case RR: if constexpr (mix_has_radix<T, LONG>(RR)) \
        { mix_stage<T, RR, NC, KIND>(p, s, Ns, lb, tw, src, dst, inv); break; } [[fallthrough]];
        FFCM_MIX_RADICES
#undef FFCM_MIX
        default: mix_stage_prime<T, NC, KIND>(p, p.radix[s], s, Ns, lb, tw, src, dst, inv); break;
    }
}

// The twiddle table W_n^e of the axis (`count` values): from shared memory at
// `sm`, where the block starts copying it, or from global memory (LONG).
template <typename T, bool LONG>
__device__ __forceinline__ const cplx<T>* mix_twiddles(cplx<T>* sm, const cplx<T>* __restrict__ table, int count) {
    if constexpr (LONG) {
        return table;
    } else {
        for (int i = threadIdx.x; i < count; i += blockDim.x) sm[i] = table[i];
        return sm;
    }
}

// Before a first stage that reads global memory: the prime stage, alone among
// them, takes twiddles in its first stage too, so it waits for the copy of the
// table (the others wait at the barrier after the stage).
template <typename T, bool LONG>
__device__ __forceinline__ void mix_first_wait(const MixPlan& p) {
    if (!LONG && !mix_has_radix<T, LONG>(p.radix[0])) __syncthreads();
}

// ---- y c2c on (kx tile) x My columns of one (c, z) plane ------------------
template <typename T, bool LONG>
__global__ void __launch_bounds__(sizeof(T) == 4 ? 512 : 256)
    k_fftm_y(cplx<T>* __restrict__ spec, int hxp, const __grid_constant__ MixPlan p, const cplx<T>* __restrict__ table,
             int lb, int inverse) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    cplx<T>* sm = reinterpret_cast<cplx<T>*>(smem_raw);
    const int n = p.n;
    MixBuf<T> cur{LONG ? sm : sm + n, 1 << lb, 0}, other{cur.p + (n << lb), 1 << lb, 0};
    const cplx<T>* tw = mix_twiddles<T, LONG>(sm, table, n);
    // whole tiles: the row pitch is a multiple of the tile width, the padding
    // columns hold whatever they held, transformed
    const MixSpan<T> g{spec + ((int64_t)blockIdx.z * gridDim.y + blockIdx.y) * n * hxp + (blockIdx.x << lb), hxp, 0};
    mix_first_wait<T, LONG>(p);
    mix_run_stage<T, LONG, 1, MIX_FIRST>(p, 0, 1, lb, tw, g, cur);
    __syncthreads();
    int Ns = p.radix[0];
    for (int s = 1; s + 1 < p.nst; ++s) {
        mix_run_stage<T, LONG, 1, MIX_MID>(p, s, Ns, lb, tw, cur, other);
        __syncthreads();
        Ns *= p.radix[s];
        const MixBuf<T> t = cur;
        cur = other;
        other = t;
    }
    if (p.nst > 1) {
        mix_run_stage<T, LONG, 1, MIX_LAST>(p, p.nst - 1, Ns, lb, tw, cur, g, inverse != 0);
    } else {
        for (int t = threadIdx.x; t < n << lb; t += blockDim.x) {
            const int i = t >> lb;
            g.p[(inverse && i > 0 ? n - i : i) * g.es + (t & ((1 << lb) - 1))] = cur.p[t];
        }
    }
}

// The Stokes projector on one mode (src/stokes_solve.jl:200-240).
template <typename T>
__device__ __forceinline__ void project_mode(T k1, T k2, T k3, T inv_mu_M, cplx<T>& f0, cplx<T>& f1, cplx<T>& f2) {
    const T ksq = k1 * k1 + k2 * k2 + k3 * k3;
    if (ksq == T(0)) {
        f0 = f1 = f2 = cplx<T>{T(0), T(0)};
        return;
    }
    const T inv_k2 = T(1) / ksq;
    const T sc = inv_mu_M * inv_k2;
    const T dre = (k1 * f0.x + k2 * f1.x + k3 * f2.x) * inv_k2;
    const T dim = (k1 * f0.y + k2 * f1.y + k3 * f2.y) * inv_k2;
    f0 = cplx<T>{sc * (f0.x - k1 * dre), sc * (f0.y - k1 * dim)};
    f1 = cplx<T>{sc * (f1.x - k2 * dre), sc * (f1.y - k2 * dim)};
    f2 = cplx<T>{sc * (f2.x - k3 * dre), sc * (f2.y - k3 * dim)};
}

// Largest last radix whose three components stay in registers through the
// projector (the host plans the z axis for it where the length allows).
template <typename T>
__host__ __device__ constexpr int mix_fuse_radix() { return sizeof(T) == 4 ? 10 : 6; }

// Last forward stage, projector and first inverse stage of the z pass, on the
// modes z = j + r m of three components.
template <typename T, int R>
__device__ __forceinline__ void mix_middle(const MixPlan& p, int s, int lb, int kx0, int nkx, const cplx<T>* tw,
                                           MixBuf<T> src, MixBuf<T> dst, bool in_place, const T* __restrict__ kxv,
                                           T k2, const T* __restrict__ kzv, T inv_mu_M) {
    const int m = p.m[s], total = m << lb, mask = (1 << lb) - 1;
    for (int t0 = 0; t0 < total; t0 += blockDim.x) {
        // threads past the end repeat the last butterfly and store nothing, so
        // that the values are defined on every path across the barrier
        const bool act = t0 + (int)threadIdx.x < total;
        const int t = min(t0 + (int)threadIdx.x, total - 1), b = t & mask, j = t >> lb;
        cplx<T> v[3][R];
        const cplx<T>*a = src.p + t, *w = tw;
        const int as = m << lb, e = j * p.step[s];
#pragma unroll
        for (int r = 0; r < R; ++r) {
#pragma unroll
            for (int c = 0; c < 3; ++c) v[c][r] = a[c * src.cs];
            if (r > 0) {
#pragma unroll
                for (int c = 0; c < 3; ++c) v[c][r] = cmul(v[c][r], *w);
            }
            a += as;
            w += e;
        }
#pragma unroll
        for (int c = 0; c < 3; ++c) MixDft<T, R>::run(v[c]);
        const T k1 = kx0 + b < nkx ? kxv[kx0 + b] : T(0);
#pragma unroll
        for (int r = 0; r < R; ++r) project_mode(k1, k2, kzv[j + r * m], inv_mu_M, v[0][r], v[1][r], v[2][r]);
#pragma unroll
        for (int c = 0; c < 3; ++c) MixDft<T, R>::run(v[c]);
        if (in_place) __syncthreads();
        if (act) {
            cplx<T>* o = dst.p + ((j * R) << lb) + b;
#pragma unroll
            for (int r = 0; r < R; ++r) {
#pragma unroll
                for (int c = 0; c < 3; ++c) o[c * dst.cs] = v[c][r];
                o += 1 << lb;
            }
        }
    }
}

// ---- z forward, Stokes projector, z inverse (all 3 components) -------------
// p: the forward stages; pi: the same radices in reverse order. fuse: the last
// forward radix is at most mix_fuse_radix and there are two stages or more.
template <typename T, bool LONG>
__global__ void __launch_bounds__(sizeof(T) == 4 ? 512 : 256, sizeof(T) == 4 ? 1 : 2)
    k_fftm_z_stokes(cplx<T>* __restrict__ spec, int nkx, int My, int hxp, const __grid_constant__ MixPlan p,
                    const __grid_constant__ MixPlan pi, int fuse, const cplx<T>* __restrict__ table, int lb,
                    const T* __restrict__ kxv, const T* __restrict__ kyv, const T* __restrict__ kzv, T inv_mu_M) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const int n = p.n, cs = n << lb;
    cplx<T>* sm = reinterpret_cast<cplx<T>*>(smem_raw);
    MixBuf<T> cur{LONG ? sm : sm + n, 1 << lb, cs}, other{cur.p + 3 * cs, 1 << lb, cs};
    const cplx<T>* tw = mix_twiddles<T, LONG>(sm, table, n);
    const int kx0 = blockIdx.x << lb, y = blockIdx.y;
    const int64_t zs = (int64_t)My * hxp;
    const MixSpan<T> g{spec + (int64_t)y * hxp + kx0, zs, n * zs};
    auto swap = [&] {
        const MixBuf<T> t = cur;
        cur = other;
        other = t;
    };
    mix_first_wait<T, LONG>(p);
    mix_run_stage<T, LONG, 3, MIX_FIRST>(p, 0, 1, lb, tw, g, cur);
    __syncthreads();
    // forward up to the stage the projector is fused with, then the inverse
    // from the stage after it; one loop, so that the stage code exists once
    const int last = p.nst - 1, nf = fuse ? last : p.nst;
    const T k2 = kyv[y];
    int s = 1, Ns = p.radix[0];
    bool forward = true;
    for (;;) {
        if (forward && s == nf) {
            if (fuse) {
                const bool here = (p.m[last] << lb) <= (int)blockDim.x;
                const MixBuf<T> to = here ? cur : other;
                switch (p.radix[last]) {
#define FFCM_MID(RR) case RR: if constexpr (RR <= mix_fuse_radix<T>() && mix_has_radix<T, LONG>(RR)) \
        mix_middle<T, RR>(p, last, lb, kx0, nkx, tw, cur, to, here, kxv, k2, kzv, inv_mu_M); break;
                    FFCM_MID(2) FFCM_MID(3) FFCM_MID(4) FFCM_MID(5) FFCM_MID(6) FFCM_MID(7) FFCM_MID(8) FFCM_MID(9)
                    FFCM_MID(10)
#undef FFCM_MID
                }
                if (!here) swap();
                s = 1;
                Ns = p.radix[last];
            } else {
                for (int t = threadIdx.x; t < cs; t += blockDim.x) {
                    const int b = t & ((1 << lb) - 1);
                    const T k1 = kx0 + b < nkx ? kxv[kx0 + b] : T(0);
                    project_mode(k1, k2, kzv[t >> lb], inv_mu_M, cur.p[t], cur.p[cs + t], cur.p[2 * cs + t]);
                }
                s = 0;
                Ns = 1;
            }
            __syncthreads();
            forward = false;
        }
        if (!forward && s == last) break;
        const MixPlan& q = forward ? p : pi;
        mix_run_stage<T, LONG, 3, MIX_MID>(q, s, Ns, lb, tw, cur, other);
        __syncthreads();
        swap();
        Ns *= q.radix[s];
        ++s;
    }
    mix_run_stage<T, LONG, 3, MIX_LAST>(pi, last, Ns, lb, tw, cur, g, true);
}

// All stages of the block's lines, between `cur` and `other`; returns the buffer with the result.
template <typename T, bool LONG>
__device__ __forceinline__ const cplx<T>* mix_lines(const MixPlan& p, MixBuf<T> cur, MixBuf<T> other, int lb,
                                                    const cplx<T>* tw) {
    int Ns = 1;
    for (int s = 0; s < p.nst; ++s) {
        mix_run_stage<T, LONG, 1, MIX_MID>(p, s, Ns, lb, tw, cur, other);
        __syncthreads();
        Ns *= p.radix[s];
        const MixBuf<T> t = cur;
        cur = other;
        other = t;
    }
    return cur.p;
}

// B bytes (4, 8, 16; both addresses aligned to them) from global to shared
// memory without passing through registers.
template <int B>
__device__ __forceinline__ void copy_async(void* shared, const void* global) {
    const unsigned to = (unsigned)__cvta_generic_to_shared(shared);
    if constexpr (B == 16) asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(to), "l"(global) : "memory");
    else asm volatile("cp.async.ca.shared.global [%0], [%1], %2;" ::"r"(to), "l"(global), "n"(B) : "memory");
}
__device__ __forceinline__ void copy_async_wait() { asm volatile("cp.async.wait_all;" ::: "memory"); }

// ---- x r2c, rows of the real grid -> rows of the spectrum -----------------
// Even Mx: the row's Mx/2 pairs as one complex line of length Mx/2 (twiddle
// stride 2). Odd Mx: two rows as the real and imaginary part of one line of
// length Mx. A block takes 1 << lb lines; the pitch is one more than that, so
// that the transposing row accesses (consecutive i) reach distinct banks.
template <typename T, bool LONG>
__global__ void __launch_bounds__(sizeof(T) == 4 ? 512 : 256)
    k_fftm_x_r2c(const T* __restrict__ f, cplx<T>* __restrict__ spec, int Mx, int nrows, int hxp,
                 const __grid_constant__ MixPlan p, const cplx<T>* __restrict__ table, int lb) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const int n = p.n, pitch = lb ? (1 << lb) + 1 : 1;
    cplx<T>* sm = reinterpret_cast<cplx<T>*>(smem_raw);
    cplx<T>* A = LONG ? sm : sm + Mx;
    const cplx<T>* tw = mix_twiddles<T, LONG>(sm, table, Mx);
    const bool even = (Mx & 1) == 0;
    const int per = even ? 1 : 2, nlines = (nrows + per - 1) / per;
    const int line0 = blockIdx.x << lb, nl = min(1 << lb, nlines - line0);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nw = blockDim.x >> 5;
    // all of the block's rows in flight at once
    for (int b = warp; b < nl; b += nw) {
        const int64_t row = (int64_t)(line0 + b) * per;
        if (even) {
            const cplx<T>* src = reinterpret_cast<const cplx<T>*>(f + row * Mx);
            for (int i = lane; i < n; i += 32) copy_async<sizeof(cplx<T>)>(A + i * pitch + b, src + i);
        } else {
            const T* src = f + row * Mx;
            const bool two = row + 1 < nrows;
            for (int i = lane; i < n; i += 32) {
                cplx<T>* to = A + i * pitch + b;
                copy_async<sizeof(T)>(&to->x, src + i);
                if (two) copy_async<sizeof(T)>(&to->y, src + Mx + i);
                else to->y = T(0);
            }
        }
    }
    copy_async_wait();
    __syncthreads();
    const cplx<T>* Z = mix_lines<T, LONG>(p, MixBuf<T>{A, pitch, 0}, MixBuf<T>{A + n * pitch, pitch, 0}, lb, tw);
    const int nk = Mx / 2 + 1;
    for (int b = warp; b < nl; b += nw) {
        const int64_t row = (int64_t)(line0 + b) * per;
        cplx<T>* dst = spec + row * hxp;
        const bool two = !even && row + 1 < nrows;
        for (int k = lane; k < nk; k += 32) {
            const cplx<T> Zk = Z[(k == n ? 0 : k) * pitch + b];
            const cplx<T> Zc = cconj(Z[(k == 0 ? 0 : n - k) * pitch + b]);
            const cplx<T> S = cadd(Zk, Zc);
            cplx<T> D = csub(Zk, Zc);
            if (even) {
                D = cmul(tw[k], D);   // X = S/2 - (i/2) W D
                dst[k] = cplx<T>{T(0.5) * (S.x + D.y), T(0.5) * (S.y - D.x)};
            } else {
                dst[k] = cplx<T>{T(0.5) * S.x, T(0.5) * S.y};
                if (two) dst[hxp + k] = cplx<T>{T(0.5) * D.y, T(-0.5) * D.x};
            }
        }
    }
}

// ---- x c2r, spectrum rows -> rows of the real velocity grid ----------------
template <typename T, bool LONG>
__global__ void __launch_bounds__(sizeof(T) == 4 ? 512 : 256)
    k_fftm_x_c2r(const cplx<T>* __restrict__ spec, T* __restrict__ u, int Mx, int nrows, int hxp,
                 const __grid_constant__ MixPlan p, const cplx<T>* __restrict__ table, int lb) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const int n = p.n, pitch = lb ? (1 << lb) + 1 : 1;
    cplx<T>* sm = reinterpret_cast<cplx<T>*>(smem_raw);
    cplx<T>* A = LONG ? sm : sm + Mx;
    const cplx<T>* tw = mix_twiddles<T, LONG>(sm, table, Mx);
    const bool even = (Mx & 1) == 0;
    const int per = even ? 1 : 2, nlines = (nrows + per - 1) / per;
    const int line0 = blockIdx.x << lb, nl = min(1 << lb, nlines - line0);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nw = blockDim.x >> 5;
    // bins k and n - k of a row make the line's values k and n - k
    if (even) {
        // all of the block's rows in flight at once (bin n lies in the second
        // buffer, which the stages use later)
        for (int b = warp; b < nl; b += nw) {
            const cplx<T>* src = spec + (int64_t)(line0 + b) * hxp;
            for (int k = lane; k <= n; k += 32) copy_async<sizeof(cplx<T>)>(A + k * pitch + b, src + k);
        }
        copy_async_wait();
        __syncthreads();
        for (int b = warp; b < nl; b += nw) {
            for (int k = lane; 2 * k <= n; k += 32) {
                cplx<T> Xk = A[k * pitch + b], Xc = A[(n - k) * pitch + b];
                if (k == 0) {
                    Xk.y = T(0);  // DC imaginary part ignored
                    Xc.y = T(0);  // Nyquist imaginary part ignored
                }
                const cplx<T> S = cadd(Xk, cconj(Xc)), D = csub(Xk, cconj(Xc));
                A[k * pitch + b] = cadd(S, mul_pi(cmul(D, cconj(tw[k]))));
                // value n - k: the conjugate sum, and minus the conjugate difference
                if (k > 0)
                    A[(n - k) * pitch + b] =
                        csub(cconj(S), mul_pi(cmul(cconj(D), cconj(tw[n - k]))));
            }
        }
    } else {
        for (int b = warp; b < nl; b += nw) {
            const int64_t row = (int64_t)(line0 + b) * per;
            const cplx<T>* src = spec + row * hxp;
            const bool two = row + 1 < nrows;
#pragma unroll 4
            for (int k = lane; 2 * k < n; k += 32) {
                cplx<T> Xa = src[k], Xb = two ? src[hxp + k] : cplx<T>{T(0), T(0)};
                if (k == 0) Xa.y = Xb.y = T(0);
                A[k * pitch + b] = cadd(Xa, mul_pi(Xb));
                if (k > 0) A[(n - k) * pitch + b] = cadd(cconj(Xa), mul_pi(cconj(Xb)));
            }
        }
    }
    __syncthreads();
    const cplx<T>* Z = mix_lines<T, LONG>(p, MixBuf<T>{A, pitch, 0}, MixBuf<T>{A + n * pitch, pitch, 0}, lb, tw);
    for (int b = warp; b < nl; b += nw) {
        const int64_t row = (int64_t)(line0 + b) * per;
        if (even) {
            cplx<T>* dst = reinterpret_cast<cplx<T>*>(u + row * Mx);
            for (int i = lane; i < n; i += 32) {
                dst[i] = Z[(i == 0 ? 0 : n - i) * pitch + b];   // inverse: element i at n - i
            }
        } else {
            const bool two = row + 1 < nrows;
            for (int i = lane; i < n; i += 32) {
                const cplx<T> z = Z[(i == 0 ? 0 : n - i) * pitch + b];
                u[row * Mx + i] = z.x;
                if (two) u[(row + 1) * Mx + i] = z.y;
            }
        }
    }
}

}  // namespace ffcm
