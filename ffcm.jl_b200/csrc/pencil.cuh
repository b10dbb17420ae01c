// Steps 3 and 5 on the real grid for any grid shape and stencils of up to
// PENCIL_MG points per axis (the assembled operator where the slab kernels do
// not apply).
//
// A pencil is 8 x 4 neighbouring x-rows of the grid, one row per lane of a
// warp. The particles whose stencil reaches a pencil are listed in order of
// their stencil's first x point (a counting sort over (pencil, first x point):
// k_pencil_count, k_pencil_offsets, k_pencil_scatter). A warp walks along a segment of
// its pencil with a window of M_G grid points per lane in registers:
//
//  * k_pencil_spread: the window holds the force sums of the next M_G points;
//    an entry adds (a0 + a2 r^2) gx gy gz F to all of them, and points that the
//    window leaves are final and go to the grid in 32-byte pieces through
//    shared memory (src/spread_forces.jl:73-130). Every grid point is written
//    once by its owner: no atomics, no zeroed grid.
//  * k_pencil_interp: the window holds the velocities; an entry takes the
//    weighted sum over all lanes' windows (src/interpolate.jl:82-136), which is
//    added to the particle's sum with one atomic per component and pencil.
//
// The weights of 32 entries at a time are evaluated by one lane per entry and
// read as broadcasts; the weight of a point is
// gx [(a0 + a2 r2x) (gy gz) + gy gz (a2 r2y + a2 r2z)]: two instructions for two
// points, with 1.34e-7 of the weights lost to Float32 rounding (M_G = 10) where
// (a0 + a2 r^2) gx (gy gz), of three, loses 1.29e-7. The velocities of the record
// configuration (N = 186,510) are 2.49e-7 off in Float32 (mean of five seeds)
// against 2.34e-7 with a warp per particle, in Float64 5.34e-16 against 5.13e-16.
//
// What bounds it: instruction issue (ncu: 63% of issue slots, the rest waits on
// shared memory): per entry and pencil 2.5 M_G two-wide multiply-adds and as
// many instructions again for its weights, loads and the walk; of the
// (M_G + 7)(M_G + 3) rows its pencils hold, an entry uses M_G^2. N = 186,510,
// 256^3, M_G = 10, Float32: spread 296 us (lists and zeroing 39 us more) against 700 us
// with global atomics, which run at one 32-byte sector per L2 slice and clock;
// interpolation 273 against 675 us, where every warp read 20 KB through L1
// (Float64: 470 and 534 against 1035 and 775 us).
#pragma once

#include "common.cuh"
#include "slab.cuh"
#include "spread_interp.cuh"

namespace ffcm {

constexpr int PENCIL_TY = 8, PENCIL_TZ = 4;   // rows of a pencil, one per lane
constexpr int PENCIL_MG = 12;                 // widest stencil with an instance
constexpr int PENCIL_WARPS = 2;               // warps per block (they share nothing)

struct PencilGeom {
    int nty, ntz;    // pencils along y and z
    int nseg, seg;   // segments of a row, points per segment
    int part;        // most entries a warp walks: longer segments go to several
};

// The warps' tasks: one per segment (its part 0), and the further parts of the
// segments whose entries exceed PencilGeom::part, so that a cluster's entries,
// which lie in few segments, do not keep a few warps busy alone. Parts of a
// segment add their sums to its grid points, zeroed by k_pencil_zero.
struct PencilTasks {
    int* parts;   // per segment: parts, 1 or more
    int2* more;   // (segment, part > 0)
    int* nmore;
};

// Pencils along one axis (tiles of TS rows out of M) that the rows s .. s + MG - 1
// (mod M, s in [0, M)) reach, each once: tile(0 .. n - 1).
template <int TS>
struct PencilReach {
    int t0, n1, n;
    __device__ __forceinline__ PencilReach(int s, int MG, int M) {
        t0 = s / TS;
        n1 = (min(s + MG, M) - 1) / TS - t0 + 1;
        n = n1 + (s + MG > M ? min((s + MG - M - 1) / TS, t0 - 1) + 1 : 0);
    }
    __device__ __forceinline__ int tile(int i) const { return i < n1 ? t0 + i : i - n1; }
};

// Most pencils one particle can reach along an axis (tiles of ts rows): one more
// where the last tile is a short one.
inline int pencil_reach(int ts, int MG, int M) {
    return std::min((M + ts - 1) / ts, (MG + ts - 2) / ts + (M % ts == 0 ? 1 : 2));
}

// First x point of a stencil, in [0, Mx).
template <typename T>
__device__ __forceinline__ int pencil_first(const StencilParams<T>& p, T y) {
    return imod(stencil_anchor(p, y) - p.half, p.Mx);
}

// PENCIL_SPLIT threads share a sorted particle: calls f(s, pencil, first x
// point) for every bin of every particle.
constexpr int PENCIL_SPLIT = 4;

template <typename T, typename F>
__device__ __forceinline__ void pencil_bins(int n_part, const vec4<T>* __restrict__ Ys, const StencilParams<T>& p,
                                            const PencilGeom& g, F f) {
    const int64_t n = (int64_t)n_part * PENCIL_SPLIT, step = (int64_t)gridDim.x * blockDim.x;
    for (int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; t < n; t += step) {
        const int s = (int)(t / PENCIL_SPLIT);
        const vec4<T> y = Ys[s];
        const int x0 = pencil_first(p, y.x);
        const PencilReach<PENCIL_TY> ry(imod(stencil_anchor(p, y.y) - p.half, p.My), p.MG, p.My);
        const PencilReach<PENCIL_TZ> rz(imod(stencil_anchor(p, y.z) - p.half, p.Mz), p.MG, p.Mz);
        for (int q = (int)(t % PENCIL_SPLIT); q < ry.n * rz.n; q += PENCIL_SPLIT) {
            const int iz = q / ry.n;
            f(s, rz.tile(iz) * g.nty + ry.tile(q - iz * ry.n), x0);
        }
    }
}

template <typename T>
__global__ void k_pencil_count(int n_part, const vec4<T>* __restrict__ Ys, StencilParams<T> p, PencilGeom g,
                               int* __restrict__ cnt, PencilTasks tasks) {
    if (blockIdx.x == 0 && threadIdx.x == 0) *tasks.nmore = 0;
    pencil_bins(n_part, Ys, p, g, [&](int, int pen, int x) { atomicAdd(&cnt[pen * p.Mx + x], 1); });
}

// The entries of a pencil whose stencil reaches its points [xs, xe), from its bin
// boundaries: first points xs - MG + 1 .. xe - 1, those below 0 from the row's
// end (entries a0 .. a0 + na - 1, the image one period lower), then b0 .. b0 +
// nb - 1.
__device__ __forceinline__ void pencil_range(const int* bins, int xs, int xe, int Mx, int MG, int& a0,
                                             int& na, int& b0, int& nb) {
    const int lo = xs - MG + 1;
    a0 = lo < 0 ? bins[lo + Mx] : 0;
    na = lo < 0 ? bins[Mx] - a0 : 0;
    b0 = bins[max(lo, 0)];
    nb = bins[xe] - b0;
}

// One warp per pencil: offsets of its Mx + 1 bin boundaries from the bin counts.
// The pencils take their parts of the entry list in any order (one atomic
// each), so no scan across pencils is needed. *used and *tasks.nmore are zero
// before (k_pencil_scatter resets the one, k_pencil_count the other).
__global__ void k_pencil_offsets(int npen, int Mx, int MG, PencilGeom g, const int* __restrict__ cnt,
                                 int* __restrict__ off, int* __restrict__ used, PencilTasks tasks) {
    const int lane = threadIdx.x & 31;
    const int pen = (int)((blockIdx.x * blockDim.x + threadIdx.x) >> 5);
    if (pen >= npen) return;   // whole warps
    const int* c = cnt + (int64_t)pen * Mx;
    int* o = off + (int64_t)pen * (Mx + 1);
    int total = 0;
    for (int x = lane; x < Mx; x += 32) total += c[x];
#pragma unroll
    for (int d = 16; d > 0; d >>= 1) total += __shfl_xor_sync(0xffffffffu, total, d);
    int base = lane == 0 && total > 0 ? atomicAdd(used, total) : 0;
    base = __shfl_sync(0xffffffffu, base, 0);
    for (int x0 = 0; x0 < Mx; x0 += 32) {
        const int v = x0 + lane < Mx ? c[x0 + lane] : 0;
        int s = v;
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
            const int t = __shfl_up_sync(0xffffffffu, s, d);
            if (lane >= d) s += t;
        }
        if (x0 + lane < Mx) o[x0 + lane] = base + s - v;
        base += __shfl_sync(0xffffffffu, s, 31);
    }
    if (lane == 0) o[Mx] = base;
    __syncwarp();
    for (int q = lane; q < g.nseg; q += 32) {
        int a0, na, b0, nb;
        pencil_range(o, q * g.seg, min((q + 1) * g.seg, Mx), Mx, MG, a0, na, b0, nb);
        const int n = max(1, (int)(((int64_t)na + nb + g.part - 1) / g.part)), seg = pen * g.nseg + q;
        tasks.parts[seg] = n;
        if (n > 1) {
            const int at = atomicAdd(tasks.nmore, n - 1);
            for (int i = 1; i < n; ++i) tasks.more[at + i - 1] = make_int2(seg, i);
        }
    }
}

// Zeroes the grid points of the segments that several warps share.
template <typename T>
__global__ void k_pencil_zero(StencilParams<T> p, PencilGeom g, PencilTasks tasks, T* __restrict__ grid) {
    const int n = *tasks.nmore;
    for (int i = blockIdx.x; i < n; i += gridDim.x) {
        const int2 t = tasks.more[i];
        if (t.y != 1) continue;   // once a segment
        const int pen = t.x / g.nseg, xs = (t.x - pen * g.nseg) * g.seg, w = min(g.seg, p.Mx - xs);
        const int y0r = pen % g.nty * PENCIL_TY, z0r = pen / g.nty * PENCIL_TZ;
        const int ny = min(PENCIL_TY, p.My - y0r), nz = min(PENCIL_TZ, p.Mz - z0r);
        for (int e = threadIdx.x; e < 3 * ny * nz * w; e += blockDim.x) {
            int r = e / w;
            const int x = e - r * w, c = r / (ny * nz);
            r -= c * ny * nz;
            const int z = r / ny, y = r - z * ny;
            grid[(((int64_t)c * p.Mz + z0r + z) * p.My + y0r + y) * p.Mx + xs + x] = T(0);
        }
    }
}

// cnt is consumed (left zero for the next count), as is *used.
template <typename T>
__global__ void k_pencil_scatter(int n_part, const vec4<T>* __restrict__ Ys, StencilParams<T> p, PencilGeom g,
                                 const int* __restrict__ off, int* __restrict__ cnt, int* __restrict__ ent,
                                 int* __restrict__ used) {
    if (blockIdx.x == 0 && threadIdx.x == 0) *used = 0;
    pencil_bins(n_part, Ys, p, g, [&](int s, int pen, int x) {
        ent[off[pen * (p.Mx + 1) + x] + atomicSub(&cnt[pen * p.Mx + x], 1) - 1] = s;
    });
}

// Per-warp shared memory: the weights of 32 entries and a staging area of XC
// grid columns (32 bytes of each row).
template <typename T, int MGT>
struct PencilWarp {
    static constexpr int XC = 32 / (int)sizeof(T);
    // x weights of an entry, read as 16-byte broadcasts; the stride is an odd
    // number of 16-byte chunks, so that the lanes' stores meet distinct banks
    static constexpr int PER = 16 / (int)sizeof(T);
    static constexpr int CH = (2 * MGT + PER - 1) / PER;
    static constexpr int SW = (CH | 1) * PER;
    T wx[32][SW];                        // gx of the M_G points, then a0 + a2 r2x
    // (ry, rz: a2 r2y, a2 r2z)
    T gy[PENCIL_TY][33], ry[PENCIL_TY][33], gz[PENCIL_TZ][33], rz[PENCIL_TZ][33];
    T stage[3][32][XC + 1];
    int x0[32];                          // first x point, relative to the segment's row
};

// The same with the forces, as pairs of equal values.
template <typename T, int MGT>
struct PencilSpreadWarp {
    PencilWarp<T, MGT> w;
    T f[32][8];
};

// Weights of the entry a lane holds into slot `lane`.
template <typename T, int MGT>
__device__ __forceinline__ void pencil_put(const StencilParams<T>& p, PencilWarp<T, MGT>& W, int lane,
                                           const vec4<T>& y, int y0r, int z0r) {
    const int sx = stencil_anchor(p, y.x) - p.half, sy = stencil_anchor(p, y.y) - p.half,
              sz = stencil_anchor(p, y.z) - p.half;
    // stencil_offset with the mode's branch taken once
    auto fill = [&](auto offset) {
        auto weight = [&](int g, T yy, T& gw, T& r2) {
            const T x = offset(g, yy);
            r2 = mul_rn(x, x);
            gw = p.inv_norm * exp_t(-r2 * p.inv_2S2);
        };
        // (the walk's window stays in registers meanwhile: little unrolling)
#pragma unroll 2
        for (int k = 0; k < MGT; ++k) {
            T gx, r2;
            weight(sx + k, y.x, gx, r2);
            if (k >= p.MG) gx = T(0);
            W.wx[lane][k] = gx;
            W.wx[lane][MGT + k] = p.a0 + p.a2 * r2;
        }
#pragma unroll 2
        for (int b = 0; b < PENCIL_TY; ++b) {
            const int d = wrap1(y0r + b - sy, p.My);
            T g, r2;
            weight(sy + d, y.y, g, r2);
            const bool hit = d < p.MG && y0r + b < p.My;
            W.gy[b][lane] = hit ? g : T(0);
            W.ry[b][lane] = hit ? p.a2 * r2 : T(0);
        }
#pragma unroll 2
        for (int b = 0; b < PENCIL_TZ; ++b) {
            const int d = wrap1(z0r + b - sz, p.Mz);
            T g, r2;
            weight(sz + d, y.z, g, r2);
            const bool hit = d < p.MG && z0r + b < p.Mz;
            W.gz[b][lane] = hit ? g : T(0);
            W.rz[b][lane] = hit ? p.a2 * r2 : T(0);
        }
    };
    if (p.comp) fill([&](int g, T yy) { return fma_t((T)g, p.h_hi, -yy) + (T)g * p.h_lo; });
    else fill([&](int g, T yy) { return sub_rn(mul_rn((T)g, p.h), yy); });
}

// n pairs from shared memory in 16-byte loads.
template <typename T, int n>
__device__ __forceinline__ void load_pairs(const T* p, pair2<T> (&v)[n]) {
    if constexpr (sizeof(T) == 4) {
        static_assert(n % 2 == 0, "whole 16-byte chunks");
#pragma unroll
        for (int i = 0; i < n / 2; ++i) {
            const ulonglong2 c = reinterpret_cast<const ulonglong2*>(p)[i];
            v[2 * i].v = c.x;
            v[2 * i + 1].v = c.y;
        }
    } else {
#pragma unroll
        for (int i = 0; i < n; ++i) {
            const double2 c = reinterpret_cast<const double2*>(p)[i];
            v[i] = pair2<T>(c.x, c.y);
        }
    }
}

// A warp's accesses to XC columns of its pencil's rows: lane (row l / XC of a
// group of 32 / XC rows, column l % XC); f(row, valid, grid offset) per group.
template <typename T, int MGT>
struct PencilRows {
    static constexpr int XC = PencilWarp<T, MGT>::XC, GROUP = 32 / XC;
    int64_t base;    // grid offset of the lane's row in the first group
    int ny, nz;      // rows of the pencil inside the grid
    __device__ __forceinline__ PencilRows(const StencilParams<T>& p, int y0r, int z0r, int lane) {
        base = ((int64_t)z0r * p.My + y0r + lane / XC) * p.Mx;
        ny = p.My - y0r - lane / XC;
        nz = p.Mz - z0r;
    }
    template <typename F>
    __device__ __forceinline__ void each(const StencilParams<T>& p, int lane, F f) const {
        const int64_t zs = (int64_t)p.My * p.Mx;
#pragma unroll
        for (int d = 0; d < PENCIL_TZ; ++d)
#pragma unroll
            for (int b = 0; b < PENCIL_TY; b += GROUP)
                f(d * PENCIL_TY + b + lane / XC, b < ny && d < nz, base + d * zs + b * p.Mx);
    }
    // staged columns added to the grid, where `on` (rolled: with the code of 96
    // atomics beside the stores, and a third more idle blocks, every spread of the
    // record configuration took 371 us instead of 335)
    __device__ __forceinline__ void add(const StencilParams<T>& p, int lane, bool on, int64_t plane, T* out,
                                     const T (*stage)[32][XC + 1]) const {
        if (!on) return;
#pragma unroll 1
        for (int i = 0; i < 3 * PENCIL_TZ * PENCIL_TY; i += GROUP) {
            const int c = i / (PENCIL_TZ * PENCIL_TY), d = i / PENCIL_TY % PENCIL_TZ, b = i % PENCIL_TY;
            if (b < ny && d < nz)
                atomicAdd(out + c * plane + base + ((int64_t)d * p.My + b) * p.Mx,
                          stage[c][d * PENCIL_TY + b + lane / XC][lane % XC]);
        }
    }
};

// The warp's task: segment and part of it; false beyond the last one.
__device__ __forceinline__ bool pencil_task(const PencilGeom& g, const PencilTasks& tasks, int& seg, int& part,
                                            int& parts) {
    const int nseg = g.nty * g.ntz * g.nseg, task = blockIdx.x * PENCIL_WARPS + (threadIdx.x >> 5);
    seg = task;
    part = 0;
    if (task >= nseg) {
        if (task - nseg >= *tasks.nmore) return false;
        const int2 t = tasks.more[task - nseg];
        seg = t.x;
        part = t.y;
    }
    parts = tasks.parts[seg];
    return true;
}

template <typename T, int MGT>
__global__ void __launch_bounds__(32 * PENCIL_WARPS, sizeof(T) == 4 ? 10 : 6)
    k_pencil_spread(const vec4<T>* __restrict__ Ys, const vec4<T>* __restrict__ Fs, const __grid_constant__
                    StencilParams<T> p, PencilGeom g, const int* __restrict__ off, const int* __restrict__ ent,
                    PencilTasks tasks, T* __restrict__ grid, T* __restrict__ Vs, int64_t nvs) {
    using Warp = PencilWarp<T, MGT>;
    constexpr int XC = Warp::XC;
    zero_sums(Vs, nvs);
    extern __shared__ __align__(32) unsigned char pencil_smem[];
    const int lane = threadIdx.x & 31;
    PencilSpreadWarp<T, MGT>& S = reinterpret_cast<PencilSpreadWarp<T, MGT>*>(pencil_smem)[threadIdx.x >> 5];
    Warp& W = S.w;
    int seg, part, parts;
    if (!pencil_task(g, tasks, seg, part, parts)) return;   // whole warps
    const int pen = seg / g.nseg;
    const int xs = (seg - pen * g.nseg) * g.seg, xe = min(xs + g.seg, p.Mx);
    const int y0r = pen % g.nty * PENCIL_TY, z0r = pen / g.nty * PENCIL_TZ;
    const PencilRows<T, MGT> rows(p, y0r, z0r, lane);
    const int64_t plane = (int64_t)p.Mx * p.My * p.Mz;
    int a0, na, b0, nb;
    pencil_range(off + (int64_t)pen * (p.Mx + 1), xs, xe, p.Mx, p.MG, a0, na, b0, nb);
    // the part's entries; parts > 1: the points they reach, added to the grid
    const int first = (int)((int64_t)(na + nb) * part / parts), total = (int)((int64_t)(na + nb) * (part + 1) / parts);
    int xend = xe;
    pair2<T> acc[3][MGT / 2];
#pragma unroll
    for (int c = 0; c < 3; ++c)
#pragma unroll
        for (int k = 0; k < MGT / 2; ++k) acc[c][k] = pair2<T>(T(0), T(0));
    int X = xs - p.MG + 1;   // x of acc[.][0]
    auto advance = [&] {
        if (X >= xs) {
            const int col = (X - xs) % XC;
#pragma unroll
            for (int c = 0; c < 3; ++c) W.stage[c][lane][col] = acc[c][0].x();
            if (col == XC - 1 || X == xend - 1) {
                __syncwarp();
                const int cc = lane % XC;
                T* out = grid + (X - col + cc);
                if (parts == 1) {
                    rows.each(p, lane, [&](int r, bool in, int64_t at) {
                        if (in && cc <= col) {
#pragma unroll
                            for (int c = 0; c < 3; ++c) out[c * plane + at] = W.stage[c][r][cc];
                        }
                    });
                } else {
                    rows.add(p, lane, cc <= col, plane, out, W.stage);
                }
                __syncwarp();
            }
        }
#pragma unroll
        for (int c = 0; c < 3; ++c) {
#pragma unroll
            for (int k = 0; k + 1 < MGT / 2; ++k) acc[c][k] = pair2<T>(acc[c][k].y(), acc[c][k + 1].x());
            acc[c][MGT / 2 - 1] = pair2<T>(acc[c][MGT / 2 - 1].y(), T(0));
        }
        ++X;
    };
    // entry i: list position and the particle, loaded one batch ahead
    int xn = 0;
    vec4<T> yn{}, fn{};
    auto fetch = [&](int i) {
        if (i < total) {
            const int s = ent[i < na ? a0 + i : b0 + i - na];
            yn = Ys[s];
            fn = Fs[s];
            xn = pencil_first(p, yn.x) - (i < na ? p.Mx : 0);
        }
    };
    fetch(first + lane);
    if (parts > 1) {   // from the chunk of the first entry's first point
        const int x = __shfl_sync(0xffffffffu, xn, 0);
        X = x < xs ? x : x - (x - xs) % XC;
    }
    for (int base = first; base < total; base += 32) {
        const int n = min(32, total - base);
        if (lane < n) {
            W.x0[lane] = xn;
            store16<T, 8>(&S.f[lane][0], {fn.x, fn.x, fn.y, fn.y, fn.z, fn.z, fn.z, fn.z});
            pencil_put<T, MGT>(p, W, lane, yn, y0r, z0r);
        }
        __syncwarp();
        fetch(base + 32 + lane);
        for (int e = 0; e < n; ++e) {
            const int x0 = W.x0[e];
            while (X < x0) advance();
            const T gyz = W.gy[lane % PENCIL_TY][e] * W.gz[lane / PENCIL_TY][e];
            const T q = gyz * (W.ry[lane % PENCIL_TY][e] + W.rz[lane / PENCIL_TY][e]);
            pair2<T> f[4];
            load_pairs<T, 4>(&S.f[e][0], f);
            const pair2<T> g2(gyz, gyz), q2(q, q);
            pair2<T> w[MGT];
            load_pairs<T, MGT>(&W.wx[e][0], w);
#pragma unroll
            for (int k = 0; k < MGT / 2; ++k) {
                const pair2<T> wgt = mul2(w[k], fma2(w[MGT / 2 + k], g2, q2));
#pragma unroll
                for (int c = 0; c < 3; ++c) acc[c][k] = fma2(wgt, f[c], acc[c][k]);
            }
        }
        __syncwarp();
    }
    if (parts > 1) xend = min(xe, X + MGT);
    while (X < xend) advance();
}

// Sums for entries in groups: every lane leaves its part of an
// entry's three components in shared memory, then one lane per (entry,
// component) adds them up.
template <typename T, int MGT>
struct PencilInterpWarp {
    static constexpr int SUM_GROUP = sizeof(T) == 4 ? 8 : 4;
    PencilWarp<T, MGT> w;
    T part[3 * SUM_GROUP][33];
    int s[32];
};

template <typename T, int MGT>
__global__ void __launch_bounds__(32 * PENCIL_WARPS, sizeof(T) == 4 ? 8 : 5)
    k_pencil_interp(const vec4<T>* __restrict__ Ys, const __grid_constant__ StencilParams<T> p, PencilGeom g,
                    const int* __restrict__ off, const int* __restrict__ ent, PencilTasks tasks,
                    const T* __restrict__ grid, T* __restrict__ Vs) {
    using Warp = PencilWarp<T, MGT>;
    constexpr int XC = Warp::XC;
    extern __shared__ __align__(32) unsigned char pencil_smem[];
    const int lane = threadIdx.x & 31;
    PencilInterpWarp<T, MGT>& I = reinterpret_cast<PencilInterpWarp<T, MGT>*>(pencil_smem)[threadIdx.x >> 5];
    Warp& W = I.w;
    constexpr int SUM_GROUP = PencilInterpWarp<T, MGT>::SUM_GROUP;
    int seg, part, parts;
    if (!pencil_task(g, tasks, seg, part, parts)) return;   // whole warps
    const int pen = seg / g.nseg;
    const int xs = (seg - pen * g.nseg) * g.seg, xe = min(xs + g.seg, p.Mx);
    const int y0r = pen % g.nty * PENCIL_TY, z0r = pen / g.nty * PENCIL_TZ;
    const PencilRows<T, MGT> rows(p, y0r, z0r, lane);
    const int64_t plane = (int64_t)p.Mx * p.My * p.Mz;
    // every entry belongs to the segment its first point lies in
    const int* bins = off + (int64_t)pen * (p.Mx + 1);
    const int b0 = bins[xs], all = bins[xe] - b0;
    const int first = (int)((int64_t)all * part / parts), total = (int)((int64_t)all * (part + 1) / parts);
    if (first == total) return;
    pair2<T> u[3][MGT / 2];
#pragma unroll
    for (int c = 0; c < 3; ++c)
#pragma unroll
        for (int k = 0; k < MGT / 2; ++k) u[c][k] = pair2<T>(T(0), T(0));
    // columns are read XC at a time, one chunk ahead of the staged one
    T next[3][32 / PencilRows<T, MGT>::GROUP];
    auto load_chunk = [&](int xb) {
        int x = xb + lane % XC;
        while (x >= p.Mx) x -= p.Mx;
        int i = 0;
        rows.each(p, lane, [&](int, bool in, int64_t at) {
#pragma unroll
            for (int c = 0; c < 3; ++c) next[c][i] = in ? __ldg(grid + c * plane + at + x) : T(0);
            ++i;
        });
    };
    int sn = 0;
    vec4<T> yn{};
    auto fetch = [&](int i) {
        if (i < total) {
            sn = ent[b0 + i];
            yn = Ys[sn];
        }
    };
    fetch(first + lane);
    // x of u[.][0]: the first column to come is the chunk of the first entry's first point
    int X = xs - MGT + (pencil_first(p, __shfl_sync(0xffffffffu, yn.x, 0)) - xs) / XC * XC;
    load_chunk(X + MGT);
    auto advance = [&] {   // shifts column X + MGT in
        const int col = (X + MGT - xs) % XC;
        if (col == 0) {
            __syncwarp();
#pragma unroll
            for (int i = 0; i < XC; ++i)
#pragma unroll
                for (int c = 0; c < 3; ++c)
                    W.stage[c][i * PencilRows<T, MGT>::GROUP + lane / XC][lane % XC] = next[c][i];
            __syncwarp();
            load_chunk(X + MGT + XC);
        }
#pragma unroll
        for (int c = 0; c < 3; ++c) {
#pragma unroll
            for (int k = 0; k + 1 < MGT / 2; ++k) u[c][k] = pair2<T>(u[c][k].y(), u[c][k + 1].x());
            u[c][MGT / 2 - 1] = pair2<T>(u[c][MGT / 2 - 1].y(), W.stage[c][lane][col]);
        }
        ++X;
    };
    for (int base = first; base < total; base += 32) {
        const int n = min(32, total - base);
        if (lane < n) {
            I.s[lane] = sn;
            W.x0[lane] = pencil_first(p, yn.x);
            pencil_put<T, MGT>(p, W, lane, yn, y0r, z0r);
        }
        __syncwarp();
        fetch(base + 32 + lane);
        for (int e0 = 0; e0 < n; e0 += SUM_GROUP) {
            const int m = min(SUM_GROUP, n - e0);
            for (int j = 0; j < m; ++j) {
                const int e = e0 + j, x0 = W.x0[e];
                while (X < x0) advance();
                const T gyz = W.gy[lane % PENCIL_TY][e] * W.gz[lane / PENCIL_TY][e];
                const T q = gyz * (W.ry[lane % PENCIL_TY][e] + W.rz[lane / PENCIL_TY][e]);
                const pair2<T> g2(gyz, gyz), q2(q, q);
                pair2<T> w[MGT];
                load_pairs<T, MGT>(&W.wx[e][0], w);
                pair2<T> v[3];
#pragma unroll
                for (int k = 0; k < MGT / 2; ++k) {
                    const pair2<T> wgt = mul2(w[k], fma2(w[MGT / 2 + k], g2, q2));
#pragma unroll
                    for (int c = 0; c < 3; ++c) v[c] = k == 0 ? mul2(wgt, u[c][0]) : fma2(wgt, u[c][k], v[c]);
                }
#pragma unroll
                for (int c = 0; c < 3; ++c) I.part[3 * j + c][lane] = v[c].x() + v[c].y();
            }
            __syncwarp();
            if (lane < 3 * m) {
                // in eight partial sums, then pairwise
                T v[8];
#pragma unroll
                for (int r = 0; r < 32; ++r) v[r % 8] = r < 8 ? I.part[lane][r] : v[r % 8] + I.part[lane][r];
                atomicAdd(Vs + 3 * (int64_t)I.s[e0 + lane / 3] + lane % 3,
                          ((v[0] + v[1]) + (v[2] + v[3])) + ((v[4] + v[5]) + (v[6] + v[7])));
            }
            __syncwarp();
        }
    }
}

template <typename T>
using PencilSpreadKernel = void (*)(const vec4<T>*, const vec4<T>*, const StencilParams<T>, PencilGeom, const int*,
                                    const int*, PencilTasks, T*, T*, int64_t);
template <typename T>
using PencilInterpKernel = void (*)(const vec4<T>*, const StencilParams<T>, PencilGeom, const int*, const int*,
                                    PencilTasks, const T*, T*);

template <typename T>
struct PencilKernels {
    PencilSpreadKernel<T> spread = nullptr;
    PencilInterpKernel<T> interp = nullptr;
    size_t smem = 0, smem_interp = 0;
};

// The instance of the next even width (the points beyond M_G carry zero
// weights); false where there is none.
template <typename T>
bool pencil_kernels(int MG, PencilKernels<T>& k) {
    auto set = [&](auto w) {
        constexpr int W = decltype(w)::value;
        k.spread = k_pencil_spread<T, W>;
        k.interp = k_pencil_interp<T, W>;
        k.smem = PENCIL_WARPS * sizeof(PencilSpreadWarp<T, W>);
        k.smem_interp = PENCIL_WARPS * sizeof(PencilInterpWarp<T, W>);
        return true;
    };
    if (MG <= 6) return set(std::integral_constant<int, 6>{});
    if (MG <= 8) return set(std::integral_constant<int, 8>{});
    if (MG <= 10) return set(std::integral_constant<int, 10>{});
    if (MG <= PENCIL_MG) return set(std::integral_constant<int, 12>{});
    return false;
}

}  // namespace ffcm
