// direct.cu — the correction solve A e = r of the Poisson refinement by fast
// diagonalisation.
//
// The 7-point operator on the unknowns (held faces or periodic axes, dx = 1) is
// a Kronecker sum of three second differences, each diagonal in an orthonormal
// basis of its axis: sines between held faces, the real Fourier basis on a
// periodic axis. e = Q (Q^T r) / (lambda_a + lambda_b + lambda_c), one
// transform per axis and direction, any axis length, so a correction is exact
// up to FP32 rounding: it lowers ||r|| to 1e-6 of it where r is noise (7e-7 at
// 63^3, 3e-6 at 255^3) and to 1e-4 where r is smooth (9e-5 and 2e-3, the rounding of
// the large e), where a V(2,1) multigrid cycle lowers it to 0.18 and, on an axis
// whose length stops coarsening early (an odd periodic one) or halves evenly between
// held faces, less or not at all. The residual
// stays FP64 and decides, as in the multigrid refinement.
//
// Transforms are dense products with the basis, halved by its parity: index
// pairs (j, j') that mirror each other enter as sum and difference, which the
// even and the odd modes see with two half-size matrices. 127^3: 0.26 GFLOP per
// transform, 1.6 GFLOP per correction (six transforms).
//
// Kernels. A CTA holds a tile of 64 lines (32 where those would not fill the
// GPU, or not fit) in shared memory, all indices of the axis, so it reads and
// writes each value once and works in place; the transform along a, the
// division and the transform back are one kernel. A thread sums 8 modes x 8
// lines of one half: a shared-memory wavefront brings one value per lane and
// the SM issues four multiply-adds per wavefront, so 16 values per 64
// multiply-adds keep both pipes even. The matrices arrive in chunks of 16 rows
// through a three-stage cp.async ring whose first stages are requested before
// the wait for the previous kernel. At 127^3 a transform takes 16 us, at 255^3
// 156 us (27 TFLOP/s of the 72 that FP32 multiply-adds reach here). There the FP32
// pipe is busy 47-49 % of the time and the issue slots 44 %: shared memory leaves
// room for one CTA, two warps a scheduler, which do not cover the waits on each
// other's results; at 127^3 the load and store phases of the 1.7 tiles an SM gets
// come on top. 4 x 4 tiles of both halves: 22 us at 127^3.
#include "direct.cuh"

#include <algorithm>
#include <cmath>
#include <vector>

namespace fopis {

namespace {

// Unknowns per axis. A correction costs O(n^4), a V-cycle O(n^3), but a solve
// takes 2 of the first where it takes 7-8 of the second; cold solves to 1e-8,
// six held faces, V-cycles against this: 127^3 1.31 / 0.26 ms, 255^3 6.9 / 2.3,
// 383^3 20.9 / 13.9, 511^3 48.2 / 32.6, 575^3 57.5 / 62.7, 639^3 77.7 / 87.3,
// 767^3 133 / 273. (From a start within 1e-6, 2 V-cycles against one correction,
// cubes cross earlier: 383^3 5.5 / 7.1, 511^3 12.3 / 16.7; within 1e-3, 4 against one,
// where they do cold.) 120 x 75 x 50 with two periodic axes (coarsening stops at 60 x 36
// x 25): 65 / 0.3 ms. So the line is where cubes cross over. It looks at the longest
// axis alone: a long thin box beyond it would still gain (513 x 18 x 18 61 / 0.4 ms,
// 767 x 63 x 63 13 / 1.0, 639 x 319 x 319 20.8 / 16.8).
constexpr int kDirectMax = 512;
constexpr int kThreads = 256;
constexpr int kWarps = kThreads / 32;
constexpr int kRows = 16;         // matrix rows per stage
constexpr int kStages = 3;
constexpr int kModes = 128;       // modes of one pass

__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void cp_async16(float* dst, const float* src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((unsigned)__cvta_generic_to_shared(dst)), "l"(src));
}
__device__ __forceinline__ void cp_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

// Modes of a pass: the axis' modes in equal passes of at most kModes.
__host__ __device__ __forceinline__ int pass_modes(int hp) {
    const int passes = (hp + kModes - 1) / kModes;
    return ((hp + passes - 1) / passes + 7) / 8 * 8;
}

// Folded index p of an axis: the mirrored pair (ja, jb), or a self-mirrored
// index (jb < 0).
__device__ __forceinline__ void fold_pair(const DirectAxis& x, int p, int& ja, int& jb) {
    if (x.per) {
        if (p < x.np) { ja = p + 1; jb = x.n - 1 - p; }
        else { ja = p == x.np ? 0 : x.n / 2; jb = -1; }
    } else {
        ja = p;
        jb = p < x.np ? x.n - 1 - p : -1;
    }
}

// Two FP32 multiply-adds in one instruction (each rounded as fmaf rounds it).
__device__ __forceinline__ void fma2(unsigned long long& d, unsigned long long a, unsigned long long b) {
    asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(d) : "l"(a), "l"(b));
}
__device__ __forceinline__ unsigned long long pack2(float lo, float hi) {
    unsigned long long v;
    asm("mov.b64 %0, {%1, %2};" : "=l"(v) : "f"(lo), "f"(hi));
    return v;
}
__device__ __forceinline__ float2 unpack2(unsigned long long v) {
    float2 f;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(f.x), "=f"(f.y) : "l"(v));
    return f;
}

// The 8 x 8 sums of a thread as pairs of modes: s[i][l] holds the products of
// modes (2i, 2i + 1) with lines (2l, 2l + 1), t[i][l] those with the lines
// swapped, so that no operand has to be duplicated.
struct Sums {
    unsigned long long s[4][4], t[4][4];
    __device__ __forceinline__ void clear() {
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
            for (int l = 0; l < 4; ++l) s[i][l] = t[i][l] = 0ull;
    }
    __device__ __forceinline__ void add(const float a[8], const float v[8]) {
        unsigned long long m[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) m[i] = pack2(a[2 * i], a[2 * i + 1]);
#pragma unroll
        for (int l = 0; l < 4; ++l) {
            const unsigned long long x = pack2(v[2 * l], v[2 * l + 1]), y = pack2(v[2 * l + 1], v[2 * l]);
#pragma unroll
            for (int i = 0; i < 4; ++i) { fma2(s[i][l], m[i], x); fma2(t[i][l], m[i], y); }
        }
    }
    __device__ __forceinline__ void get(float d[8][8]) const {
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
            for (int l = 0; l < 4; ++l) {
                const float2 x = unpack2(s[i][l]), y = unpack2(t[i][l]);
                d[2 * i][2 * l] = x.x; d[2 * i + 1][2 * l + 1] = x.y;
                d[2 * i][2 * l + 1] = y.x; d[2 * i + 1][2 * l] = y.y;
            }
    }
};

// Rows [p0, p0 + kRows) of both matrices, columns [mb, mb + wm), into a stage.
__device__ __forceinline__ void stage_rows(const DirectAxis& x, const float* We, const float* Wo, int p0, int mb, int wm,
                                           float* st) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int m = 4 * lane;
#pragma unroll
    for (int t = 0; t < 2 * kRows / kWarps; ++t) {
        const int r = warp + t * kWarps, row = r & (kRows - 1);
        if (p0 + row < x.hp && m < wm && mb + m < x.hp)
            cp_async16(st + r * wm + m, (r < kRows ? We : Wo) + (long long)(p0 + row) * x.hp + mb + m);
    }
}

// Requests the first two stages of a product's first pass.
__device__ __forceinline__ void product_begin(const DirectAxis& x, const float* We, const float* Wo, float* ring) {
    const int wm = pass_modes(x.hp);
    stage_rows(x, We, Wo, 0, 0, wm, ring);
    cp_commit();
    stage_rows(x, We, Wo, kRows, 0, wm, ring + 2 * kRows * wm);
    cp_commit();
}

// d[i][l] = sum over p of W[p][m0 + i] U[p][line l] for one half (odd: the
// second one), for every pass of modes, into V[half][m0 + i][line l] after
// scale(odd, m0, l0, d). U and V are [2][hp] rows of TS floats, T of them lines;
// a thread's lines are 4 l0 + {0..3} and T/2 + 4 l0 + {0..3}. Every thread of
// the block calls it, after product_begin.
template <int T, int TS, typename Scale>
__device__ __forceinline__ void product(const DirectAxis& x, const float* We, const float* Wo, const float* U, float* V,
                                        float* ring, Scale scale) {
    constexpr int LG = T / 8;                    // threads over the lines
    const int wm = pass_modes(x.hp), stage = 2 * kRows * wm, chunks = (x.hp + kRows - 1) / kRows;
    const int per = wm / 8 * LG;                 // threads of a half
    const int odd = threadIdx.x >= per, rest = threadIdx.x - odd * per;
    const int l0 = 4 * (rest % LG), g = rest / LG * 8;
    const float* Uh = U + odd * x.hp * TS + l0;
    for (int mb = 0; mb < x.hp; mb += wm) {
        const bool on = (int)threadIdx.x < 2 * per && mb + g < x.hp;
        Sums sum;
        sum.clear();
        if (mb > 0) {
            __syncthreads();   // the ring is free
            stage_rows(x, We, Wo, 0, mb, wm, ring);
            cp_commit();
            stage_rows(x, We, Wo, kRows, mb, wm, ring + stage);
            cp_commit();
        }
        for (int ch = 0; ch < chunks; ++ch) {
            cp_wait<1>();
            __syncthreads();
            stage_rows(x, We, Wo, (ch + 2) * kRows, mb, wm, ring + (ch + 2) % kStages * stage);
            cp_commit();
            if (!on) continue;
            const float* w = ring + ch % kStages * stage + odd * kRows * wm + g;
            const float* u = Uh + ch * kRows * TS;
            const int rows = min(kRows, x.hp - ch * kRows);   // a multiple of 8
            // the operands of row r + 1 are read while row r multiplies
            float a[2][8], v[2][8];
            auto fetch = [&](int r, int to) {
                *reinterpret_cast<float4*>(a[to]) = *reinterpret_cast<const float4*>(w + r * wm);
                *reinterpret_cast<float4*>(a[to] + 4) = *reinterpret_cast<const float4*>(w + r * wm + 4);
                *reinterpret_cast<float4*>(v[to]) = *reinterpret_cast<const float4*>(u + r * TS);
                *reinterpret_cast<float4*>(v[to] + 4) = *reinterpret_cast<const float4*>(u + r * TS + T / 2);
            };
            fetch(0, 0);
            for (int r = 0; r < rows; r += 8) {
#pragma unroll
                for (int q = 0; q < 8; ++q) {
                    if (q < 7) fetch(r + q + 1, (q + 1) & 1);
                    else if (r + 8 < rows) fetch(r + 8, 0);
                    sum.add(a[q & 1], v[q & 1]);
                }
            }
        }
        if (on) {
            float d[8][8];
            sum.get(d);
            scale(odd, mb + g, l0, d);
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                float* o = V + (odd * x.hp + mb + g + i) * TS + l0;
                *reinterpret_cast<float4*>(o) = make_float4(d[i][0], d[i][1], d[i][2], d[i][3]);
                *reinterpret_cast<float4*>(o + T / 2) = make_float4(d[i][4], d[i][5], d[i][6], d[i][7]);
            }
        }
    }
    cp_wait<0>();
    __syncthreads();
}
struct NoScale {
    __device__ __forceinline__ void operator()(int, int, int, float (&)[8][8]) const {}
};

// First address of line q of the lines along b (q = (a, c)) or a (q = (b, c)).
__device__ __forceinline__ long long line_start(const DirectShape& S, int axis, int q) {
    if (axis == 0) return q;
    const int a = q / S.n2;
    return (long long)a * S.n1 * S.n2 + (q - a * S.n2);
}

// MODE 0: forward along b. MODE 1: forward along a, division by the
// eigenvalue sum, back along a. MODE 2: back along b. In place on X.
template <int MODE, int T>
__global__ void __launch_bounds__(kThreads, 2) direct_cols_kernel(DirectShape S, float* X) {
    extern __shared__ __align__(16) float sm[];
    constexpr int kAxis = MODE == 1 ? 0 : 1;
    constexpr int kBatch = 8;                    // indices whose loads are in flight together
    constexpr int kStep = kThreads / T;          // indices the block loads at a time
    const DirectAxis& x = S.ax[kAxis];
    float* U = sm;
    float* V = U + 2 * x.hp * T;
    float* ring = V + 2 * x.hp * T;
    const float *we = MODE == 2 ? x.te : x.we, *wo = MODE == 2 ? x.to : x.wo;
    product_begin(x, we, wo, ring);
    pdl_wait();
    const int lines = kAxis == 0 ? S.n1 * S.n2 : S.n0 * S.n2;
    const long long stride = kAxis == 0 ? S.n1 * S.n2 : S.n2;
    const int l = threadIdx.x % T, first = threadIdx.x / T;
    const int q = blockIdx.x * T + l;
    float* line = X + line_start(S, kAxis, min(q, lines - 1));
    for (int p0 = first; p0 < x.hp; p0 += kBatch * kStep) {
        float a[kBatch], b[kBatch];
#pragma unroll
        for (int t = 0; t < kBatch; ++t) {
            const int p = p0 + t * kStep;
            int ja = p, jb = x.he + p;
            if (MODE != 2) fold_pair(x, p, ja, jb);
            a[t] = p < x.he ? line[ja * stride] : 0.0f;
            b[t] = p < x.np ? line[jb * stride] : 0.0f;
        }
#pragma unroll
        for (int t = 0; t < kBatch; ++t) {
            const int p = p0 + t * kStep;
            if (p >= x.hp) break;
            U[p * T + l] = MODE == 2 ? a[t] : a[t] + b[t];
            U[(x.hp + p) * T + l] = MODE == 2 ? b[t] : (p < x.np ? a[t] - b[t] : 0.0f);
        }
    }
    const float* out = V;
    if (MODE == 1) {
        product<T, T>(x, we, wo, U, V, ring, [&](int odd, int m0, int l0, float (&d)[8][8]) {
            float bc[8];
#pragma unroll
            for (int c = 0; c < 8; ++c) {
                const int r = min((int)blockIdx.x * T + l0 + (c & 3) + (c >> 2) * (T / 2), lines - 1);
                const int b = r / S.n2;
                bc[c] = S.ax[1].lam[b] + S.ax[2].lam[r - b * S.n2];
            }
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                const float la = m0 + i < (odd ? x.np : x.he) ? x.lam[odd * x.he + m0 + i] : 1.0f;
#pragma unroll
                for (int c = 0; c < 8; ++c) {
                    const float e = la + bc[c];   // zero only for the mean of an all-periodic box
                    d[i][c] = e > 0.0f ? d[i][c] / e : 0.0f;
                }
            }
        });
        product_begin(x, x.te, x.to, ring);
        product<T, T>(x, x.te, x.to, V, U, ring, NoScale{});
        out = U;
    } else {
        product<T, T>(x, we, wo, U, V, ring, NoScale{});
    }
    if (q >= lines) return;
    for (int p = first; p < x.he; p += kStep) {
        const float e = out[p * T + l], o = out[(x.hp + p) * T + l];
        int ja = p, jb = x.he + p;
        if (MODE != 0) fold_pair(x, p, ja, jb);
        line[ja * stride] = MODE == 0 || p >= x.np ? e : e + o;
        if (p < x.np) line[jb * stride] = MODE == 0 ? o : e - o;
    }
}

// Along the contiguous axis. BACK false: X = Q_c^T X in place. BACK true: the
// transform back, added to phi in FP64. Lines are rows (a, b); the tile is kept
// index by index like the other axes' (rows of T + 4 floats, so that a warp's
// consecutive indices of one line meet four to a bank).
template <bool BACK, int T>
__global__ void __launch_bounds__(kThreads, 2) direct_rows_kernel(DirectShape S, DirectOuter O, float* X, double* phi) {
    extern __shared__ __align__(16) float sm[];
    constexpr int TS = T + 4;
    constexpr int kBatch = T / kWarps < 4 ? T / kWarps : 4;
    static_assert(T % (kBatch * kWarps) == 0, "whole batches of lines");
    const DirectAxis& x = S.ax[2];
    float* U = sm;
    float* V = U + 2 * x.hp * TS;
    float* ring = V + 2 * x.hp * TS;
    const float *we = BACK ? x.te : x.we, *wo = BACK ? x.to : x.wo;
    product_begin(x, we, wo, ring);
    pdl_wait();
    const int lines = S.n0 * S.n1;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int row0 = blockIdx.x * T;
    for (int p = lane; p < x.hp; p += 32) {
        int ja = p, jb = x.he + p;
        if (!BACK) fold_pair(x, p, ja, jb);
        for (int m0 = warp; m0 < T; m0 += kBatch * kWarps) {
            float a[kBatch], b[kBatch];
#pragma unroll
            for (int t = 0; t < kBatch; ++t) {
                const float* v = X + (long long)min(row0 + m0 + t * kWarps, lines - 1) * x.n;
                a[t] = p < x.he ? v[ja] : 0.0f;
                b[t] = p < x.np ? v[jb] : 0.0f;
            }
#pragma unroll
            for (int t = 0; t < kBatch; ++t) {
                const int m = m0 + t * kWarps;
                U[p * TS + m] = BACK ? a[t] : a[t] + b[t];
                U[(x.hp + p) * TS + m] = BACK ? b[t] : (p < x.np ? a[t] - b[t] : 0.0f);
            }
        }
    }
    product<T, TS>(x, we, wo, U, V, ring, NoScale{});
    for (int p = lane; p < x.he; p += 32) {
        int ja = p, jb = x.he + p;
        if (BACK) fold_pair(x, p, ja, jb);
        const bool pair = p < x.np;
        for (int m0 = warp; m0 < T; m0 += kBatch * kWarps) {
            if (BACK) {
                double *out[kBatch], da[kBatch], db[kBatch];
#pragma unroll
                for (int t = 0; t < kBatch; ++t) {
                    const int row = min(row0 + m0 + t * kWarps, lines - 1), a = row / S.n1, b = row - a * S.n1;
                    out[t] = phi + ((long long)(a + O.o[0]) * O.cy + b + O.o[1]) * O.cz + O.o[2];
                    da[t] = out[t][ja];
                    db[t] = pair ? out[t][jb] : 0.0;
                }
#pragma unroll
                for (int t = 0; t < kBatch; ++t) {
                    const int m = m0 + t * kWarps;
                    if (row0 + m >= lines) break;
                    const float e = V[p * TS + m], o = V[(x.hp + p) * TS + m];
                    out[t][ja] = da[t] + (double)(pair ? e + o : e);
                    if (pair) out[t][jb] = db[t] + (double)(e - o);
                }
            } else {
#pragma unroll
                for (int t = 0; t < kBatch; ++t) {
                    const int m = m0 + t * kWarps;
                    if (row0 + m >= lines) break;
                    float* out = X + (long long)(row0 + m) * x.n;
                    out[p] = V[p * TS + m];
                    if (pair) out[x.he + p] = V[(x.hp + p) * TS + m];
                }
            }
        }
    }
}

__device__ __forceinline__ long long glue_at(const DirectOuter& O, int i, int j, int k) {
    return ((long long)i * O.cy + j) * O.cz + k;
}
__device__ __forceinline__ int wrap_node(int idx, int per, int nref) {
    if (per) { if (idx == 0) return nref; if (idx == nref + 1) return 1; }
    return idx;
}

// A thread's share of the residual's sums (rsum where every axis is periodic).
struct ResidualSums {
    double f2 = 0.0, r2 = 0.0, rsum = 0.0, worst = 0.0;
};

__device__ __forceinline__ double warp_sum(double v) {
    for (int o = 16; o; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
    return v;
}
__device__ __forceinline__ double warp_max(double v) {
    for (int o = 16; o; o >>= 1) { const double w = __shfl_down_sync(0xffffffffu, v, o); v = w > v ? w : v; }
    return v;
}

// Block totals of the sums in thread 0 (fixed order).
__device__ ResidualSums block_sums(ResidualSums s, bool allper) {
    __shared__ double red[4][kWarps];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    s.f2 = warp_sum(s.f2); s.r2 = warp_sum(s.r2); s.worst = warp_max(s.worst);
    if (allper) s.rsum = warp_sum(s.rsum);
    __syncthreads();
    if (lane == 0) { red[0][warp] = s.f2; red[1][warp] = s.r2; red[2][warp] = s.worst; red[3][warp] = s.rsum; }
    __syncthreads();
    if (threadIdx.x == 0)
        for (int w = 1; w < kWarps; ++w) {
            s.f2 += red[0][w]; s.r2 += red[1][w]; s.rsum += red[3][w];
            s.worst = red[2][w] > s.worst ? red[2][w] : s.worst;
        }
    return s;
}

// The end of a residual: the refinement's scalars, and with DIRECT_LOOP whether
// the graph's loop takes another correction (tolerance not met, cap not
// reached, residual finite). In an all-periodic box the mean of f, subtracted as a
// rounded number, leaves a constant of a rounding or so in f and in every r, which
// no phi can lower: it is taken out of both norms. And charge that differs from its
// mean by less than a rounding of the mean over the tolerance (1e-8 of it at 1e-8)
// is solved to that rounding instead: fm carries it.
__device__ void decide(const DirectStep& d, const DirectOuter& O, const ResidualSums& t, double fm) {
    double* red = d.sc->red;
    const double constant = O.allper ? t.rsum * t.rsum * O.inv_m : 0.0;
    const double r2 = t.r2 >= constant ? t.r2 - constant : (isfinite(t.r2) ? 0.0 : t.r2), worst = t.worst;
    const double res = sqrt(r2);
    if (d.mode & DIRECT_START) {
        red[6] = d.host->red[6];
        red[7] = d.host->red[7];
        double fn = sqrt(fmax(t.f2 - constant, 0.0));
        if (O.allper) fn = fmax(fn, 0x1p-53 * fabs(fm) * O.root_m / red[6]);
        red[5] = fn > 0.0 ? fn : 1.0;
        red[8] = 0.0;
        red[9] = res;
    } else {
        red[8] += 1.0;
    }
    red[2] = r2;
    d.sc->pointwise_bits = (unsigned long long)__double_as_longlong(worst);
    d.host->red[2] = r2;
    d.host->red[5] = red[5];
    d.host->red[8] = red[8];
    d.host->red[9] = red[9];
    if (d.mode & DIRECT_LOOP)
        cudaGraphSetConditional(d.loop, isfinite(res) && res > red[6] * red[5] && red[8] < red[7] ? 1u : 0u);
}

// X = f - A phi in FP64 (f = rho / eps0, less its mean when every axis is
// periodic), stored FP32, with the sums of f^2 and r^2 and
// RootGrid::checkPhiResidual's pointwise measure max |r / f|
// (src/Grid/RootGrid/RootGridField.cpp:267-317; a NaN stays out of the maximum).
// A block takes tiles of 32 unknowns along c, 8 rows b and kResA consecutive a,
// whose loads a thread issues together; L2-bound. The last block to finish
// totals the blocks' sums in their order and takes the refinement's decision.
constexpr int kResA = 4;
__global__ void __launch_bounds__(kThreads) direct_residual_kernel(DirectShape S, DirectOuter O,
                                                                   const double* __restrict__ rho0,
                                                                   const double* __restrict__ phi, float* X,
                                                                   double* partial, DirectStep step) {
    __shared__ int s_last;
    const int ntc = (S.n2 + 31) / 32, ntb = (S.n1 + 7) / 8, nta = (S.n0 + kResA - 1) / kResA;
    const int tiles = ntc * ntb * nta;
    const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
    pdl_wait();
    const double fm = O.allper ? step.sc->red[4] : 0.0;
    ResidualSums sums;
    for (int t = blockIdx.x; t < tiles; t += gridDim.x) {
        const int tc = t % ntc, rest = t / ntc, tb = rest % ntb, ta = rest / ntb;
        const int c = tc * 32 + tx, b = tb * 8 + ty;
        if (c >= S.n2 || b >= S.n1) continue;
        const int j = b + O.o[1], k = c + O.o[2];
        const int jm = wrap_node(j - 1, O.per[1], O.nref[1]), jp = wrap_node(j + 1, O.per[1], O.nref[1]);
        const int km = wrap_node(k - 1, O.per[2], O.nref[2]), kp = wrap_node(k + 1, O.per[2], O.nref[2]);
        double r[kResA], src[kResA];
#pragma unroll
        for (int e = 0; e < kResA; ++e) {
            const int i = min(ta * kResA + e, S.n0 - 1) + O.o[0];
            const int im = wrap_node(i - 1, O.per[0], O.nref[0]), ip = wrap_node(i + 1, O.per[0], O.nref[0]);
            // rho / eps0 as the reference rounds it: the product with the reciprocal, corrected once
            const double rho = rho0[glue_at(O, i, j, k)], q = rho * O.inv_eps0;
            src[e] = fma(fma(-q, O.eps0, rho), O.inv_eps0, q) - fm;
            const double op = phi[glue_at(O, im, j, k)] + phi[glue_at(O, ip, j, k)] + phi[glue_at(O, i, jm, k)] +
                              phi[glue_at(O, i, jp, k)] + phi[glue_at(O, i, j, km)] + phi[glue_at(O, i, j, kp)] -
                              6.0 * phi[glue_at(O, i, j, k)];
            r[e] = op + src[e];
        }
#pragma unroll
        for (int e = 0; e < kResA; ++e) {
            const int a = ta * kResA + e;
            if (a >= S.n0) break;
            X[((long long)a * S.n1 + b) * S.n2 + c] = (float)r[e];
            sums.f2 += src[e] * src[e];
            sums.r2 += r[e] * r[e];
            if (O.allper) sums.rsum += r[e];
            if (src[e] != 0.0 && fabs(r[e]) > sums.worst * fabs(src[e])) sums.worst = fmax(sums.worst, fabs(r[e] / src[e]));
        }
    }
    sums = block_sums(sums, O.allper);
    if (threadIdx.x == 0) {
        double* p = partial + kDirectPartials * (long long)blockIdx.x;
        p[0] = sums.f2; p[1] = sums.r2; p[2] = sums.worst; p[3] = sums.rsum;
        __threadfence();
        s_last = atomicInc(&step.sc->ticket, gridDim.x - 1) == gridDim.x - 1;
    }
    __syncthreads();
    if (!s_last) return;
    __threadfence();
    ResidualSums t;
    for (int b = threadIdx.x; b < (int)gridDim.x; b += blockDim.x) {
        const volatile double* p = partial + kDirectPartials * (long long)b;
        t.f2 += p[0]; t.r2 += p[1]; t.rsum += p[3];
        const double w = p[2];
        t.worst = w > t.worst ? w : t.worst;
    }
    t = block_sums(t, O.allper);
    if (threadIdx.x != 0) return;
    decide(step, O, t, fm);
}

size_t ring_smem(const DirectAxis& x) { return sizeof(float) * kStages * 2 * kRows * pass_modes(x.hp); }
size_t tile_smem(const DirectAxis& x, int row) { return sizeof(float) * 4 * x.hp * row + ring_smem(x); }
constexpr size_t kMostSmem = 224 * 1024;
// Lines of a tile: 64 while such CTAs give every SM one and fit its shared memory,
// else 32; 16 on axes (beyond 640 unknowns) of which 32 lines do not fit:
// 213 KB on the longest, 1020 unknowns, with a quarter of the threads multiplying.
int tile_lines(const DirectAxis& x, int lines, int pad) {
    if (lines >= 64 * 148 && tile_smem(x, 64 + pad) <= kMostSmem) return 64;
    return tile_smem(x, 32 + pad) <= kMostSmem ? 32 : 16;
}

// One axis' basis: folded index p (pairs, then self-mirrored ones) times mode
// (even modes, then odd ones), both halves padded to hp with zeros; the
// transposes for the way back.
void build_axis(DirectAxis& x, int n, int per) {
    x.n = n;
    x.per = per;
    x.np = per ? (n - 1) / 2 : n / 2;
    x.he = n - x.np;
    x.hp = (x.he + 7) / 8 * 8;
    const double pi = 3.14159265358979323846;
    std::vector<float> w(4 * (size_t)x.hp * x.hp, 0.0f), lam(n);
    float *we = w.data(), *wo = we + (size_t)x.hp * x.hp, *te = wo + (size_t)x.hp * x.hp, *to = te + (size_t)x.hp * x.hp;
    for (int m = 0; m < x.he; ++m) {
        // even mode m and odd mode m: their number along the axis
        const int ke = per ? m : 2 * m, ko = per ? m + 1 : 2 * m + 1;
        auto lambda = [&](int k) {
            const double s = per ? std::sin(pi * k / n) : std::sin(0.5 * pi * (k + 1) / (n + 1));
            return (float)(4.0 * s * s);
        };
        lam[m] = lambda(ke);
        if (m < x.np) lam[x.he + m] = lambda(ko);
        for (int p = 0; p < x.he; ++p) {
            int j;
            if (per) j = p < x.np ? p + 1 : (p == x.np ? 0 : n / 2);
            else j = p;
            double e, o;
            if (per) {
                const bool once = ke == 0 || 2 * ke == n;   // constant and alternating modes
                e = std::sqrt((once ? 1.0 : 2.0) / n) * std::cos(2.0 * pi * (double)(((long long)j * ke) % n) / n);
                o = std::sqrt(2.0 / n) * std::sin(2.0 * pi * (double)(((long long)j * ko) % n) / n);
            } else {
                const long long P = 2 * (n + 1);
                e = std::sqrt(2.0 / (n + 1)) * std::sin(pi * (double)(((long long)(j + 1) * (ke + 1)) % P) / (n + 1));
                o = std::sqrt(2.0 / (n + 1)) * std::sin(pi * (double)(((long long)(j + 1) * (ko + 1)) % P) / (n + 1));
            }
            we[(size_t)p * x.hp + m] = te[(size_t)m * x.hp + p] = (float)e;
            if (m < x.np && p < x.np) wo[(size_t)p * x.hp + m] = to[(size_t)m * x.hp + p] = (float)o;
        }
    }
    float* d = nullptr;
    FOPIS_CUDA(cudaMalloc(&d, sizeof(float) * (w.size() + lam.size())));
    x.we = d;
    x.wo = d + (size_t)x.hp * x.hp;
    x.te = d + 2 * (size_t)x.hp * x.hp;
    x.to = d + 3 * (size_t)x.hp * x.hp;
    x.lam = d + w.size();
    FOPIS_CUDA(cudaMemcpy(d, w.data(), sizeof(float) * w.size(), cudaMemcpyHostToDevice));
    FOPIS_CUDA(cudaMemcpy(d + w.size(), lam.data(), sizeof(float) * lam.size(), cudaMemcpyHostToDevice));
}

}  // namespace

bool direct_first(const int n[3]) { return n[0] <= kDirectMax && n[1] <= kDirectMax && n[2] <= kDirectMax; }

int direct_blocks(const int n[3]) {
    const long long tiles = (long long)((n[2] + 31) / 32) * ((n[1] + 7) / 8) * ((n[0] + kResA - 1) / kResA);
    return (int)std::min<long long>(tiles, 148 * 8);
}

namespace {
template <typename K>
void allow_smem(K* kernel) {
    FOPIS_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kMostSmem));
}
template <int T>
void allow_tile() {
    allow_smem(direct_cols_kernel<0, T>);
    allow_smem(direct_cols_kernel<1, T>);
    allow_smem(direct_cols_kernel<2, T>);
    allow_smem(direct_rows_kernel<false, T>);
    allow_smem(direct_rows_kernel<true, T>);
}
template <int MODE>
void launch_cols(const DirectShape& S, float* X, bool pdl, cudaStream_t st) {
    const DirectAxis& x = S.ax[MODE == 1 ? 0 : 1];
    const int lines = MODE == 1 ? S.n1 * S.n2 : S.n0 * S.n2, T = tile_lines(x, lines, 0);
    const dim3 grid((lines + T - 1) / T);
    auto* kernel = T == 64 ? direct_cols_kernel<MODE, 64> : (T == 32 ? direct_cols_kernel<MODE, 32> : direct_cols_kernel<MODE, 16>);
    launch_k(pdl, kernel, grid, dim3(kThreads), tile_smem(x, T), st, S, X);
}
template <bool BACK>
void launch_rows(const DirectShape& S, const DirectOuter& O, float* X, double* phi, bool pdl, cudaStream_t st) {
    const DirectAxis& x = S.ax[2];
    const int lines = S.n0 * S.n1, T = tile_lines(x, lines, 4);
    const dim3 grid((lines + T - 1) / T);
    auto* kernel = T == 64 ? direct_rows_kernel<BACK, 64> : (T == 32 ? direct_rows_kernel<BACK, 32> : direct_rows_kernel<BACK, 16>);
    launch_k(pdl, kernel, grid, dim3(kThreads), tile_smem(x, T + 4), st, S, O, X, phi);
}
}  // namespace

void direct_setup(DirectShape& S, const int n[3], const int per[3]) {
    S.n0 = n[0]; S.n1 = n[1]; S.n2 = n[2];
    for (int a = 0; a < 3; ++a) build_axis(S.ax[a], n[a], per[a]);
    // the attribute belongs to the function, which contexts of other sizes share
    allow_tile<64>();
    allow_tile<32>();
    for (const auto& x : S.ax)
        if (tile_smem(x, 32 + 4) > kMostSmem) { allow_tile<16>(); break; }
}

void direct_free(DirectShape& S) {
    for (auto& x : S.ax) {
        if (x.we) cudaFree(const_cast<float*>(x.we));
        x = DirectAxis{};
    }
}

// X = f - A phi and the decision of `step`.
int direct_residual(const DirectShape& S, const DirectOuter& O, const double* rho0, const double* phi, float* X,
                    double* partial, const DirectStep& step, bool pdl, cudaStream_t st) {
    const int n[3] = {S.n0, S.n1, S.n2};
    launch_k(pdl, direct_residual_kernel, dim3(direct_blocks(n)), dim3(kThreads), 0, st, S, O, rho0, phi, X, partial, step);
    return 1;
}

// phi += A^-1 X.
int direct_correct(const DirectShape& S, const DirectOuter& O, float* X, double* phi, bool pdl, cudaStream_t st) {
    launch_rows<false>(S, O, X, phi, pdl, st);
    launch_cols<0>(S, X, pdl, st);
    launch_cols<1>(S, X, pdl, st);
    launch_cols<2>(S, X, pdl, st);
    launch_rows<true>(S, O, X, phi, pdl, st);
    return 5;
}

}  // namespace fopis
