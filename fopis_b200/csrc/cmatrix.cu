// cmatrix.cu — conductors: surface-node maps, the capacity matrix and the
// per-step equipotential correction.
//
// Capacity matrix (RootGrid::initializeObjectsCmatrix, RootGridObject.cpp:77-148):
// column c of B holds phi at every surface node for rho = 1 at surface node c:
// values of the grid's Green's function, from one table over node differences
// and sums (one solve per column where the table takes more than 4 GiB or cannot
// be allocated); C = B^-1 by blocked in-place Gauss-Jordan
// elimination in FP64 on the device (B is symmetric positive definite, so no
// pivoting). Per step (Spacecraft::redistributeChargeForPerfectConductor,
// Spacecraft.cpp:708-758): V = (sum_ij C_ij phi_j + Q) / sum_ij C_ij, or the
// fixed potential, then rho0[node_i] += sum_j C_ij (V - phi_j).
#include "internal.cuh"

#include <algorithm>
#include <cmath>
#include <cstring>

namespace fopis {

namespace {

constexpr int kT = 256;

__device__ __forceinline__ double wsum(double v) {
    for (int o = 16; o; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
    return v;
}
__device__ double bsum(double v) {
    __shared__ double red[32];
    v = wsum(v);
    const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
    __syncthreads();
    if (l == 0) red[w] = v;
    __syncthreads();
    v = 0.0;
    if (w == 0) {
        v = (l < (int)(blockDim.x >> 5)) ? red[l] : 0.0;
        v = wsum(v);
    }
    return v;
}

__global__ void gather_kernel(const double* phi, const int32_t* nodes, int n, double* out) {
    for (int t = blockIdx.x * blockDim.x + threadIdx.x; t < n; t += gridDim.x * blockDim.x) out[t] = phi[nodes[t]];
}

__global__ void set_node_kernel(double* a, long long idx, double v) { a[idx] = v; }

// Green's function of the 7-point operator with the solve's closure. Along an
// axis between held faces the eigenvectors are sines, and a product of two is
// half a difference of cosines of the node difference and the node sum; along a
// periodic axis only the difference enters. So phi at node r for a charge at
// node c is a signed sum of at most eight entries of
//   T[u][v][w] = sum_klm Ca[k][u] Cb[l][v] Cc[m][w] / (lambda_k + lambda_l + lambda_m)
// over the offsets u, v, w the surface has (differences, then sums), three small
// FP64 contractions. The mean mode of an all-periodic box is left out, as the
// solve leaves it out. With the inverse, 47^3 unknowns and 218 nodes: 190 ms by
// V-cycles, 29 ms by direct corrections, 0.5 ms this way; 255^3 and 3586 nodes:
// 27 s by V-cycles, 16 ms this way.
struct GreenAxis {
    int n, per;      // unknowns, periodic
    int lo, span;    // smallest 1-based unknown of the surface, largest minus smallest
    int count;       // offsets: span + 1 differences, then 2 span + 1 sums between held faces
    double* cosines; // [n][count]
    double* lambda;  // [n]
};

__global__ void green_axis_kernel(GreenAxis x) {
    for (int t = blockIdx.x * blockDim.x + threadIdx.x; t < x.n * x.count; t += gridDim.x * blockDim.x) {
        const int k = t / x.count, u = t - k * x.count;
        const int offset = u <= x.span ? u : 2 * x.lo + (u - x.span - 1);
        if (x.per) {
            x.cosines[t] = cospi(2.0 * (double)(((long long)offset * k) % x.n) / x.n) / x.n;
            if (u == 0) { const double q = sinpi((double)k / x.n); x.lambda[k] = 4.0 * q * q; }
        } else {
            x.cosines[t] = cospi((double)(((long long)offset * (k + 1)) % (2 * (x.n + 1))) / (x.n + 1)) / (x.n + 1);
            if (u == 0) { const double q = sinpi(0.5 * (k + 1) / (x.n + 1)); x.lambda[k] = 4.0 * q * q; }
        }
    }
}

// R[k][l][w] = sum_m Cc[m][w] / (lambda_k + lambda_l + lambda_m): kGreenL values
// of l per CTA share the reads of Cc.
constexpr int kGreenL = 4, kGreenThreads = 128;
__global__ void __launch_bounds__(kGreenThreads) green_sum_kernel(GreenAxis a, GreenAxis b, GreenAxis c, double* R) {
    extern __shared__ double inv[];   // [kGreenL][c.n]
    const int k = blockIdx.y, l0 = blockIdx.x * kGreenL;
    for (int t = threadIdx.x; t < kGreenL * c.n; t += kGreenThreads) {
        const int l = min(l0 + t / c.n, b.n - 1);
        const double e = a.lambda[k] + b.lambda[l] + c.lambda[t % c.n];
        inv[t] = e > 0.0 ? 1.0 / e : 0.0;
    }
    __syncthreads();
    for (int w = threadIdx.x; w < c.count; w += kGreenThreads) {
        double s[kGreenL] = {};
#pragma unroll 4
        for (int m = 0; m < c.n; ++m) {
            const double q = c.cosines[(long long)m * c.count + w];
#pragma unroll
            for (int e = 0; e < kGreenL; ++e) s[e] += q * inv[e * c.n + m];
        }
        for (int e = 0; e < kGreenL && l0 + e < b.n; ++e) R[((long long)k * b.n + l0 + e) * c.count + w] = s[e];
    }
}

// out[o][u][q] = sum_k C[k][u] in[o][k][q]: one axis' contraction, q of the
// `inner` trailing values per thread, kGreenU offsets u of it.
constexpr int kGreenU = 4;
__global__ void __launch_bounds__(kGreenThreads) green_contract_kernel(GreenAxis x, const double* in, int inner,
                                                                       double* out) {
    const int q = blockIdx.x * kGreenThreads + threadIdx.x, u0 = blockIdx.y * kGreenU;
    if (q >= inner) return;
    in += (long long)blockIdx.z * x.n * inner + q;
    double s[kGreenU] = {};
#pragma unroll 4
    for (int k = 0; k < x.n; ++k) {
        const double v = in[(long long)k * inner];
#pragma unroll
        for (int e = 0; e < kGreenU; ++e) s[e] += x.cosines[(long long)k * x.count + min(u0 + e, x.count - 1)] * v;
    }
    for (int e = 0; e < kGreenU && u0 + e < x.count; ++e)
        out[((long long)blockIdx.z * x.count + u0 + e) * inner + q] = s[e];
}

// B from the table; u: the surface nodes' 1-based unknowns per axis, [3][n].
__global__ void green_matrix_kernel(GreenAxis a, GreenAxis b, GreenAxis c, const double* T, const int32_t* u, int n,
                                    double inv_eps0, double* B) {
    const GreenAxis ax[3] = {a, b, c};
    const long long total = (long long)n * n;
    for (long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x; t < total; t += (long long)gridDim.x * blockDim.x) {
        const int i = (int)(t / n), j = (int)(t % n);
        int diff[3], sum[3];
#pragma unroll
        for (int d = 0; d < 3; ++d) {
            const int p = u[d * n + i], q = u[d * n + j];
            diff[d] = abs(p - q);
            sum[d] = ax[d].span + 1 + p + q - 2 * ax[d].lo;
        }
        double v = 0.0;
        for (int x = 0; x < (a.per ? 1 : 2); ++x)
            for (int y = 0; y < (b.per ? 1 : 2); ++y)
                for (int z = 0; z < (c.per ? 1 : 2); ++z) {
                    const double g = T[((long long)(x ? sum[0] : diff[0]) * b.count + (y ? sum[1] : diff[1])) * c.count +
                                       (z ? sum[2] : diff[2])];
                    v += (x + y + z) & 1 ? -g : g;
                }
        B[t] = v * inv_eps0;
    }
}

// Blocked in-place Gauss-Jordan inversion without pivoting, kGj pivots a step:
// with K the pivots' rows and columns, D = A_KK, the row panel becomes R = D^-1
// A_K (its own columns D^-1), every other row A_i -= A_iK R (its own columns
// starting from zero). One pass over the matrix per 32 pivots instead of one per
// pivot. panel: R into `row`, A_:K into `col` ([n][kGj]); every CTA inverts D.
constexpr int kGj = 32, kGjTile = 64;
__global__ void __launch_bounds__(256) gj_panel_kernel(const double* A, int n, int k0, double* row, double* col,
                                                       unsigned* bad) {
    __shared__ double D[kGj][kGj + 1], pivot_row[kGj], pivot_col[kGj];
    const int nb = min(kGj, n - k0), tid = threadIdx.x;
    for (int t = tid; t < kGj * kGj; t += 256) {
        const int i = t / kGj, j = t % kGj;
        D[i][j] = i < nb && j < nb ? A[(long long)(k0 + i) * n + k0 + j] : (i == j ? 1.0 : 0.0);
    }
    __syncthreads();
    for (int k = 0; k < nb; ++k) {
        if (tid < kGj) { pivot_row[tid] = D[k][tid]; pivot_col[tid] = D[tid][k]; }
        __syncthreads();
        const double akk = pivot_row[k], p = 1.0 / akk;
        if (blockIdx.x == 0 && tid == 0 && !(akk > 0.0)) atomicOr(bad, 1u);
        for (int t = tid; t < kGj * kGj; t += 256) {
            const int i = t / kGj, j = t % kGj;
            D[i][j] = i == k ? (j == k ? p : pivot_row[j] * p)
                             : (j == k ? -pivot_col[i] * p : D[i][j] - pivot_col[i] * pivot_row[j] * p);
        }
        __syncthreads();
    }
    for (int j = blockIdx.x * 256 + tid; j < n; j += gridDim.x * 256) {
        double a[kGj];
#pragma unroll
        for (int q = 0; q < kGj; ++q) a[q] = q < nb ? A[(long long)(k0 + q) * n + j] : 0.0;
        const int own = j - k0;
        for (int i = 0; i < nb; ++i) {
            double s = 0.0;
#pragma unroll
            for (int q = 0; q < kGj; ++q) s += D[i][q] * a[q];
            row[(long long)i * n + j] = own >= 0 && own < nb ? D[i][own] : s;
        }
#pragma unroll
        for (int q = 0; q < kGj; ++q) col[(long long)j * kGj + q] = q < nb ? A[(long long)j * n + k0 + q] : 0.0;
    }
}
__global__ void __launch_bounds__(256) gj_update_kernel(double* A, int n, int k0, const double* row, const double* col) {
    __shared__ double R[kGj][kGjTile], C[kGjTile][kGj + 1];
    const int nb = min(kGj, n - k0), tid = threadIdx.x;
    const int i0 = blockIdx.y * kGjTile, j0 = blockIdx.x * kGjTile;
    for (int t = tid; t < kGj * kGjTile; t += 256) {
        const int q = t / kGjTile, j = j0 + t % kGjTile;
        R[q][t % kGjTile] = q < nb && j < n ? row[(long long)q * n + j] : 0.0;
        const int i = i0 + t / kGj;
        C[t / kGj][t % kGj] = i < n ? col[(long long)i * kGj + t % kGj] : 0.0;
    }
    __syncthreads();
    const int tx = tid & 15, ty = tid >> 4;   // columns tx + 16 q, rows ty + 16 p
    double s[4][4] = {};
    for (int q = 0; q < nb; ++q) {
        double c[4], r[4];
#pragma unroll
        for (int e = 0; e < 4; ++e) { c[e] = C[ty + 16 * e][q]; r[e] = R[q][tx + 16 * e]; }
#pragma unroll
        for (int x = 0; x < 4; ++x)
#pragma unroll
            for (int y = 0; y < 4; ++y) s[x][y] += c[x] * r[y];
    }
#pragma unroll
    for (int x = 0; x < 4; ++x)
#pragma unroll
        for (int y = 0; y < 4; ++y) {
            const int i = i0 + ty + 16 * x, j = j0 + tx + 16 * y;
            if (i >= n || j >= n) continue;
            double* v = A + (long long)i * n + j;
            if (i >= k0 && i < k0 + nb) *v = R[i - k0][tx + 16 * y];
            else *v = (j >= k0 && j < k0 + nb ? 0.0 : *v) - s[x][y];
        }
}

// colsum_j = sum_i C_ij; scal[3] = sum_ij C_ij (Cmatrix::total, Cmatrix.hpp:36-44).
__global__ void colsum_kernel(const double* C, int n, double* colsum) {
    for (int j = blockIdx.x * blockDim.x + threadIdx.x; j < n; j += gridDim.x * blockDim.x) {
        double s = 0.0;
        for (int i = 0; i < n; ++i) s += C[(long long)i * n + j];
        colsum[j] = s;
    }
}
__global__ void total_kernel(const double* colsum, int n, double* out) {
    double s = 0.0;
    for (int t = threadIdx.x; t < n; t += blockDim.x) s += colsum[t];
    s = bsum(s);
    if (threadIdx.x == 0) *out = s;
}

// Spacecraft::initializeChargeMapOffset (Spacecraft.cpp:160-183):
// charge_map[0][i] += sum_j C_ij * offset.
__global__ void offset_kernel(const double* C, int n, double offset, double* charge_map) {
    const int warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
    const int nw = (gridDim.x * blockDim.x) >> 5;
    for (int i = warp; i < n; i += nw) {
        double s = 0.0;
        for (int j = lane; j < n; j += 32) s += C[(long long)i * n + j] * offset;
        s = wsum(s);
        if (lane == 0) charge_map[i] += s;
    }
}

// Spacecraft::sumWholeCharge (Spacecraft.cpp:615-626) for the fixed-point
// temporary map, then the total charge (getTotalCharge, :248-259) into scal[1].
__global__ void sum_charge_kernel(long long* tmp, double* map, int nsp, int n, const double* scale, double* scal) {
    double q = 0.0;
    for (int t = threadIdx.x; t < nsp * n; t += blockDim.x) {
        const int s = t / n;
        const long long v = tmp[t];
        if (v) { map[t] += scale[s] * (double)v; tmp[t] = 0; }
        q += map[t];
    }
    q = bsum(q);
    if (threadIdx.x == 0) scal[1] = q;
}

// V of the perfect conductor into scal[0]; scal[2] = sum_j colsum_j phi_j.
// On a dielectric surface (Spacecraft::redistributeChargeForDielectric,
// Spacecraft.cpp:641-706) every node with a capacitance sees phi_j - Q_j / c_j,
// Q_j its accumulated charge over the species: the same formulas then give V
// and delta rho, so phis holds that effective potential.
__global__ void potential_kernel(const double* phi, const int32_t* nodes, const double* colsum, int n, double total,
                                 int fixed, double fixedV, double* phis, double* scal, const double* cap,
                                 const double* charge_map, int nsp) {
    double s = 0.0;
    for (int j = threadIdx.x; j < n; j += blockDim.x) {
        double p = phi[nodes[j]];
        if (cap && cap[j] > 0.0) {
            double q = 0.0;
            for (int sp = 0; sp < nsp; ++sp) q += charge_map[(long long)sp * n + j];
            p -= q / cap[j];
        }
        phis[j] = p;
        s += colsum[j] * p;
    }
    s = bsum(s);
    if (threadIdx.x == 0) {
        scal[2] = s;
        scal[0] = fixed ? fixedV : (s + scal[1]) / total;
    }
}

// delta rho_i = sum_j C_ij (V - phi_j), added to rho0 at surface node i and
// kept in drho_out for the start of the second solve.
__global__ void drho_kernel(const double* C, int n, const double* phis, const double* scal, const int32_t* nodes,
                            double* rho0, double* drho_out) {
    const int warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
    const int nw = (gridDim.x * blockDim.x) >> 5;
    const double V = scal[0];
    for (int i = warp; i < n; i += nw) {
        double s = 0.0;
        const double* row = C + (long long)i * n;
        for (int j = lane; j < n; j += 32) s += row[j] * (V - phis[j]);
        s = wsum(s);
        if (lane == 0) { rho0[nodes[i]] += s; drho_out[i] = s; }
    }
}

// Start of the second solve: this step's redistributed charge d0 fitted in
// least squares by the two previous steps' (d1, d2) over the surface nodes of
// every object; the coefficients scale the conductor responses those charges
// produced. One term while only one response is recorded, and alpha = 1 (the
// previous response as it is) when the fit is degenerate.
struct ConductorFit {
    int nobj;
    int terms;
    const double* d0[FOPIS_MAX_OBJECTS];
    const double* d1[FOPIS_MAX_OBJECTS];
    const double* d2[FOPIS_MAX_OBJECTS];
    int n[FOPIS_MAX_OBJECTS];
};

__global__ void conductor_fit_kernel(ConductorFit f, double* alpha) {
    double s11 = 0.0, s12 = 0.0, s22 = 0.0, b1 = 0.0, b2 = 0.0;
    for (int o = 0; o < f.nobj; ++o)
        for (int i = threadIdx.x; i < f.n[o]; i += blockDim.x) {
            const double x0 = f.d0[o][i], x1 = f.d1[o][i], x2 = f.terms > 1 ? f.d2[o][i] : 0.0;
            s11 += x1 * x1; s12 += x1 * x2; s22 += x2 * x2; b1 += x0 * x1; b2 += x0 * x2;
        }
    s11 = bsum(s11); s12 = bsum(s12); s22 = bsum(s22); b1 = bsum(b1); b2 = bsum(b2);
    if (threadIdx.x == 0) {
        double a1 = 1.0, a2 = 0.0;
        const double det = s11 * s22 - s12 * s12;
        if (f.terms > 1 && det > 1e-10 * s11 * s22) {
            a1 = (b1 * s22 - b2 * s12) / det;
            a2 = (b2 * s11 - b1 * s12) / det;
        } else if (s11 > 0.0) {
            a1 = b1 / s11;
        }
        alpha[0] = a1;
        alpha[1] = a2;
    }
}

__global__ void conductor_start_kernel(double* phi, const double* r1, const double* r2, const double* alpha,
                                       long long N) {
    const double a1 = alpha[0], a2 = alpha[1];
    for (long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x; t < N; t += (long long)gridDim.x * blockDim.x)
        phi[t] += a1 * r1[t] + (a2 != 0.0 ? a2 * r2[t] : 0.0);
}

// Spacecraft::is{X,Y,Z}surfacePoint at an integer node (dx1 = 0), host side.
struct HostObj {
    const Ctx* c;
    std::vector<uint8_t> cells;   // [nx+1][ny+1][nz+1]
    std::vector<int32_t> node_cmat;
    bool valid_cell(int i, int j, int k) const {
        return i >= 0 && i < c->nx + 1 && j >= 0 && j < c->ny + 1 && k >= 0 && k < c->nz + 1;
    }
    bool in(int i, int j, int k) const {
        if (!valid_cell(i, j, k)) return false;
        return cells[((size_t)i * (c->ny + 1) + j) * (c->nz + 1) + k] != 0;
    }
    bool is_cmat(int i, int j, int k) const {
        if (i < 0 || j < 0 || k < 0 || i >= c->cx || j >= c->cy || k >= c->cz) return false;
        return node_cmat[((size_t)i * c->cy + j) * c->cz + k] >= 0;
    }
    bool surface_point(int ax, int i, int j, int k, int sign) const {
        const int di = ax == 0, dj = ax == 1, dk = ax == 2;
        if (valid_cell(i, j, k) && valid_cell(i - di, j - dj, k - dk)) {
            const bool here = in(i, j, k), below = in(i - di, j - dj, k - dk);
            return sign > 0 ? (here && !below) : (!here && below);
        }
        if (ax == 0) return is_cmat(i, j, k) && is_cmat(i, j + 1, k) && is_cmat(i, j, k + 1) && is_cmat(i, j + 1, k + 1);
        if (ax == 1) return is_cmat(i, j, k) && is_cmat(i + 1, j, k) && is_cmat(i, j, k + 1) && is_cmat(i + 1, j, k + 1);
        return is_cmat(i, j, k) && is_cmat(i + 1, j, k) && is_cmat(i, j + 1, k) && is_cmat(i + 1, j + 1, k);
    }
};

// A buffer of the context's stream, given back in its order.
template <typename T>
struct StreamBuffer {
    Ctx& c;
    T* p = nullptr;
    explicit StreamBuffer(Ctx& x) : c(x) {}
    ~StreamBuffer() { if (p) cudaFreeAsync(p, c.st); }
    bool alloc(size_t n) {
        if (cudaMallocAsync((void**)&p, sizeof(T) * n, c.st) == cudaSuccess) return true;
        cudaGetLastError();
        p = nullptr;
        return false;
    }
};

int grid1(long long n) { return (int)std::max<long long>(1, std::min<long long>((n + kT - 1) / kT, 148LL * 16)); }

}  // namespace

void object_upload(Ctx& c, ObjectDev& o, const fopis_object_desc* d, int id) {
    if (d->n_cmat <= 0 || d->n_cmat >= (1 << 24)) throw ApiError{FOPIS_ERR_ARG, "n_cmat out of range"};
    o.n = d->n_cmat;
    o.nodes_ijk.assign(d->cmat_nodes, d->cmat_nodes + 3 * (size_t)o.n);
    HostObj h;
    h.c = &c;
    h.cells.assign((size_t)(c.nx + 1) * (c.ny + 1) * (c.nz + 1), 0);
    std::vector<int32_t> lin(o.n);
    std::vector<int32_t> ncm(c.N);
    FOPIS_CUDA(cudaMemcpy(ncm.data(), c.node_cmat, sizeof(int32_t) * c.N, cudaMemcpyDeviceToHost));
    h.node_cmat.assign(c.N, -1);
    for (int m = 0; m < o.n; ++m) {
        const int i = d->cmat_nodes[3 * m], j = d->cmat_nodes[3 * m + 1], k = d->cmat_nodes[3 * m + 2];
        if (i < 0 || j < 0 || k < 0 || i >= c.cx || j >= c.cy || k >= c.cz)
            throw ApiError{FOPIS_ERR_ARG, "surface node outside the grid"};
        const size_t L = ((size_t)i * c.cy + j) * c.cz + k;
        if (ncm[L] >= 0) throw ApiError{FOPIS_ERR_ARG, "surface node shared by two objects"};
        ncm[L] = (id << 24) | m;
        h.node_cmat[L] = m;
        lin[m] = (int32_t)L;
    }
    std::vector<uint8_t> cmap(c.N);
    FOPIS_CUDA(cudaMemcpy(cmap.data(), c.cellmap, c.N, cudaMemcpyDeviceToHost));
    for (int m = 0; m < d->n_cells; ++m) {
        const int i = d->cells[3 * m], j = d->cells[3 * m + 1], k = d->cells[3 * m + 2];
        if (i < 0 || j < 0 || k < 0 || i > c.nx || j > c.ny || k > c.nz) throw ApiError{FOPIS_ERR_ARG, "cell outside the grid"};
        cmap[((size_t)i * c.cy + j) * c.cz + k] = (uint8_t)(id + 1);
        h.cells[((size_t)i * (c.ny + 1) + j) * (c.nz + 1) + k] = 1;
    }
    // in the order of c.st, which a plain copy is not ordered with: it may return before
    // its last piece is on the device, and the marks are read from the map only here
    copy_to_device(c, c.node_cmat, ncm.data(), sizeof(int32_t) * c.N);
    copy_to_device(c, c.cellmap, cmap.data(), c.N);
    mark_brick_bodies(c);
    FOPIS_CUDA(cudaMalloc(&o.nodes, sizeof(int32_t) * o.n));
    copy_to_device(c, o.nodes, lin.data(), sizeof(int32_t) * o.n);
    FOPIS_CUDA(cudaMalloc(&o.C, sizeof(double) * (size_t)o.n * o.n));
    FOPIS_CUDA(cudaMalloc(&o.colsum, sizeof(double) * o.n));
    FOPIS_CUDA(cudaMalloc(&o.charge_tmp, sizeof(long long) * (size_t)c.nsp * o.n));
    FOPIS_CUDA(cudaMalloc(&o.charge_map, sizeof(double) * (size_t)c.nsp * o.n));
    FOPIS_CUDA(cudaMalloc(&o.phis, sizeof(double) * o.n));
    FOPIS_CUDA(cudaMalloc(&o.drho_buf, sizeof(double) * 3 * o.n));
    FOPIS_CUDA(cudaMemsetAsync(o.drho_buf, 0, sizeof(double) * 3 * o.n, c.st));
    for (int q = 0; q < 3; ++q) o.drho[q] = o.drho_buf + (size_t)q * o.n;
    FOPIS_CUDA(cudaMalloc(&o.scal, sizeof(double) * 8));
    FOPIS_CUDA(cudaMemsetAsync(o.charge_tmp, 0, sizeof(long long) * (size_t)c.nsp * o.n, c.st));
    FOPIS_CUDA(cudaMemsetAsync(o.charge_map, 0, sizeof(double) * (size_t)c.nsp * o.n, c.st));
    FOPIS_CUDA(cudaMemsetAsync(o.scal, 0, sizeof(double) * 8, c.st));
    o.is_fixed = d->is_potential_fixed;
    o.fixed_potential = d->fixed_potential;
    o.offset = d->initial_potential_offset;
    o.emit_species = d->emit_species;
    o.secondary_species = -1;
    if (d->secondary_species >= 0) {
        if (d->secondary_species >= c.nsp || c.p.species[d->secondary_species].kind != FOPIS_SPECIES_SECONDARY)
            throw ApiError{FOPIS_ERR_ARG, "secondary_species must name a species of kind FOPIS_SPECIES_SECONDARY"};
        if (!(c.p.energy_ev > 0.0)) throw ApiError{FOPIS_ERR_ARG, "secondary emission needs params.energy_ev"};
        o.secondary_species = d->secondary_species;
        if (c.inc.cap == 0) {   // one incident list per context, as long as the absorbed list
            c.inc.cap = c.ab.cap;
            double** fl[7] = {&c.inc.x, &c.inc.y, &c.inc.z, &c.inc.vx, &c.inc.vy, &c.inc.vz, &c.inc.trem};
            for (auto* q : fl) FOPIS_CUDA(cudaMalloc(q, sizeof(double) * c.inc.cap));
            FOPIS_CUDA(cudaMalloc(&c.inc.species, c.inc.cap));
            FOPIS_CUDA(cudaMalloc(&c.inc.object, c.inc.cap));
            FOPIS_CUDA(cudaMalloc(&c.inc.axis, c.inc.cap));
            FOPIS_CUDA(cudaMalloc(&c.inc.count, sizeof(int32_t) * c.inc.cap));
        }
    }
    o.dielectric = d->dielectric ? 1 : 0;
    if (o.dielectric) {
        if (!d->capacitance) throw ApiError{FOPIS_ERR_ARG, "a dielectric surface needs its node capacitances"};
        FOPIS_CUDA(cudaMalloc(&o.capacitance, sizeof(double) * o.n));
        copy_to_device(c, o.capacitance, d->capacitance, sizeof(double) * o.n);
    }
    // lit nodes of the emitting face (Spacecraft::emitParticles, Spacecraft.cpp:836-886)
    std::vector<int32_t> lit, lit_ijk;
    if (o.emit_species >= 0 && o.emit_species < c.nsp &&
        c.p.species[o.emit_species].kind == FOPIS_SPECIES_PHOTOELECTRON) {
        int eaxis = -1;
        for (int q = 0; q < 3; ++q) if (std::fabs(c.p.shine_vector[q]) == 1.0) { eaxis = q; break; }
        if (eaxis >= 0) {
            const int sign = c.p.shine_vector[eaxis] > 0.0 ? 1 : -1;
            for (int m = 0; m < o.n; ++m) {
                const int i = d->cmat_nodes[3 * m], j = d->cmat_nodes[3 * m + 1], k = d->cmat_nodes[3 * m + 2];
                if (h.surface_point(eaxis, i, j, k, sign)) {
                    lit.push_back(m);
                    lit_ijk.push_back((i << 20) | (j << 10) | k);
                }
            }
        }
    }
    o.n_lit = (int)lit.size();
    if (o.n_lit) {
        FOPIS_CUDA(cudaMalloc(&o.lit, sizeof(int32_t) * 2 * o.n_lit));
        copy_to_device(c, o.lit, lit.data(), sizeof(int32_t) * o.n_lit);
        copy_to_device(c, o.lit + o.n_lit, lit_ijk.data(), sizeof(int32_t) * o.n_lit);
    }
}

static void finish_C(Ctx& c, ObjectDev& o) {
    ++c.launches;
    colsum_kernel<<<grid1(o.n), kT, 0, c.st>>>(o.C, o.n, o.colsum);
    ++c.launches;
    total_kernel<<<1, 1024, 0, c.st>>>(o.colsum, o.n, o.scal + 3);
    FOPIS_LAUNCH_CHECK();
    double tot = 0.0;
    FOPIS_CUDA(cudaMemcpyAsync(&tot, o.scal + 3, sizeof(double), cudaMemcpyDeviceToHost, c.st));
    FOPIS_CUDA(cudaStreamSynchronize(c.st));
    o.total = tot;
    o.has_C = true;
    if (o.offset != 0.0) {
        o.potential = o.offset;
        ++c.launches;
        offset_kernel<<<grid1((long long)o.n * 32), kT, 0, c.st>>>(o.C, o.n, o.offset, o.charge_map);
        FOPIS_LAUNCH_CHECK();
    }
}

// B of an object from the table; false where the table does not fit. A surface
// node that is no unknown of the Poisson solve (it lies on a face or beyond) takes
// no charge: its column of B is zero.
static bool green_matrix(Ctx& c, const ObjectDev& o, double* B) {
    const MGLevel& m = c.mg[0];
    GreenAxis ax[3];
    std::vector<int32_t> u(3 * (size_t)o.n);
    for (int d = 0; d < 3; ++d) {
        const int first = m.per[d] ? 1 : 2;   // glue index of the first unknown
        int lo = 1 << 30, hi = 0;
        for (int t = 0; t < o.n; ++t) {
            const int q = o.nodes_ijk[3 * (size_t)t + d] - first + 1;
            if (q < 1 || q > m.n[d])
                throw ApiError{FOPIS_ERR_DEVICE, "capacity matrix B is not positive definite: a surface node is on a face"};
            u[(size_t)d * o.n + t] = q;
            lo = std::min(lo, q);
            hi = std::max(hi, q);
        }
        const int span = hi - lo;
        ax[d] = GreenAxis{m.n[d], m.per[d], lo, span, m.per[d] ? span + 1 : 3 * span + 2, nullptr, nullptr};
    }
    const size_t first = (size_t)ax[0].n * ax[1].n * ax[2].count, second = (size_t)ax[0].n * ax[1].count * ax[2].count;
    const size_t third = (size_t)ax[0].count * ax[1].count * ax[2].count;
    size_t tables = 0;
    for (const auto& x : ax) tables += (size_t)x.n * (x.count + 1);
    const size_t doubles = tables + first + second + third;
    if (doubles > (size_t)1 << 29) return false;   // 4 GiB
    StreamBuffer<double> pool(c);
    StreamBuffer<int32_t> du(c);
    if (!pool.alloc(doubles) || !du.alloc(u.size())) return false;
    FOPIS_CUDA(cudaMemcpyAsync(du.p, u.data(), sizeof(int32_t) * u.size(), cudaMemcpyHostToDevice, c.st));
    double* next = pool.p;
    for (auto& x : ax) {
        x.cosines = next;
        x.lambda = next + (size_t)x.n * x.count;
        next = x.lambda + x.n;
        ++c.launches;
        green_axis_kernel<<<grid1((long long)x.n * x.count), kT, 0, c.st>>>(x);
    }
    double *R1 = next, *R2 = R1 + first, *T = R2 + second;
    c.launches += 4;
    green_sum_kernel<<<dim3((ax[1].n + kGreenL - 1) / kGreenL, ax[0].n), kGreenThreads, sizeof(double) * kGreenL * ax[2].n,
                       c.st>>>(ax[0], ax[1], ax[2], R1);
    auto contract = [&](const GreenAxis& x, const double* in, int inner, int outer, double* out) {
        green_contract_kernel<<<dim3((inner + kGreenThreads - 1) / kGreenThreads, (x.count + kGreenU - 1) / kGreenU, outer),
                                kGreenThreads, 0, c.st>>>(x, in, inner, out);
    };
    contract(ax[1], R1, ax[2].count, ax[0].n, R2);
    contract(ax[0], R2, ax[1].count * ax[2].count, 1, T);
    green_matrix_kernel<<<grid1((long long)o.n * o.n), kT, 0, c.st>>>(ax[0], ax[1], ax[2], T, du.p, o.n, 1.0 / c.p.eps0, B);
    FOPIS_LAUNCH_CHECK();
    FOPIS_CUDA(cudaStreamSynchronize(c.st));   // the node list is a local
    return true;
}

// B column by column: one solve per surface node.
static void solved_matrix(Ctx& c, const ObjectDev& o, double* B) {
    const int n = o.n;
    const double tol = std::min(c.p.poisson_tol > 0 ? c.p.poisson_tol : 1e-8, 1e-10);
    for (int col = 0; col < n; ++col) {
        const long long node = ((long long)o.nodes_ijk[3 * col] * c.cy + o.nodes_ijk[3 * col + 1]) * c.cz + o.nodes_ijk[3 * col + 2];
        ++c.launches;
        set_node_kernel<<<1, 1, 0, c.st>>>(c.rho0, node, 1.0);
        FOPIS_CUDA(cudaMemsetAsync(c.phi, 0, sizeof(double) * c.N, c.st));
        const int rc = mg_solve(c, tol, 200);
        if (rc != FOPIS_OK) throw ApiError{rc, "capacity-matrix column solve did not converge"};
        // capacity_matrix(col, row) = phi at row (RootGridObject.cpp:114-126)
        ++c.launches;
        gather_kernel<<<grid1(n), kT, 0, c.st>>>(c.phi, o.nodes, n, B + (size_t)col * n);
        ++c.launches;
        set_node_kernel<<<1, 1, 0, c.st>>>(c.rho0, node, 0.0);
        FOPIS_LAUNCH_CHECK();
    }
}

void cmatrix_build(Ctx& c, int id) {
    ObjectDev& o = c.objs[id];
    const int n = o.n;
    double* B = o.C;
    // keep the user's fields: the reference builds C before any particle exists
    FOPIS_CUDA(cudaMemsetAsync(c.rho0, 0, sizeof(double) * c.N, c.st));
    if (!green_matrix(c, o, B)) solved_matrix(c, o, B);
    FOPIS_CUDA(cudaMemsetAsync(c.phi, 0, sizeof(double) * c.N, c.st));
    StreamBuffer<double> panels(c);
    StreamBuffer<unsigned> bad(c);
    if (!panels.alloc((size_t)2 * kGj * n) || !bad.alloc(1)) FOPIS_CUDA(cudaErrorMemoryAllocation);
    double *row = panels.p, *col = row + (size_t)kGj * n;
    FOPIS_CUDA(cudaMemsetAsync(bad.p, 0, sizeof(unsigned), c.st));
    const int tiles = (n + kGjTile - 1) / kGjTile;
    for (int k = 0; k < n; k += kGj) {
        c.launches += 2;
        gj_panel_kernel<<<(n + 255) / 256, 256, 0, c.st>>>(B, n, k, row, col, bad.p);
        gj_update_kernel<<<dim3(tiles, tiles), 256, 0, c.st>>>(B, n, k, row, col);
    }
    FOPIS_LAUNCH_CHECK();
    unsigned hbad = 0;
    FOPIS_CUDA(cudaMemcpyAsync(&hbad, bad.p, sizeof(unsigned), cudaMemcpyDeviceToHost, c.st));
    FOPIS_CUDA(cudaStreamSynchronize(c.st));
    if (hbad) throw ApiError{FOPIS_ERR_DEVICE, "capacity matrix B is not positive definite"};
    finish_C(c, o);
}

void cmatrix_set(Ctx& c, int id, const double* hostC) {
    ObjectDev& o = c.objs[id];
    copy_to_device(c, o.C, hostC, sizeof(double) * (size_t)o.n * o.n);
    finish_C(c, o);
}

void objects_step_begin(Ctx& c) {
    FOPIS_CUDA(cudaMemsetAsync(&c.d_sc->absorbed_n, 0, sizeof(unsigned long long), c.st));
    FOPIS_CUDA(cudaMemsetAsync(c.d_sc->absorbed_by, 0, sizeof(c.d_sc->absorbed_by), c.st));
    FOPIS_CUDA(cudaMemsetAsync(c.d_sc->emitted_by, 0, sizeof(c.d_sc->emitted_by), c.st));
}

// Moves the step's fixed-point surface charge into the charge maps and the
// total charge into scal[1] (RootGrid::updateRho's sumWholeCharge).
void objects_step_end(Ctx& c) {
    for (auto& o : c.objs) {
        double sc[FOPIS_MAX_SPECIES];
        for (int s = 0; s < c.nsp; ++s) sc[s] = c.p.species[s].charge * c.p.species[s].size * kSurfaceUnit;
        double* dsc = c.scratch64;   // small staging area
        FOPIS_CUDA(cudaMemcpyAsync(dsc, sc, sizeof(double) * c.nsp, cudaMemcpyHostToDevice, c.st));
        ++c.launches;
        sum_charge_kernel<<<1, 1024, 0, c.st>>>(o.charge_tmp, o.charge_map, c.nsp, o.n, dsc, o.scal);
        FOPIS_LAUNCH_CHECK();
        FOPIS_CUDA(cudaStreamSynchronize(c.st));
    }
}

void redistribute(Ctx& c) {
    for (auto& o : c.objs) {
        if (!o.has_C) throw ApiError{FOPIS_ERR_STATE, "capacity matrix not built"};
        ++c.launches;
        potential_kernel<<<1, 1024, 0, c.st>>>(c.phi, o.nodes, o.colsum, o.n, o.total, o.is_fixed, o.fixed_potential,
                                                o.phis, o.scal, o.dielectric ? o.capacitance : nullptr, o.charge_map,
                                                c.nsp);
        ++c.launches;
        drho_kernel<<<grid1((long long)o.n * 32), kT, 0, c.st>>>(o.C, o.n, o.phis, o.scal, o.nodes, c.rho0, o.drho[0]);
        FOPIS_LAUNCH_CHECK();
        double sc[2];
        FOPIS_CUDA(cudaMemcpyAsync(sc, o.scal, sizeof(double) * 2, cudaMemcpyDeviceToHost, c.st));
        FOPIS_CUDA(cudaStreamSynchronize(c.st));
        o.potential = sc[0];
        o.total_charge = sc[1];
    }
    glue_copy(c, c.rho0);
}

// phi (the first solve's result) += the fitted conductor responses.
void conductor_start(Ctx& c) {
    if (c.obj_hist < 1 || c.objs.empty()) return;
    ConductorFit f{};
    f.nobj = (int)c.objs.size();
    f.terms = c.obj_hist >= 2 ? 2 : 1;
    for (int o = 0; o < f.nobj; ++o) {
        f.d0[o] = c.objs[o].drho[0]; f.d1[o] = c.objs[o].drho[1]; f.d2[o] = c.objs[o].drho[2];
        f.n[o] = c.objs[o].n;
    }
    double* alpha = &c.d_sc->red[12];
    ++c.launches;
    conductor_fit_kernel<<<1, 1024, 0, c.st>>>(f, alpha);
    ++c.launches;
    conductor_start_kernel<<<grid1((long long)c.N), kT, 0, c.st>>>(c.phi, c.phi_obj, c.phi_obj2, alpha, (long long)c.N);
    FOPIS_LAUNCH_CHECK();
}

// After the second solve: the response phi_final - phi_first becomes the
// newest history entry, with this step's redistributed charge.
void conductor_record(Ctx& c, const double* phi_first) {
    std::swap(c.phi_obj, c.phi_obj2);
    phi_axpy(c, c.phi_obj, c.phi, phi_first, -1.0);
    for (auto& o : c.objs) {
        double* oldest = o.drho[2];
        o.drho[2] = o.drho[1];
        o.drho[1] = o.drho[0];
        o.drho[0] = oldest;
    }
    c.obj_hist = std::min(2, c.obj_hist + 1);
}

}  // namespace fopis
