// fields.cu — node-field kernels: charge fold and conversion, boundary
// conditions of phi, nodal electric field, field energy and exports.
#include "internal.cuh"

#include <algorithm>

namespace fopis {

namespace {

constexpr int kT = 256;

struct G {
    int cx, cy, cz;
    int n[3];
    int per[6];
};
G make_g(const Ctx& c) {
    G g;
    g.cx = c.cx; g.cy = c.cy; g.cz = c.cz;
    g.n[0] = c.nx; g.n[1] = c.ny; g.n[2] = c.nz;
    for (int t = 0; t < 6; ++t) g.per[t] = c.per[t];
    return g;
}
__device__ __forceinline__ long long L(const G& g, int i, int j, int k) {
    return ((long long)i * g.cy + j) * g.cz + k;
}
int blocks(long long n) {
    long long b = (n + kT - 1) / kT;
    return (int)(b < 148LL * 32 ? (b < 1 ? 1 : b) : 148LL * 32);
}

// A fixed-point fold sum that passed 2^64 (unsigned wrap) is latched as
// FOPIS_DEV_RHO_OVERFLOW; FP64 sums have no such limit.
__device__ __forceinline__ bool fold_wrapped(unsigned long long sum, unsigned long long a) { return sum < a; }
__device__ __forceinline__ bool fold_wrapped(double, double) { return false; }

struct Scales { double v[FOPIS_MAX_SPECIES]; };

// A species accumulator as a number: unsigned 64-bit fixed point (mixed mode;
// the weights are nonnegative and the deposit latches any wrap) or the FP64
// weight sum (FP64 mode).
__device__ __forceinline__ double weight_value(unsigned long long w) { return (double)w; }
__device__ __forceinline__ double weight_value(double w) { return w; }

// rho[0] = sum_s q_s size_s W_s (x 2^-51 in fixed point) (RootGridField.cpp:1206-1214),
// with the periodic folds of every species array before it
// (MPIw::Environment::sendRecvNodeScalar self-exchange, glue size 2,
// src/MPI/Communicator.cpp:497-574, axis after axis): along a periodic axis nodes
// 0 and n both become their sum, nodes 1 and n+1 likewise. A thread takes one
// class of nodes that the folds join (1, 2, 4 or 8 of them; along a periodic axis
// class 0 is {0, n}, class 1 is {1, n+1}, the rest single), sums it in the order
// of the axes and writes all of it, so one launch does what one per axis and the
// conversion did.
template <typename W>
__global__ void convert_kernel(W* rho, int nsp, long long N, G g, Scales sc, double* rho0, unsigned* status) {
    const int m[3] = {g.per[0] ? g.cx - 2 : g.cx, g.per[2] ? g.cy - 2 : g.cy, g.per[4] ? g.cz - 2 : g.cz};
    const long long total = (long long)m[0] * m[1] * m[2];
    for (long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x; t < total; t += (long long)gridDim.x * blockDim.x) {
        const unsigned u = (unsigned)t;   // fewer than 2^31 nodes
        const int k = (int)(u % (unsigned)m[2]), r = (int)(u / (unsigned)m[2]), j = r % m[1], i = r / m[1];
        const long long p = L(g, i, j, k);
        // distance to the joined node along each axis, 0 where there is none
        const long long dx = g.per[0] && i < 2 ? (long long)(g.cx - 2) * g.cy * g.cz : 0,
                        dy = g.per[2] && j < 2 ? (long long)(g.cy - 2) * g.cz : 0, dz = g.per[4] && k < 2 ? g.cz - 2 : 0;
        double v = 0.0;
        if (dx == 0 && dy == 0 && dz == 0) {
            for (int s = 0; s < nsp; ++s) v += sc.v[s] * weight_value(rho[(long long)s * N + p]);
            rho0[p] = v;
            continue;
        }
        for (int s = 0; s < nsp; ++s) {
            W* a = rho + (long long)s * N + p;
            bool wrapped = false;
            auto add = [&](W x, W y) { const W z = x + y; wrapped = wrapped || fold_wrapped(z, x); return z; };
            W sum = 0;
            for (int z = 0; z < (dz ? 2 : 1); ++z) {
                W w = 0;
                for (int y = 0; y < (dy ? 2 : 1); ++y) {
                    W x = a[z * dz + y * dy];
                    if (dx) x = add(x, a[z * dz + y * dy + dx]);
                    w = y ? add(w, x) : x;
                }
                sum = z ? add(sum, w) : w;
            }
            if (wrapped) atomicOr(status, (unsigned)FOPIS_DEV_RHO_OVERFLOW);
            for (int q = 0; q < 8; ++q)
                if ((!(q & 1) || dx) && (!(q & 2) || dy) && (!(q & 4) || dz))
                    a[((q & 1) ? dx : 0) + ((q & 2) ? dy : 0) + ((q & 4) ? dz : 0)] = sum;
            v += sc.v[s] * weight_value(sum);
        }
        for (int q = 0; q < 8; ++q)
            if ((!(q & 1) || dx) && (!(q & 2) || dy) && (!(q & 4) || dz))
                rho0[p + ((q & 1) ? dx : 0) + ((q & 2) ? dy : 0) + ((q & 4) ? dz : 0)] = v;
    }
}

template <typename W>
__global__ void convert_species_kernel(const W* rho, long long N, double scale, double* out) {
    for (long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x; t < N; t += (long long)gridDim.x * blockDim.x)
        out[t] = scale * weight_value(rho[t]);
}

// Glue copies of every periodic axis at once: node 0 <- node n, node n+1 <-
// node 1 (Communicator::sendRecvFieldX/Y/Z self branch, Communicator.cpp:290-299,
// axis after axis): a glue node takes the node with all its periodic indices
// wrapped, which no copy writes. Nodes on two planes are written twice, alike.
struct Planes {
    long long start[7];   // first item of each plane or face
    int axis[6], side[6];
    int n;
};
__global__ void glue_kernel(double* a, G g, Planes f) {
    const int dims[3] = {g.cx, g.cy, g.cz};
    for (long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x; t < f.start[f.n]; t += (long long)gridDim.x * blockDim.x) {
        int q = 0;
        while (t >= f.start[q + 1]) ++q;
        const int axis = f.axis[q], a1 = axis == 0 ? 1 : 0, a2 = axis == 2 ? 1 : 2;
        const int r = (int)(t - f.start[q]);
        int idx[3], src[3];
        idx[a1] = r / dims[a2];
        idx[a2] = r % dims[a2];
        idx[axis] = f.side[q] ? dims[axis] - 1 : 0;
        for (int d = 0; d < 3; ++d) {
            src[d] = idx[d];
            if (g.per[2 * d]) src[d] = idx[d] == 0 ? dims[d] - 2 : (idx[d] == dims[d] - 1 ? 1 : idx[d]);
        }
        a[L(g, idx[0], idx[1], idx[2])] = a[L(g, src[0], src[1], src[2])];
    }
}

// Field::setDirichletPhi / setNeumannPhi (src/Grid/Field.cpp:34-96) on every
// face in one launch: the face planes over the interior of the other two axes,
// in the reference's order x-, x+, y-, ... A node on several faces keeps the
// last one's value: zero, or the node one step inwards as the faces before it
// left that, so the walk goes down the axes; it ends off the faces, at nodes
// that nothing here writes.
__global__ void phi_face_kernel(double* phi, G g, Planes f, unsigned neumann) {
    const int dims[3] = {g.cx, g.cy, g.cz};
    for (long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x; t < f.start[f.n]; t += (long long)gridDim.x * blockDim.x) {
        int q = 0;
        while (t >= f.start[q + 1]) ++q;
        const int axis = f.axis[q], a1 = axis == 0 ? 1 : 0, a2 = axis == 2 ? 1 : 2;
        const int r = (int)(t - f.start[q]), m2 = dims[a2] - 2;
        int idx[3], src[3];
        idx[a1] = 1 + r / m2;
        idx[a2] = 1 + r % m2;
        idx[axis] = f.side[q] ? dims[axis] - 2 : 1;
        bool held = false;
        for (int d = 2; d >= 0; --d) {
            src[d] = idx[d];
            if (held || g.per[2 * d]) continue;
            const int hi = idx[d] == dims[d] - 2;
            if (!hi && idx[d] != 1) continue;
            if ((neumann >> (2 * d + hi)) & 1u) src[d] = hi ? dims[d] - 3 : 2;
            else held = true;
        }
        phi[L(g, idx[0], idx[1], idx[2])] = held ? 0.0 : phi[L(g, src[0], src[1], src[2])];
    }
}

// Maps an index of a periodic axis onto its interior image.
__device__ __forceinline__ int wrapi(const G& g, int axis, int idx) {
    if (g.per[2 * axis]) {
        const int n = g.n[axis];
        if (idx == 0) return n;
        if (idx == n + 1) return 1;
    }
    return idx;
}

__device__ __forceinline__ void store_e(float4* o, const double e[3]) {
    *o = make_float4((float)e[0], (float)e[1], (float)e[2], 0.0f);
}
__device__ __forceinline__ void store_e(Vec4d* o, const double e[3]) { *o = Vec4d{e[0], e[1], e[2], 0.0}; }

// Nodal E of RootGrid::updateEfield + updateReferenceEfield
// (RootGridField.cpp:456-582): centred 0.5 (phi[i-1] - phi[i+1]) per axis,
// one-sided second order on Dirichlet/Neumann faces, zero glue on those axes,
// periodic images on periodic axes (sendRecvField self-copies).
template <typename Out>
__global__ void efield_kernel(const double* phi, G g, Out* out, double* outx, double* outy, double* outz) {
    const long long N = (long long)g.cx * g.cy * g.cz;
    for (long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x; t < N; t += (long long)gridDim.x * blockDim.x) {
        const int i0 = (int)(t / ((long long)g.cy * g.cz));
        const int j0 = (int)((t / g.cz) % g.cy);
        const int k0 = (int)(t % g.cz);
        int id[3] = {wrapi(g, 0, i0), wrapi(g, 1, j0), wrapi(g, 2, k0)};
        const int dims[3] = {g.cx, g.cy, g.cz};
        bool outside = false;
        for (int a = 0; a < 3; ++a) if (id[a] == 0 || id[a] == dims[a] - 1) outside = true;
        double e[3] = {0.0, 0.0, 0.0};
        if (!outside) {
            for (int a = 0; a < 3; ++a) {
                int lo[3] = {id[0], id[1], id[2]}, hi[3] = {id[0], id[1], id[2]};
                const int X = dims[a];
                if (!g.per[2 * a] && id[a] == 1) {
                    int p2[3] = {id[0], id[1], id[2]}, p3[3] = {id[0], id[1], id[2]};
                    p2[a] = 2; p3[a] = 3;
                    e[a] = 0.5 * (phi[L(g, p3[0], p3[1], p3[2])] - 4.0 * phi[L(g, p2[0], p2[1], p2[2])] +
                                  3.0 * phi[L(g, id[0], id[1], id[2])]);
                } else if (!g.per[2 * a + 1] && id[a] == X - 2) {
                    int p2[3] = {id[0], id[1], id[2]}, p3[3] = {id[0], id[1], id[2]};
                    p2[a] = X - 3; p3[a] = X - 4;
                    e[a] = 0.5 * (-phi[L(g, p3[0], p3[1], p3[2])] + 4.0 * phi[L(g, p2[0], p2[1], p2[2])] -
                                  3.0 * phi[L(g, id[0], id[1], id[2])]);
                } else {
                    lo[a] = id[a] - 1; hi[a] = id[a] + 1;   // glue neighbours hold periodic images
                    e[a] = 0.5 * ((phi[L(g, lo[0], lo[1], lo[2])] - phi[L(g, id[0], id[1], id[2])]) +
                                  (phi[L(g, id[0], id[1], id[2])] - phi[L(g, hi[0], hi[1], hi[2])]));
                }
            }
        }
        if (out) store_e(out + t, e);
        if (outx) { outx[t] = e[0]; outy[t] = e[1]; outz[t] = e[2]; }
    }
}

__device__ __forceinline__ double bsum(double v) {
    __shared__ double red[32];
    for (int o = 16; o; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
    const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
    __syncthreads();
    if (l == 0) red[w] = v;
    __syncthreads();
    v = 0.0;
    if (w == 0) {
        v = (l < (int)(blockDim.x >> 5)) ? red[l] : 0.0;
        for (int o = 16; o; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
    }
    return v;
}

// Field::getEfieldEnergy (src/Grid/Field.cpp:194-213) from the edge fields
// ex[i] = phi[i] - phi[i+1] (RootGridField.cpp:470-478); per-block partials.
__global__ void field_energy_kernel(const double* phi, G g, double* partial) {
    const long long M = (long long)(g.cx - 2) * (g.cy - 2) * (g.cz - 2);
    double en = 0.0;
    for (long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x; t < M; t += (long long)gridDim.x * blockDim.x) {
        const int i = 1 + (int)(t / ((long long)(g.cy - 2) * (g.cz - 2)));
        const int j = 1 + (int)((t / (g.cz - 2)) % (g.cy - 2));
        const int k = 1 + (int)(t % (g.cz - 2));
        const double p = phi[L(g, i, j, k)];
        if (i < g.cx - 2) { const double d = p - phi[L(g, i + 1, j, k)]; en += d * d; }
        if (j < g.cy - 2) { const double d = p - phi[L(g, i, j + 1, k)]; en += d * d; }
        if (k < g.cz - 2) { const double d = p - phi[L(g, i, j, k + 1)]; en += d * d; }
    }
    en = bsum(en);
    if (threadIdx.x == 0) partial[blockIdx.x] = en;
}

__global__ void sum_partials_kernel(const double* partial, int n, double* out) {
    double v = 0.0;
    for (int t = threadIdx.x; t < n; t += blockDim.x) v += partial[t];
    v = bsum(v);
    if (threadIdx.x == 0) *out = v;
}

}  // namespace

// Charge of one unit of a species' accumulator: q size 2^-51 for the
// fixed-point weights, q size for the FP64 weights.
double species_rho_scale(const Ctx& c, int s) {
    return c.p.species[s].charge * c.p.species[s].size * (c.fp64 ? 1.0 : kDepositUnit);
}

void rho_zero(Ctx& c) {
    FOPIS_CUDA(cudaMemsetAsync(c.rho_i64, 0, sizeof(unsigned long long) * c.N * c.nsp, c.st));
}

static void add_plane(Planes& f, int axis, int side, long long items) {
    f.axis[f.n] = axis;
    f.side[f.n] = side;
    f.start[f.n + 1] = f.start[f.n] + items;
    ++f.n;
}

void glue_copy(Ctx& c, double* a) {
    const G g = make_g(c);
    const long long planes[3] = {(long long)c.cy * c.cz, (long long)c.cx * c.cz, (long long)c.cx * c.cy};
    Planes f{};
    for (int axis = 0; axis < 3; ++axis)
        for (int side = 0; side < 2 && c.per[2 * axis]; ++side) add_plane(f, axis, side, planes[axis]);
    if (f.n == 0) return;
    ++c.launches;
    glue_kernel<<<blocks(f.start[f.n]), kT, 0, c.st>>>(a, g, f);
    FOPIS_LAUNCH_CHECK();
}

void rho_finalize(Ctx& c) {
    const G g = make_g(c);
    Scales sc{};
    for (int s = 0; s < c.nsp; ++s) sc.v[s] = species_rho_scale(c, s);
    ++c.launches;
    if (c.fp64)
        convert_kernel<<<blocks((long long)c.N), kT, 0, c.st>>>(reinterpret_cast<double*>(c.rho_i64), c.nsp, (long long)c.N,
                                                                g, sc, c.rho0, &c.d_sc->status);
    else
        convert_kernel<<<blocks((long long)c.N), kT, 0, c.st>>>(c.rho_i64, c.nsp, (long long)c.N, g, sc, c.rho0,
                                                                &c.d_sc->status);
    FOPIS_LAUNCH_CHECK();
}

// After a solve: the periodic glue copies first (the last halo exchange of the
// reference's doPSOR), then Field::setBoundaryConditionPhi on the D/N faces
// (RootGridField.cpp:65-103 calls it after the sweeps and exchanges nothing
// afterwards), so a glue node beside a Neumann face keeps the value it had
// before the face copy, as in the reference.
void phi_boundary(Ctx& c) {
    const G g = make_g(c);
    glue_copy(c, c.phi);
    Planes f{};
    unsigned neumann = 0;
    const long long m[3] = {(long long)(c.cy - 2) * (c.cz - 2), (long long)(c.cx - 2) * (c.cz - 2),
                            (long long)(c.cx - 2) * (c.cy - 2)};
    for (int axis = 0; axis < 3; ++axis)
        for (int side = 0; side < 2; ++side) {
            const char b = c.p.boundary[2 * axis + side];
            if (b == 'P') continue;
            if (b == 'N') neumann |= 1u << (2 * axis + side);
            add_plane(f, axis, side, m[axis]);
        }
    if (f.n == 0) return;
    ++c.launches;
    phi_face_kernel<<<blocks(f.start[f.n]), kT, 0, c.st>>>(c.phi, g, f, neumann);
    FOPIS_LAUNCH_CHECK();
}

void efield_update(Ctx& c) {
    const G g = make_g(c);
    ++c.launches;
    if (c.fp64) efield_kernel<Vec4d><<<blocks((long long)c.N), kT, 0, c.st>>>(c.phi, g, c.E64, nullptr, nullptr, nullptr);
    else efield_kernel<float4><<<blocks((long long)c.N), kT, 0, c.st>>>(c.phi, g, c.E, nullptr, nullptr, nullptr);
    FOPIS_LAUNCH_CHECK();
}

void field_export(Ctx& c, int which, double* host) {
    const G g = make_g(c);
    const size_t bytes = sizeof(double) * c.N;
    if (which == FOPIS_FIELD_PHI) {
        copy_to_host(c, host, c.phi, bytes);
    } else if (which == FOPIS_FIELD_RHO0) {
        copy_to_host(c, host, c.rho0, bytes);
    } else if (which >= FOPIS_FIELD_EXREF && which <= FOPIS_FIELD_EZREF) {
        double* tmp = nullptr;
        FOPIS_CUDA(cudaMallocAsync(&tmp, 3 * bytes, c.st));
        ++c.launches;
        efield_kernel<float4><<<blocks((long long)c.N), kT, 0, c.st>>>(c.phi, g, nullptr, tmp, tmp + c.N, tmp + 2 * c.N);
        FOPIS_LAUNCH_CHECK();
        copy_to_host(c, host, tmp + (which - FOPIS_FIELD_EXREF) * c.N, bytes);
        FOPIS_CUDA(cudaFreeAsync(tmp, c.st));
    } else if (which >= FOPIS_FIELD_RHO_SPECIES && which < FOPIS_FIELD_RHO_SPECIES + c.nsp) {
        const int s = which - FOPIS_FIELD_RHO_SPECIES;
        const double scale = species_rho_scale(c, s);
        ++c.launches;
        if (c.fp64)
            convert_species_kernel<<<blocks((long long)c.N), kT, 0, c.st>>>(
                reinterpret_cast<const double*>(c.rho_i64) + (size_t)s * c.N, (long long)c.N, scale, c.scratch64);
        else
            convert_species_kernel<<<blocks((long long)c.N), kT, 0, c.st>>>(c.rho_i64 + (size_t)s * c.N, (long long)c.N,
                                                                           scale, c.scratch64);
        FOPIS_LAUNCH_CHECK();
        copy_to_host(c, host, c.scratch64, bytes);
    } else {
        throw ApiError{FOPIS_ERR_ARG, "unknown field selector"};
    }
}

double efield_energy(Ctx& c) {
    const G g = make_g(c);
    const int nb = 148 * 4;
    double* part = c.red_partials;
    ++c.launches;
    field_energy_kernel<<<nb, kT, 0, c.st>>>(c.phi, g, part);
    ++c.launches;
    sum_partials_kernel<<<1, 1024, 0, c.st>>>(part, nb, &c.d_sc->red[15]);
    FOPIS_LAUNCH_CHECK();
    double v = 0.0;
    FOPIS_CUDA(cudaMemcpyAsync(&v, &c.d_sc->red[15], sizeof(double), cudaMemcpyDeviceToHost, c.st));
    FOPIS_CUDA(cudaStreamSynchronize(c.st));
    return 0.5 * c.p.eps0 * v;
}

namespace {
__global__ void __launch_bounds__(256) axpy_kernel(double* dst, const double* a, const double* b, double sb, long long n) {
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x)
        dst[i] = a[i] + sb * b[i];
}
}  // namespace

void phi_axpy(Ctx& c, double* dst, const double* a, const double* b, double sb) {
    const long long n = (long long)c.N;
    ++c.launches;
    axpy_kernel<<<(int)std::min<long long>((n + 255) / 256, 148 * 16), 256, 0, c.st>>>(dst, a, b, sb, n);
    FOPIS_LAUNCH_CHECK();
}

}  // namespace fopis
