// direct.cuh — interface of the fast-diagonalisation correction solve
// (direct.cu) to the Poisson refinement (multigrid.cu).
#pragma once

#include "internal.cuh"

#include <utility>

namespace fopis {

// The FP64 side on the glue-layout arrays.
struct DirectOuter {
    int cx, cy, cz;
    int o[3];             // glue index of unknown 0
    int per[3], nref[3];  // periodic axes and their node counts
    int allper;
    double eps0, inv_eps0;
    double inv_m, root_m;   // of the unknowns' number m: 1 / m and its square root
};

// What the residual kernel's last block does with the sums: keep them (the
// host decides), or start / continue the device-side loop of the solve graph.
// The scalars of DevScalars::red are those of multigrid.cu; `host` is the
// pinned mirror, which receives them too (no copy node in the graph).
enum DirectMode { DIRECT_START = 1, DIRECT_LOOP = 2 };   // bits: first residual of a solve; set the loop condition
struct DirectStep {
    DevScalars* sc;
    DevScalars* host;
    int mode;
    cudaGraphConditionalHandle loop;
};

constexpr int kDirectPartials = 4;   // doubles per block of direct_residual's `partial`

bool direct_first(const int n[3]);   // corrections by this from the start, and not only where V-cycles fail
int direct_blocks(const int n[3]);
void direct_setup(DirectShape& S, const int n[3], const int per[3]);
void direct_free(DirectShape& S);
int direct_residual(const DirectShape& S, const DirectOuter& O, const double* rho0, const double* phi, float* X,
                    double* partial, const DirectStep& step, bool pdl, cudaStream_t st);
int direct_correct(const DirectShape& S, const DirectOuter& O, float* X, double* phi, bool pdl, cudaStream_t st);

}  // namespace fopis
