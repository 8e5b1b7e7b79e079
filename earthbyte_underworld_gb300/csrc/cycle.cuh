// Small multigrid levels in one cooperative launch (cycle.cu).
#pragma once

#include "internal.cuh"

namespace uwg {

constexpr int kCyMaxLevels = 8;     // levels one launch covers
constexpr int kCyMaxDegree = 8;     // Chebyshev degrees it carries coefficients for
constexpr int kCyPass = 64;         // entries of an H column per Gram-Schmidt pass

struct CycleOpts {
    bool cheb;      // Chebyshev smoothing, else symmetric colour Gauss-Seidel
    int down, up;   // sweeps or degrees
    int cycle;      // 1: V-cycle
};

// First level of the part of the hierarchy that one launch runs; nlevels: none; 0: all of it, and a
// velocity solve's whole FGMRES iteration.
int cycle_first_level(const Context& c, const CycleOpts& o);
// x = one V-cycle over levels first .. nlevels - 1 applied to b (zero initial guess).
template <typename T>
void cycle_run(Context& c, const CycleOpts& o, int first, const T* b, T* x);
// One FGMRES iteration: z = V-cycle(V_k), w = A z orthogonalised against V_0 .. V_k (classical
// Gram-Schmidt, twice), vnext = w / ||w||.  host_out (pinned): the coefficients of the two passes at 0
// and kCyPass, ||w||^2 at 2 kCyPass, valid once the stream has been synchronised.
template <typename T>
void cycle_fgmres_iteration(Context& c, const CycleOpts& o, const T* V, int k, int64_t n, T* z, T* w, T* vnext,
                            double* host_out);
// A launch that gives up on a barrier leaves a flag.  cycle_begin clears it at the start of a solve (an earlier one may
// have ended early); cycle_check throws if it is set (synchronises the stream).  A solve that fails checks as well:
// the values such a launch leaves unfinished make it fail in some other way sooner or later.
void cycle_begin(Context& c);
void cycle_check(Context& c);

}  // namespace uwg
