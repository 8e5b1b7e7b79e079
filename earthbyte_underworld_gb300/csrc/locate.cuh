// Element search along one axis of the regular mesh (Mesh_RegularAlgorithms_SearchElements,
// StgDomain/Mesh/src/Mesh_RegularAlgorithms.c:194-226 with the separations of :154-175 and Num_Approx's 1e-12,
// StGermain/Base/Foundation/src/Numerics.c:37-41), shared by the mapper and the advection.
#pragma once

#include <cmath>

#include "internal.cuh"

namespace uwg {

// One axis of the mesh.  The reference rule divides: index = trunc(RN((x - mn) / sep)), one less when the
// fraction is within 1e-12 of zero, with tests at both ends.  FP64 division costs tens of FP64 instructions
// at 1/64 of the FP32 rate, and k_locate and k_advect were bound by it.  So one FMA places x in fixed point
// (32 fraction bits in the low word of m = x inv + (1.5 2^20 - mn inv)); its error is below 2^-31, so when
// the fraction is 2^-29 or more away from both ends of the cell and the index is inside the mesh, the rule
// gives that index.  All other points, and meshes beyond the bounds of `fast`, take the rule itself.
struct AxisMap {
    double mn, mx, sep, inv, off;
    int nel, fast;
};

inline AxisMap axis_map(double mn, double mx, int nel) {
    AxisMap a;
    a.mn = mn;
    a.mx = mx;
    a.nel = nel;
    a.sep = (mx - mn) / nel;
    a.inv = 1.0 / a.sep;
    const double shift = mn * a.inv;
    a.off = 1572864.0 - shift;
    // |x inv| and |mn inv| stay below 2^19; the 1e-12 window at the upper end is less than a quarter cell
    a.fast = nel <= (1 << 18) && std::isfinite(a.inv) && std::fabs(shift) <= 262144.0 && 1e-12 * a.inv < 0.25;
    return a;
}

__device__ __forceinline__ bool axis_approx(double var, double val) {
    const double eps = 1e-12;
    return var >= val - eps && var <= val + eps;
}

// the rule itself; false when x is outside the mesh or not finite
static __device__ __noinline__ bool axis_rule(const AxisMap& a, double x, int& idx) {
    if (!isfinite(x)) return false;
    if (axis_approx(x - a.mx, 0.0)) {
        idx = a.nel - 1;
        return true;
    }
    if (x < a.mn || x > a.mx) return false;
    const double out = __ddiv_rn(x - a.mn, a.sep);
    const double integer = trunc(out);
    const double frac = out - integer;   // exact: modf of a non-negative value
    unsigned i = (unsigned)integer;
    if (i > 0 && axis_approx(frac, 0.0)) i--;
    // a value that rounds onto the upper face is still inside the last element
    if (i >= (unsigned)a.nel) i = (unsigned)a.nel - 1;
    idx = (int)i;
    return true;
}

__device__ __forceinline__ bool axis_index(const AxisMap& a, double x, int& idx) {
    const double m = fma(x, a.inv, a.off);
    const int i = __double2hiint(m) - 0x41380000;
    const unsigned frac = (unsigned)__double2loint(m);
    if (a.fast && (unsigned)i < (unsigned)a.nel && frac - 8u < 0xfffffff0u) {
        idx = i;
        return true;
    }
    return axis_rule(a, x, idx);
}

}  // namespace uwg
