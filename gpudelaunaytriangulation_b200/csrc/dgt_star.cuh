// What the kernels of the first stage (dgt_star.cu, dgt_wrap.cu) share: the hull of inverted
// offsets.  Inversion d -> d' = d / |d|^2 about the point p (all offsets relative to p) turns the
// circle through p, a and b into the line through a' and b', and "d strictly inside that circle"
// into "d' strictly on the far side of that line from the origin": the Delaunay ring of p among
// a set of candidates is the convex hull of their inverted offsets.
//
// Error bound of a turn (u the unit roundoff of T).  Inverted coordinates: offset rounding u,
// |d|^2 4u, reciprocal 4u, product u, so each lies within 10.1u |d'| of its exact value.  For
// the turn o = (b' - a') x (c' - a') the three displacements contribute at most
// 10.1u (|a'||b'-c'| + |b'||c'-a'| + |c'||b'-a'|) <= 10.1u (|c'-a'|(|a'|+|b'|) + |b'-a'|(|a'|+|c'|)),
// the arithmetic 4u |b'-a'||c'-a'| <= 4u |b'-a'|(|a'|+|c'|): the test uses 16u of the sum, with
// one-norms in place of the Euclidean ones.
#pragma once
#include "dgt_builder.cuh"

namespace dgt {

// the hardware approximations (2^-23 and 2^-22.9 relative), without denormal handling: their
// arguments are kept in range
__device__ __forceinline__ float rcp_fast(float x)
{
    float r;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
}
__device__ __forceinline__ double rcp_fast(double x) { return 1.0 / x; }
// at least sqrt(x)
__device__ __forceinline__ float sqrt_over(float x)
{
    float r;
    asm("sqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r * 1.000001f;
}
__device__ __forceinline__ double sqrt_over(double x) { return sqrt(x) * (1.0 + 4e-16); }

// 16u times the one-norm
template <typename T>
__device__ __forceinline__ T err1(typename Prec<T>::T2 a)
{
    return (fabs(a.x) + fabs(a.y)) * ((T)16 * Prec<T>::u());
}

// the filter's answer at the turn a, b, c (inverted offsets and their err1): o > bnd a left
// turn, o < -bnd a right turn
template <typename T>
__device__ __forceinline__ void turn(typename Prec<T>::T2 a, typename Prec<T>::T2 b, typename Prec<T>::T2 c, T ea, T eb,
                                     T ec, T &o, T &bnd)
{
    const T ux = b.x - a.x, uy = b.y - a.y, vx = c.x - a.x, vy = c.y - a.y;
    o = ux * vy - uy * vx;
    bnd = (fabs(vx) + fabs(vy)) * (ea + eb) + ((fabs(ux) + fabs(uy)) * (ea + ec) + Prec<T>::tiny());
}

// offset of candidate id relative to p; negative ids are the virtual corners
template <bool GEN>
__device__ __forceinline__ double2 star_off(const double2 *P, const SetDesc *S, double2 p, int id)
{
    if (GEN) return off64g(P, p, S, id);
    return off64(P, p, S->Lx, S->hLx, S->Ly, S->hLy, S->V, id);
}

// float64 decision of the turn a, b, c: +1 left (b is a vertex), -1 right, 0 undecided (with
// EXACT: c exactly on the circle through p, a and b)
template <bool GEN, bool EXACT>
__device__ __noinline__ int star_recheck(const double2 *P, const SetDesc *S, double2 p, int ia, int ib, int ic)
{
    const double2 a = star_off<GEN>(P, S, p, ia), b = star_off<GEN>(P, S, p, ib), c = star_off<GEN>(P, S, p, ic);
    const int r = incircle64(a.x, a.y, b.x, b.y, c.x, c.y);
    if (r != 0 || !EXACT) return -r;
    return -incircle_exact(a.x, a.y, b.x, b.y, c.x, c.y);
}

}  // namespace dgt
