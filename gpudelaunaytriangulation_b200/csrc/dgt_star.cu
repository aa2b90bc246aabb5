// One-ring construction from a bounded set of candidates (k_star): the first stage of builds and
// rebuilds of many points; what it cannot finish goes to the warp-per-point hull kernel
// (dgt_wrap.cu), and only that kernel's leftovers to the incremental warp kernel (dgt_ring.cu).
//
// Inversion d -> d' = d / |d|^2 about the point p (all offsets relative to p) turns the circle
// through p, a and b into the line through a' and b', and "d strictly inside that circle" into
// "d' strictly on the far side of that line from the origin".  The Delaunay ring of p among a
// set of candidates is therefore the convex hull of their inverted offsets, which a warp of 32
// points finds in lockstep with hardly any divergence:
//   1. gather: up to 32 candidates of a window of cells around p (cells of one row are one
//      range of the cell order), their inverted offsets in shared memory;
//   2. sort them by angle: 23-bit angles relative to the nearest candidate (always on the
//      hull), a 32-element sorting network in registers;
//   3. one Graham pass over the sorted candidates: every step either pops the top of the stack
//      (a right turn: its circle test says the top is no neighbour) or pushes the next one;
//   4. certify: every circle of the ring lies inside the window (and inside the radius the
//      candidates were cut at), so no point outside it can change the ring; if not, one more
//      pass over the cells the circles reach, with the candidates that lie in some circle.
// What bounds it: instruction issue (67% of the issue slots at 20 warps per SM, 22 of 32 lanes
// active; the incremental kernel has 53% and 10 lanes, and several times the instructions).  4M
// uniform points: 5.79 ms in the incremental kernel, 1.26 + 0.50 ms in these two launches; 1M
// lattice sites 0.56 -> 0.23 ms; 1M points with float64 predicates 2.75 -> 0.67 + 0.26 ms.
//
// Every decision is certain or the point is handed on: a turn the filter cannot decide is
// re-evaluated with the float64 in-circle predicate; angles closer than their rounding errors
// are settled by dropping the farther candidate where that is provably interior.
//
// Angles.  r = y / (|x| + |y|) continued over the four quadrants has an error of at most 16u =
// two units of 2^-21; keys whose difference exceeds four units are in their true order.
#include <type_traits>
#include "dgt_star.cuh"

namespace dgt {

namespace {

constexpr int STAR_CAP = 32;        // candidates of one pass (5-bit index in the sort key)
constexpr int STAR_BLOCK = 64;
constexpr int STAR_SEGS = 12;       // row ranges of a window (10-bit counts in two 64-bit words)
constexpr int STAR_SEG_MAX = 1023;
constexpr int STAR_TARGET = 22;     // candidates a radius cut aims at (a few more stay below STAR_CAP)
constexpr unsigned STAR_ANGLE_TOL = 5u << 9;

// ---- sorting network (Batcher odd-even merge sort), every index a compile-time constant
__device__ __forceinline__ void cmp_swap(unsigned &a, unsigned &b)
{
    const unsigned lo = min(a, b);
    b = max(a, b);
    a = lo;
}
template <int LO, int N, int R>
struct OeMerge {
    static __device__ __forceinline__ void run(unsigned (&k)[STAR_CAP])
    {
        if constexpr (2 * R < N) {
            OeMerge<LO, N, 2 * R>::run(k);
            OeMerge<LO + R, N, 2 * R>::run(k);
#pragma unroll
            for (int i = LO + R; i + R < LO + N; i += 2 * R) cmp_swap(k[i], k[i + R]);
        } else {
            cmp_swap(k[LO], k[LO + R]);
        }
    }
};
template <int LO, int N>
struct OeSort {
    static __device__ __forceinline__ void run(unsigned (&k)[STAR_CAP])
    {
        if constexpr (N > 1) {
            OeSort<LO, N / 2>::run(k);
            OeSort<LO + N / 2, N / 2>::run(k);
            OeMerge<LO, N, 1>::run(k);
        }
    }
};

// angle of (x, y) as a 23-bit fraction of the full turn in the top bits: with r = y / (|x| + |y|),
// 5 + r for x >= 0 and 7 - r for x < 0, in [4, 8] where one ulp is 2^-21 (8 wraps to 4)
__device__ __forceinline__ unsigned angle_key(float x, float y)
{
    const float r1 = fmaf(y, rcp_fast(fabsf(x) + fabsf(y)), -1.0f);
    const float sgn = __uint_as_float((__float_as_uint(x) & 0x80000000u) | 0x3f800000u);
    return __float_as_uint(fmaf(sgn, r1, 6.0f)) << 9;
}

// k_star's passes over one point: both in turn, or one per launch (the second over the list of
// points that the first could not certify)
enum { STAR_BOTH = 0, STAR_FIRST = 1, STAR_SECOND = 2 };

enum { S_TODO = 0, S_OK = 1, S_FAIL = 2 };

// ring of entry k of the second pass's list: its length, then up to STAR_RING - 1 slots
constexpr int STAR_RING = 16;
__device__ __forceinline__ int *second_ring(const RingArgs &A, int k)
{
    const int e = A.second_base + k;
    return e < A.second_split ? A.second_rings[0] + (size_t)e * STAR_RING
                              : A.second_rings[1] + (size_t)(e - A.second_split) * STAR_RING;
}

// Shared memory of a block, a column per thread.  SMALL (first pass with the float32 filter):
// slots as 16-bit offsets from the point's own slot, so that 20 warps fit an SM instead of 16 (4M
// uniform points: 1.49 -> 1.33 ms).  Taken when windows span at most 16,000 slots at the sets' mean
// densities; a point with a range further off than 16 bits reach is handed on (add_seg).
template <typename T, bool SMALL> struct StarMem {
    typedef typename Prec<T>::T2 V2;
    static constexpr int B = SMALL ? 128 : STAR_BLOCK;
    V2 q[SMALL ? STAR_CAP : STAR_CAP + 1][B];   // inverted offsets, behind them the stack's sentinel; the finished ring's indices
    typedef typename std::conditional<SMALL, short, int>::type Slot;
    Slot s[STAR_CAP][B];  // slot (build) or index (repair) of a candidate
    // the sorted order, and the hull stack in its place: candidate numbers, the sentinel's first
    // and the first candidate's again at the end
    unsigned char o[STAR_CAP + 2][B];
    // row ranges until they are taken: their starts, from the end of an array that fills from the front
    __device__ __forceinline__ int &start(int k, int t)
    {
        return SMALL ? *reinterpret_cast<int *>(&q[STAR_CAP - k][t]) : *reinterpret_cast<int *>(&s[STAR_CAP - k][t]);
    }
};

template <typename T, bool SMALL>
struct StarRing {
    StarMem<T, SMALL> &M;
    int t;
    __device__ __forceinline__ int idx(int k) const { return *reinterpret_cast<const int *>(&M.q[k][t]); }
    __device__ __forceinline__ void set(int k, int v) { *reinterpret_cast<int *>(&M.q[k][t]) = v; }
};

// Candidates whose angles may be out of order (bit k of close: sorted positions k - 1 and k; wrap:
// the last one and the first).  Let a, d have directions within 2.7e-4 rad (31 links of nine units)
// and |d'| (1 + 2^-10) < |a'|.  The hull contains the cone from a' to the disc of radius 1 / wmax
// about the origin (wmax: the largest diameter of a circle of the ring), which at distance |d'|
// from the origin is at least (1 - |d'| / |a'|) / wmax > 2^-10.01 / wmax wide on either side of the
// segment to a'; d' lies within 2.7e-4 |d'| of that segment.  So d' is interior, and d is
// dropped, if wmax |d'| < 3.6, which certify() checks.  Other pairs hand the point on.
// Returns the candidates left (-1: hand on); drop: the largest |d'|^2 of those dropped.
template <typename T, bool SMALL>
__device__ __noinline__ int settle_angles(StarMem<T, SMALL> *M, int t, int n, unsigned close, bool wrap, T *drop)
{
    auto at = [&](int k) { return &M->o[k + 1][t]; };
    auto len2 = [&](int k) { return M->q[k][t].x * M->q[k][t].x + M->q[k][t].y * M->q[k][t].y; };
    const T far2 = (T)1.001956;   // (1 + 2^-10)^2 and the rounding of the squares
    int out = 1;
    T most = (T)0;
    for (int k = 1; k < n; ++k) {
        const int cur = *at(k);
        if ((close >> k) & 1u) {
            const T lc = len2(cur), lk = len2(*at(out - 1));
            if (lk > lc * far2) {
                most = lc > most ? lc : most;
                continue;
            }
            if (!(lc > lk * far2)) return -1;
            most = lk > most ? lk : most;
            *at(out - 1) = (unsigned char)cur;
            continue;
        }
        *at(out++) = (unsigned char)cur;
    }
    if (wrap && out > 1) {
        const T lc = len2(*at(out - 1));
        if (!(len2(*at(0)) > lc * far2)) return -1;
        most = lc > most ? lc : most;
        --out;
    }
    *drop = most;
    return out;
}

// the slot (or index) of the candidate at place k of a column
template <typename T, bool SMALL>
__device__ __forceinline__ int star_slot(const StarMem<T, SMALL> &M, int t, const SetDesc &S, int self, int k)
{
    if (!SMALL) return M.s[k][t];
    int v = self + M.s[k][t];
    if (v < S.point_base) v += S.n;
    else if (v >= S.point_base + S.n) v -= S.n;
    return v;
}

// How far the circles of a ring reach: extents along the cell axes (twice those of the circles) and
// the largest diameter; good: all of them are bounded and well conditioned
template <typename T, bool GEN>
struct Reach {
    typedef typename Prec<T>::T2 V2;
    T sx, sy, g11, g12, g21, g22;
    T ulo = Prec<T>::inf(), uhi = -Prec<T>::inf(), vlo = Prec<T>::inf(), vhi = -Prec<T>::inf(), wmax = (T)0;
    bool good = true;
    __device__ __forceinline__ Reach(const SetDesc &S)
        : sx(GEN ? (T)S.gnx : (T)S.icw), sy(GEN ? (T)S.gny : (T)S.ich), g11((T)S.g11), g12((T)S.g12), g21((T)S.g21),
          g22((T)S.g22)
    {
    }
    // the circle through p and neighbours with the inverted offsets b and c (eb, ec: their err1)
    __device__ __forceinline__ void add(V2 b, V2 c, T eb, T ec)
    {
        const T g = b.x * c.y - b.y * c.x;
        // relative error of g below 24u 2^9 (2^-10.4 in float), of the pole below 2^-9.4
        // (eb and ec are the one-norms times 16u)
        good &= g > ((T)0.001953125 / ((T)256 * Prec<T>::u() * Prec<T>::u())) * eb * ec;
        const T ig = rcp_fast(g);
        const T wx = (c.y - b.y) * ig, wy = (b.x - c.x) * ig;
        const T w2 = wx * wx + wy * wy;
        const T hw = sqrt_over(w2) * (T)1.00390625;   // 1 + 2^-8
        wmax = hw > wmax ? hw : wmax;
        const T uc = GEN ? g11 * wx + g12 * wy : wx * sx, vc = GEN ? g21 * wx + g22 * wy : wy * sy;
        const T hu = hw * sx, hv = hw * sy;
        ulo = fmin(ulo, uc - hu);
        uhi = fmax(uhi, uc + hu);
        vlo = fmin(vlo, vc - hv);
        vhi = fmax(vhi, vc + hv);
    }
};

// Ring vertices whose turns are unsure (bit k: the k-th), in float64.  A vertex at a right turn is
// interior, as in the pass over the stack, and leaves the ring; its neighbours' turns are looked at
// again.  The ring's new length and reach (good: false too if a turn is not decided).
// Near-cocircular lattices need it, half of whose diagonals stay on the stack (handing such points on
// instead: 62,500 squares with a jitter of 1e-6 354 us, 111 in the incremental kernels, 118 so); out of
// line, since it is rare elsewhere.
template <typename T, bool GEN> struct Settled {
    Reach<T, GEN> R;
    int m;
    unsigned u32, u64, mism;
};
template <typename T, bool GEN, bool SMALL>
__device__ __noinline__ Settled<T, GEN> settle_ring(StarMem<T, SMALL> *M, int t, const SetDesc *S, const double2 *P, double2 p,
                                                    int self, int m, unsigned unsure, bool check)
{
    auto ord = [&](int k) { return M->o[k + 1][t]; };
    Settled<T, GEN> r{ Reach<T, GEN>(*S), m, 0, 0, 0 };
    while (unsure) {
        const int k = 31 - __clz(unsure);
        unsure ^= 1u << k;
        const int ka = ord(k > 0 ? k - 1 : m - 1), kb = ord(k), kc = ord(k + 1 < m ? k + 1 : 0);
        const typename Prec<T>::T2 a = M->q[ka][t], b = M->q[kb][t], c = M->q[kc][t];
        T o, bnd;
        turn<T>(a, b, c, err1<T>(a), err1<T>(b), err1<T>(c), o, bnd);
        if (o > bnd && !check) continue;   // (a neighbour of one that left)
        const int e = star_recheck<GEN, false>(P, S, p, star_slot(*M, t, *S, self, ka), star_slot(*M, t, *S, self, kb),
                                               star_slot(*M, t, *S, self, kc));
        if (o > bnd) {
            r.mism += e < 0;
            continue;
        }
        ++r.u32;
        r.u64 += e == 0;
        if (e > 0) continue;
        if (e < 0) {
            for (int j = k; j + 1 < m; ++j) M->o[j + 1][t] = M->o[j + 2][t];
            --m;
        }
        if (e == 0 || m < 3) {
            r.R.good = false;
            return r;
        }
        const unsigned below = (1u << k) - 1u;
        unsure = (unsure & below) | ((unsure >> 1) & ~below) | 1u << (k > 0 ? k - 1 : m - 1) | 1u << (k < m ? k : 0);
    }
    r.m = m;
    for (int k = 0; k < m; ++k) {
        const typename Prec<T>::T2 b = M->q[ord(k)][t], c = M->q[ord(k + 1 < m ? k + 1 : 0)][t];
        r.R.add(b, c, err1<T>(b), err1<T>(c));
    }
    return r;
}

template <typename T, bool IDX, bool GEN, bool SMALL, bool CHECK>
struct Star {
    typedef Prec<T> PR;
    typedef typename PR::T2 V2;
    const RingArgs &A;
    const SetDesc &S;
    StarMem<T, SMALL> &M;
    const int t;
    double2 p;
    int self;        // own slot (build) or index (repair)
    int ocx, ocy;
    double fx, fy;
    int status = S_TODO;
    // window of cells relative to the own cell, and its row ranges
    int x0 = 0, x1 = 0, y0 = 0, y1 = 0, nseg = 0, total = 0;
    unsigned long long c0 = 0, c1 = 0;
    int n = 0, m = 0;
    int spare = 0;   // SMALL: the place behind the candidates gathered
    unsigned cand = 0, tests = 0, u32 = 0, u64 = 0, ins = 0, mism = 0, cells = 0;

    __device__ Star(const RingArgs &a, const SetDesc &s, StarMem<T, SMALL> &mm, double2 pp, int self_)
        : A(a), S(s), M(mm), t(threadIdx.x), p(pp), self(self_)
    {
        const double2 f = cell_pos<GEN>(S, p);
        ocx = min(max((int)floor(f.x), 0), S.xsize - 1);
        ocy = min(max((int)floor(f.y), 0), S.ysize - 1);
        fx = f.x - (double)ocx;
        fy = f.y - (double)ocy;
    }

    // the candidate at place k
    __device__ __forceinline__ int slot(int k) const { return star_slot(M, t, S, self, k); }
    // candidate number k of the order / of the ring (the sentinel is number -1)
    __device__ __forceinline__ int ord(int k) { return M.o[k + 1][t]; }
    // W cells per axis: centred on the own cell (odd W), or on its half that holds p (even W)
    __device__ __forceinline__ void window(int W)
    {
        const int h = (W - 1) >> 1;
        const bool even = (W & 1) == 0;
        x0 = -h - (even && fx < 0.5 ? 1 : 0);
        x1 = x0 + W - 1;
        y0 = -h - (even && fy < 0.5 ? 1 : 0);
        y1 = y0 + W - 1;
    }

    __device__ __forceinline__ void add_seg(int row, int xa, int row2, int xb)
    {
        const int base = S.cell_base;
        const int s = __ldg(&A.cstart[base + row * S.xsize + xa]);
        const int c = __ldg(&A.cstart[base + row2 * S.xsize + xb + 1]) - s;
        if (c <= 0) return;
        total += c;
        if (nseg >= STAR_SEGS || c > STAR_SEG_MAX) {
            nseg = STAR_SEGS + 1;
            return;
        }
        if (SMALL) {
            // The offsets from the own slot must fit 16 bits as gather() takes them: the nearest way
            // round the set's slots if the warp wraps, as it does where this window crosses the
            // box's edge, else the plain difference (over half of the set where most points lie in
            // a few rows).  (The nearest way in every gather instead: 4M uniform points 2.12 -> 2.17 ms.
            // Branches between the conditions: 1M lattice sites 290 -> 293 us.)
            const int d = abs(s - self);
            if ((d + c > 32767) & ((min(d, S.n - d) + c > 32767) | ((ocy + y0 >= 0) & (ocy + y1 < S.ysize)))) {
                nseg = STAR_SEGS + 1;
                return;
            }
        }
        // a stack: starts from the end of the candidate array down, counts in the 120-bit c1:c0
        ++nseg;
        M.start(nseg, t) = s;
        c1 = (c1 << 10) | (c0 >> 50);
        c0 = ((c0 << 10) & ((1ull << 60) - 1ull)) | (unsigned)c;
    }
    // the ranges of the window's rows; a window over the x seam takes the tail of one row and
    // the head of the next as one range, since they follow each other in the cell order
    __device__ __forceinline__ void build_segs()
    {
        nseg = 0;
        total = 0;
        c0 = c1 = 0;
        int xa = ocx + x0, xb = ocx + x1;
        const bool seam = xa < 0 || xb >= S.xsize;
        if (xa < 0) xa += S.xsize;
        if (xb >= S.xsize) xb -= S.xsize;
        if (!seam) {
#pragma unroll 1
            for (int r = y0; r <= y1; ++r) {
                const int cy = wrapi(ocy + r, S.ysize);
                add_seg(cy, xa, cy, xb);
            }
        } else {
            int prev = -1;   // row whose tail is pending
            for (int r = y0; r <= y1; ++r) {
                const int cy = wrapi(ocy + r, S.ysize);
                if (prev >= 0 && cy == prev + 1) {
                    add_seg(prev, xa, cy, xb);
                } else {
                    if (prev >= 0) add_seg(prev, xa, prev, S.xsize - 1);
                    add_seg(cy, 0, cy, xb);
                }
                prev = cy;
            }
            add_seg(prev, xa, prev, S.xsize - 1);
        }
    }

    // candidates of the ranges into shared memory.  r2: largest |d|^2 taken; nw > 0: only those
    // that may lie in one of the nw circles {2c} held in q[31 - k], wmax the largest diameter.
    // WRAP: some lane's window crosses the box's edge (elsewhere an offset is the plain
    // difference: both points lie in the box and less than half of it apart)
    template <bool WRAP>
    __device__ __forceinline__ void gather(T r2, int nw, T wmax, int &near, T &ndmin, T &ndmax)
    {
        n = 0;
        near = 0;
        ndmin = PR::inf();
        ndmax = (T)0;
        // The ranges are taken from the last (lowest start word) on.  Without a cut the total fits
        // and every range left holds a candidate at least, so a candidate never reaches the words
        // of the ranges still to come; else the capacity leaves them alone.
        // (SMALL leaves a place for the sentinel; the point itself is in the total)
        const int cap = total <= STAR_CAP ? STAR_CAP - nw - (SMALL ? 1 : 0) : STAR_CAP - max(nw, nseg);
        int seg = nseg, left = 0, sl = 0, id = -1, shift = self;
        double2 c = make_double2(0.0, 0.0);
        // the next candidate's position is loaded a step ahead of its use
        auto next = [&]() {
            if (left == 0) {
                if (seg == 0) {
                    id = -1;
                    return;
                }
                sl = M.start(seg, t);
                if (SMALL && WRAP) {
                    // the nearest way round the set's slots
                    shift = self;
                    if (2 * (sl - self) > S.n) shift += S.n;
                    else if (2 * (sl - self) < -S.n) shift -= S.n;
                }
                --seg;
                left = (int)(c0 & 1023u);
                c0 = (c0 >> 10) | ((c1 & 1023u) << 50);
                c1 >>= 10;
            }
            id = sl++;
            --left;
            if (IDX) id = __ldg(&A.sidx[id]);
            c = __ldg(IDX ? &A.pos[id] : &A.spos[id]);
        };
        next();
        while (id >= 0) {
            const int cur = id, off = id - shift;
            double2 d64;
            if (GEN) d64 = gen_off(c, p, S);
            else if (WRAP) d64 = make_double2(wrap_off(c.x, p.x, S.Lx, S.hLx), wrap_off(c.y, p.y, S.Ly, S.hLy));
            else d64 = make_double2(__dsub_rn(c.x, p.x), __dsub_rn(c.y, p.y));
            next();
            const T dx = PR::from64(d64.x), dy = PR::from64(d64.y);
            const T nd = dx * dx + dy * dy;
            // not the point itself (nor one that coincides with it)
            bool keep = cur != self && nd <= r2 && !(d64.x == 0.0 && d64.y == 0.0);
            if (nw > 0 && keep) {
                const T tol = -(fabs(dx) + fabs(dy)) * wmax * (T)0.00390625;   // 2^-8 |d| wmax
                keep = false;
                for (int k = 0; k < nw; ++k) {
                    const V2 w = M.q[STAR_CAP - 1 - k][t];
                    keep |= dx * w.x + dy * w.y - nd > tol;
                }
            }
            if (!keep) continue;
            if (n >= cap) {
                status = S_FAIL;
                break;
            }
            const T iv = rcp_fast(nd);
            M.q[n][t] = PR::mk2(dx * iv, dy * iv);
            M.s[n][t] = SMALL ? off : cur;
            if (nd < ndmin) {
                ndmin = nd;
                near = n;
            }
            ndmax = nd > ndmax ? nd : ndmax;
            ++n;
        }
    }

    // keys of the candidates, sorted by angle from the nearest one; the order goes to shared
    // memory.  dropped: largest |d'|^2 of a candidate dropped for its angle (0: none)
    __device__ __forceinline__ void sort(int near, T &dropped)
    {
        dropped = (T)0;
        const V2 q0 = M.q[near][t];
        const unsigned key0 = angle_key((float)q0.x, (float)q0.y);
        unsigned key[STAR_CAP];
#pragma unroll
        for (int k = 0; k < STAR_CAP; ++k) {
            const V2 q = M.q[k][t];
            const unsigned a = angle_key((float)q.x, (float)q.y) - key0 + (unsigned)k;
            key[k] = k < n ? a : 0xffffffffu;
        }
        OeSort<0, STAR_CAP>::run(key);
        if (status != S_TODO) return;   // a finished lane keeps its order
#pragma unroll
        for (int k = 0; k < STAR_CAP; ++k) M.o[k + 1][t] = (unsigned char)key[k];   // (bits 5..8 are 0)
        unsigned gap = 0xffffffffu;
#pragma unroll
        for (int k = 0; k + 1 < STAR_CAP; ++k) gap = min(gap, key[k + 1] - key[k] - 1u);
        // padding keys end the full turn, so the last gap closes it; without padding:
        if (n == STAR_CAP) gap = min(gap, 0u - key[STAR_CAP - 1]);
        if (gap >= STAR_ANGLE_TOL) return;
        // rare: angles that may be out of order
        unsigned close = 0u, last = 0u;
#pragma unroll
        for (int k = 0; k < STAR_CAP; ++k) {
            if (k < n) last = key[k];
            if (k > 0 && k < n && key[k] - key[k > 0 ? k - 1 : 0] - 1u < STAR_ANGLE_TOL) close |= 1u << k;
        }
        T drop = (T)0;
        n = settle_angles<T, SMALL>(&M, t, n, close, 0u - last - 1u <= STAR_ANGLE_TOL, &drop);
        dropped = drop;
        if (n < 3) status = S_FAIL;
    }

    // the float64 answer (for candidates at these places): +1 left, -1 right, 0 undecided
    __device__ __forceinline__ int recheck(int ka, int kb, int kc)
    {
        return star_recheck<GEN, false>(IDX ? A.pos : A.spos, &S, p, slot(ka), slot(kb), slot(kc));
    }

    // Graham pass over the sorted candidates, the stack in place of the order: the ring is
    // then order[0 .. m).  Only a certain right turn pops, so what is popped is interior; a turn
    // that is not certainly left may stay and is settled by certify() if it is still there at the
    // end.  The stack begins with the mirror image of the first candidate: the turn there is the
    // side of the next direction, and a pop there means an open ring.
    __device__ __forceinline__ void hull()
    {
        if (status != S_TODO) return;   // a finished lane keeps its ring
        const int first = ord(0);
        if (!CHECK) {
            // A pass without a stack first: a candidate at a certain right turn between the last one
            // kept and the next one is interior.  It drops more than half of them at half the
            // instructions that the pass with the stack spends on one (4M uniform points: 1.42 ->
            // 1.28 ms; a second such pass gains nothing, and unrolled over the sorted keys it lost 6%
            // to instruction fetch).  Check mode leaves every decision to the loop that counts them.
            M.o[n + 1][t] = (unsigned char)first;
            int kept = 0, cur = ord(1);
            V2 a = M.q[first][t], b = M.q[cur][t];
            T ea = err1<T>(a), eb = err1<T>(b);
#pragma unroll 1
            for (int k = 1; k < n; ++k) {
                const int next = ord(k + 1);
                const V2 c = M.q[next][t];
                const T ec = err1<T>(c);
                T o, bnd;
                turn<T>(a, b, c, ea, eb, ec, o, bnd);
                if (!(o < -bnd)) {
                    ++kept;
                    M.o[kept + 1][t] = (unsigned char)cur;
                    a = b;
                    ea = eb;
                }
                b = c;
                eb = ec;
                cur = next;
            }
            tests += (unsigned)(n - 1);
            n = kept + 1;
        }
        V2 b = M.q[first][t], a = PR::mk2(-b.x, -b.y);
        const int sentinel = SMALL ? spare : STAR_CAP;
        M.q[sentinel][t] = a;
        M.o[0][t] = (unsigned char)sentinel;
        M.o[n + 1][t] = (unsigned char)first;
        int top = 0, i = 1, ci = ord(1);
        V2 c = M.q[ci][t];
        T ea = err1<T>(b), eb = ea, ec = err1<T>(c);
        bool pop;
        for (;;) {
            T o, bnd;
            turn<T>(a, b, c, ea, eb, ec, o, bnd);
            pop = o < -bnd;
            if (CHECK && pop && top > 0) mism += recheck(ord(top - 1), ord(top), ci) > 0;
            if (pop ? top == 0 : i >= n) break;
            // one load serves both: the candidate below the new top, or the next in the order
            const int e = ord(pop ? top - 2 : i + 1);
            const V2 l = M.q[e][t];
            const T el = err1<T>(l);
            if (!pop) M.o[top + 2][t] = (unsigned char)ci;
            top += pop ? -1 : 1;
            i += pop ? 0 : 1;
            const V2 pa = a, pb = b;
            const T pe = ea, pf = eb;
            a = pop ? l : pb;
            ea = pop ? el : pf;
            b = pop ? pa : c;
            eb = pop ? pe : ec;
            c = pop ? c : l;
            ec = pop ? ec : el;
            ci = pop ? ci : e;
        }
        m = top + 1;
        tests += (unsigned)(2 * i - m);
        ins += (unsigned)(i - 1);
        if (pop || m < 3) status = S_FAIL;   // open
    }

    // The circles of the ring (2 x centre = the pole of the line through a' and b'): S_OK when they
    // all lie inside the window and within |d|^2 <= r2.  Otherwise the window they reach, with
    // the circles in q[31 - k] and the largest diameter in wmax; S_FAIL when some circle is not
    // bounded (ill-conditioned or open) or that window is too large.  leave: only the
    // verdict is wanted.
    __device__ __forceinline__ void certify(T r2, T dropped, bool leave, bool again, T &wmax)
    {
        Reach<T, GEN> R(S);
        V2 a = M.q[ord(m - 1)][t], b = M.q[ord(0)][t];
        T ea = err1<T>(a), eb = err1<T>(b);
        unsigned unsure = 0;
        for (int k = 0; k < m; ++k) {
            const V2 c = M.q[ord(k + 1 < m ? k + 1 : 0)][t];
            const T ec = err1<T>(c);
            T o, bnd;
            turn<T>(a, b, c, ea, eb, ec, o, bnd);
            unsure |= (unsigned)!(o > bnd) << k;
            R.add(b, c, eb, ec);
            a = b;
            b = c;
            ea = eb;
            eb = ec;
        }
        // turns of the ring the filter left open: in float64
        if (CHECK) unsure = m == 32 ? ~0u : (1u << m) - 1u;
        if (R.good && unsure) {
            const Settled<T, GEN> r = settle_ring<T, GEN, SMALL>(&M, t, &S, IDX ? A.pos : A.spos, p, self, m, unsure, CHECK);
            R = r.R;
            m = r.m;
            u32 += r.u32;
            u64 += r.u64;
            mism += r.mism;
        }
        const T ulo = R.ulo, uhi = R.uhi, vlo = R.vlo, vhi = R.vhi;
        const bool good = R.good;
        wmax = R.wmax;
        if (!good || !(wmax < (T)1e15) || (dropped > (T)0 && !(wmax * wmax * dropped < (T)8))) {
            status = S_FAIL;
            return;
        }
        // cells reached (the extents are twice those of the circles), widened far beyond rounding
        const T eu0 = (T)0.5 * ulo, eu1 = (T)0.5 * uhi, ev0 = (T)0.5 * vlo, ev1 = (T)0.5 * vhi;
        const T hxs = (T)0.5 * (T)S.xsize, hys = (T)0.5 * (T)S.ysize;
        const T sk = A.skin ? (T)*A.skin : (T)0;
        const T mg = (T)1e-4 + sk;
        const T a0 = (T)fx + eu0 - mg, a1 = (T)fx + eu1 + mg, b0 = (T)fy + ev0 - mg, b1 = (T)fy + ev1 + mg;
        // circles past half the box: minimum-image offsets are not unique there (the incremental
        // path decides and flags it)
        if (eu0 < -hxs || eu1 > hxs || ev0 < -hys || ev1 > hys) {
            status = S_FAIL;
            return;
        }
        const bool in_cut = wmax * wmax <= r2;
        if (in_cut && a0 >= (T)x0 && a1 <= (T)(x1 + 1) && b0 >= (T)y0 && b1 <= (T)(y1 + 1)) {
            status = S_OK;
            return;
        }
        if (again || m > STAR_CAP / 2) {
            status = S_FAIL;
            return;
        }
        if (SMALL || leave) return;
        x0 = (int)floor(a0);
        x1 = (int)floor(a1);
        y0 = (int)floor(b0);
        y1 = (int)floor(b1);
        if (x1 - x0 >= S.xsize || y1 - y0 >= S.ysize || x1 - x0 > 63 || y1 - y0 >= STAR_SEGS) {
            status = S_FAIL;
            return;
        }
        // the circles to the top of q, by way of the candidate array (as float pairs)
        a = M.q[ord(0)][t];
        for (int k = 0; k < m; ++k) {
            const V2 c = M.q[ord(k + 1 < m ? k + 1 : 0)][t];
            const T ig = rcp_fast(a.x * c.y - a.y * c.x);
            M.s[SMALL ? 0 : 2 * k][t] = __float_as_int((float)((c.y - a.y) * ig));
            M.s[SMALL ? 0 : 2 * k + 1][t] = __float_as_int((float)((a.x - c.x) * ig));
            a = c;
        }
        for (int k = 0; k < m; ++k)
            M.q[STAR_CAP - 1 - k][t] = PR::mk2((T)__int_as_float(M.s[SMALL ? 0 : 2 * k][t]), (T)__int_as_float(M.s[SMALL ? 0 : 2 * k + 1][t]));
    }

    // the window of the first pass
    __device__ __forceinline__ void first_window(T &r2)
    {
        int W = S.star_win;
        if (S.xsize < W + 1 || S.ysize < W + 1) {
            status = S_FAIL;
            return;
        }
        window(W);
        build_segs();
        if (total > STAR_CAP) {
            // denser than the set's mean: the smallest window that holds a disc of STAR_TARGET
            // candidates at the local density, cut to that disc
            const float disc = (float)STAR_TARGET / 3.14159265f;
            const int V = max(3, (int)ceilf(1.0f + 2.0f * sqrtf(disc * (float)(W * W) / (float)total)));
            if (V < W) {
                W = V;
                window(W);
                build_segs();
            }
            if (total > STAR_CAP) {
                const T area = GEN ? (T)fabs(S.m11 * S.m22 - S.m12 * S.m21) / ((T)S.xsize * (T)S.ysize)
                                   : (T)(S.cw * S.ch);
                r2 = (T)(disc * (float)(W * W) / (float)total) * area;
            }
        }
        cells += (unsigned)(W * W);
        if (nseg > STAR_SEGS || total > A.work_budget || total < 4) status = S_FAIL;
    }
    // the window of the second pass (set by certify)
    __device__ __forceinline__ void second_window()
    {
        build_segs();
        cells += (unsigned)((x1 - x0 + 1) * (y1 - y0 + 1));
        if (nseg > STAR_SEGS || total > A.work_budget) status = S_FAIL;
    }
    // whether an offset from the window may have to go round the box
    __device__ __forceinline__ bool wraps() const
    {
        return ocx + x0 < 0 || ocx + x1 >= S.xsize || ocy + y0 < 0 || ocy + y1 >= S.ysize ||
               2 * (max(-x0, x1) + 1) > S.xsize || 2 * (max(-y0, y1) + 1) > S.ysize;
    }

    // one pass: candidates, angular order, hull
    __device__ __forceinline__ void pass(T r2, int nw, T wmax, T &dropped)
    {
        int near = 0;
        T ndmin = (T)1, ndmax = (T)1;
        // (cell lists older than the positions may list a point across the edge)
        const bool wrap = IDX || __any_sync(0xffffffffu, status == S_TODO && wraps());
        if (status == S_TODO) {
            cand += (unsigned)total;
            if (IDX || GEN || wrap) gather<true>(r2, nw, wmax, near, ndmin, ndmax);
            else gather<false>(r2, nw, wmax, near, ndmin, ndmax);
            // a safe range for squares and reciprocals, and enough for a ring
            if (status == S_TODO && (n < 3 || !(ndmin > (T)1e-30) || !(ndmax < (T)1e30))) status = S_FAIL;
        }
        if (SMALL) spare = min(n, STAR_CAP - 1);
        __syncwarp();
        sort(near, dropped);
        __syncwarp();
        hull();
    }

    // Every lane of the warp calls these (votes inside); active: lanes with a point.  Afterwards
    // status is S_OK, S_FAIL, or (first pass only) S_TODO with the ring of the pass
    __device__ __forceinline__ void run(int mode, bool active)
    {
        if (!active) status = S_FAIL;
        T r2 = PR::inf(), wmax = (T)0, dropped = (T)0;
        if (mode != STAR_SECOND) {
            if (status == S_TODO) first_window(r2);
            pass(r2, 0, wmax, dropped);
            if (status == S_TODO) certify(r2, dropped, mode == STAR_FIRST, false, wmax);
            if (mode == STAR_FIRST || !__any_sync(0xffffffffu, status == S_TODO)) return;
        } else if (status == S_TODO) {
            // the first pass's ring is in place: its circles
            certify((T)0, (T)0, false, false, wmax);
        }
        const int nw = m;
        // the second pass's circles lie inside these
        r2 = wmax * wmax * (T)1.0078125;
        if (status == S_TODO) second_window();
        pass(r2, nw, wmax, dropped);
        if (status == S_TODO) certify(r2, dropped, false, true, wmax);
    }

    // second pass: the ring of the first as the candidates 0 .. m - 1
    __device__ __forceinline__ void load_ring(const int *row)
    {
        m = *row++;
        for (int k = 0; k < m; ++k) {
            const int sl = row[k];
            const double2 c = __ldg(&A.spos[sl]);
            double2 d64;
            if (GEN) d64 = gen_off(c, p, S);
            else d64 = make_double2(wrap_off(c.x, p.x, S.Lx, S.hLx), wrap_off(c.y, p.y, S.Ly, S.hLy));
            const T dx = PR::from64(d64.x), dy = PR::from64(d64.y);
            const T iv = rcp_fast(dx * dx + dy * dy);
            M.q[k][t] = PR::mk2(dx * iv, dy * iv);
        }
        for (int k = 0; k < m; ++k) {
            M.s[SMALL ? 0 : k][t] = row[k];
            M.o[k + 1][t] = (unsigned char)k;
        }
    }
};

template <typename T, int MODE, bool IDX, bool GEN, bool SMALL, bool CHECK>
// (SMALL in general boxes: without the bound 106 registers, four blocks per SM instead of five, and
// 454 us for 1M points instead of 318; in rectangles it has 96 without one, and the bound makes 4M
// points 2.06 -> 2.09 ms.  0: no bound, which is not the same as 1.)
__global__ void __launch_bounds__(SMALL ? 128 : STAR_BLOCK, SMALL && GEN ? 5 : 0) k_star(RingArgs A)
{
    __shared__ StarMem<T, SMALL> M;
    constexpr int B = StarMem<T, SMALL>::B;
    const int t = threadIdx.x;
    Ctr ctr = { 0, 0, 0, 0, 0, 0, 0 };
    unsigned pts = 0;
    int maxr = 0;
    const int n = MODE == STAR_SECOND ? min(*A.second_count, A.second_cap) : item_count(A);
    if (A.count_round && blockIdx.x == 0 && t == 0 && n > 0) {
        atomicAdd(&A.st->repaired, (unsigned long long)n);
        atomicMax(&A.st->rounds, A.round + 1);
    }
    if (IDX && n <= A.wrap_items) return;   // a short list: k_wrap takes it
    const int mode = IDX && n <= A.star_once ? STAR_FIRST : MODE;
    if ((int)blockIdx.x * B >= n) return;
    for (int base = blockIdx.x * B; base < n; base += gridDim.x * B) {
        const int it = base + t;
        const bool act = it < n;
        int pid = -1, slot = -1;
        if (act) {
            if (IDX) pid = A.worklist[it];
            else slot = MODE == STAR_SECOND ? A.second_list[it] : A.item_base + it;
        }
        const SetDesc &S = A.sets[(act && A.set_of) ? __ldg(&A.set_of[IDX ? pid : slot]) : 0];
        const double2 p = !act ? make_double2(0.0, 0.0) : (IDX ? __ldg(&A.pos[pid]) : __ldg(&A.spos[slot]));
        Star<T, IDX, GEN, SMALL, CHECK> b(A, S, M, p, IDX ? pid : slot);
        if (act && !IDX) pid = __ldg(&A.sidx[slot]);
        if (MODE == STAR_SECOND && act) b.load_ring(second_ring(A, it));
        b.run(mode, act);
        if (act) {
            StarRing<T, SMALL> ring{ M, t };
            if (b.status == S_OK) {
                pts++;
                // (four loads in flight: 4M uniform points 1.68 -> 1.61 ms)
                for (int k = 0; k < b.m; k += 4) {
                    int e[4];
#pragma unroll
                    for (int j = 0; j < 4; ++j) e[j] = b.slot(k + j < b.m ? b.ord(k + j) : b.ord(k));
#pragma unroll
                    for (int j = 0; j < 4; ++j)
                        if (!IDX) e[j] = __ldg(&A.sidx[e[j]]);
#pragma unroll
                    for (int j = 0; j < 4; ++j)
                        if (k + j < b.m) ring.set(k + j, e[j]);
                }
                if (IDX) finish_repair(A, pid, ring, b.m);
                store_ring(A, pid, ring, b.m, maxr);
            } else {
                // not certified: the ring's slots wait for the second pass
                int at = A.second_cap;
                if (MODE == STAR_FIRST && b.status == S_TODO && b.m < STAR_RING) at = atomicAdd(A.second_count, 1);
                if (at < A.second_cap) {
                    A.second_list[at] = slot;
                    int *row = second_ring(A, at);
                    row[0] = b.m;
                    for (int k = 0; k < b.m; ++k) row[k + 1] = b.slot(b.ord(k));
                } else {
                    A.star_list[atomicAdd(A.star_count, 1)] = pid;
                }
            }
        }
        ctr.cand += b.cand;
        ctr.tests += b.tests;
        ctr.u32 += b.u32;
        ctr.u64 += b.u64;
        ctr.ins += b.ins;
        ctr.mism += b.mism;
        ctr.cells += b.cells;
        __syncwarp();
    }
    flush_counters(A, ctr, pts, maxr);
}

template <typename T, int MODE, bool IDX, bool GEN, bool SMALL>
cudaError_t launch_star_t(const RingArgs &a, int sms, cudaStream_t s)
{
    constexpr int B = StarMem<T, SMALL>::B;
    int blocks = (a.n_items + B - 1) / B;
    const int most = sms * (SMALL ? 5 : 8);
    if (blocks > most) blocks = most;
    if (a.check) k_star<T, MODE, IDX, GEN, SMALL, true><<<blocks, B, 0, s>>>(a);
    else k_star<T, MODE, IDX, GEN, SMALL, false><<<blocks, B, 0, s>>>(a);
    return cudaGetLastError();
}

template <typename T, bool GEN>
cudaError_t launch_star_g(const RingArgs &a, int sms, int *launches, cudaStream_t s)
{
    *launches += 1;
    if (a.cand_by_index) return launch_star_t<T, STAR_BOTH, true, GEN, false>(a, sms, s);
    cudaError_t e;
    if (sizeof(T) == 4 && a.star_small) e = launch_star_t<T, STAR_FIRST, false, GEN, sizeof(T) == 4>(a, sms, s);
    else e = launch_star_t<T, STAR_FIRST, false, GEN, false>(a, sms, s);
    if (e != cudaSuccess || a.second_cap <= 0) return e;
    *launches += 1;
    return launch_star_t<T, STAR_SECOND, false, GEN, false>(a, sms, s);
}

}  // namespace

cudaError_t launch_star(const RingArgs &a, int mode, int sms, int *launches, cudaStream_t s)
{
    if (a.n_items <= 0) return cudaSuccess;
    if (a.general) return mode == MODE_F64 ? launch_star_g<double, true>(a, sms, launches, s) : launch_star_g<float, true>(a, sms, launches, s);
    return mode == MODE_F64 ? launch_star_g<double, false>(a, sms, launches, s) : launch_star_g<float, false>(a, sms, launches, s);
}

}  // namespace dgt
