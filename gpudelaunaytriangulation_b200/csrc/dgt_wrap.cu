// One-ring construction with a warp per point (k_wrap): builds of few points, the points that
// the thread-per-point first stage (dgt_star.cu) cannot finish, and the rebuild rounds.
//
// The ring is the convex hull of the candidates' inverted offsets (dgt_star.cuh).  The 32 lanes
// gather the candidates of a window of cells (one range of the cell order per row) and walk
// round the hull: from a vertex a', the next one is the candidate with the smallest slope in the
// frame of a' (one warp-wide minimum), and every other candidate must then lie certainly to the
// left of the edge, so each accepted edge is a hull edge whatever the rounding of the slopes
// (undecided turns go to float64 and exact arithmetic; an exactly cocircular candidate hands the
// point on).  Afterwards one lane per edge computes its circle.  While some circle reaches out
// of the window the window grows towards the circles' cells, at most tripling per pass, and only
// candidates that may lie inside a circle join the ring for the next walk: a candidate outside
// every circle stays outside, since the union of the circles only shrinks.  A ring that is open
// in its first window takes four virtual corners along, like the incremental kernels.
//
// What bounds it: the latency of one point's chain (some 2000 instructions, a few microseconds,
// against 95 us for a point of the incremental thread-per-point kernel) while the points fit the
// chip at once, instruction issue beyond (53% of the issue slots at 10,000 points).  1,000 points:
// 20 us against 96 us; 10,000: 42 us against 117 us.
#include "dgt_star.cuh"

namespace dgt {

namespace {

constexpr int WRAP_CAP = 128;      // candidates of one pass
constexpr int WRAP_K = WRAP_CAP / 32;
constexpr int WRAP_WARPS = 4;      // points per block
constexpr int WRAP_PASSES = 64;
constexpr float WRAP_TARGET = 50.0f;   // candidates a first window is sized for
// Points whose circles reach over more cells per axis, or that scan more candidates, go to the
// incremental warp kernel, which skips empty space by occupancy blocks and scans nearest tiles
// first (points in the voids between dense clusters, and on their rims).  Geometric mean over
// twelve clustered sets of 0.25 to 1M points: 3.29 / 3.17 / 3.24 / 3.53 / 3.69 ms at 48 / 70 / 100 /
// 300 / 900 cells, 4.77 without the first limit; at 70 cells and 8,192 / 16,384 / 32,768 candidates
// 3.50 / 3.17 / 3.18 ms.
constexpr int WRAP_REACH = 71;
constexpr unsigned WRAP_WORK = 16384;
constexpr unsigned FULL = 0xffffffffu;

template <typename T> struct WrapMem {
    typedef typename Prec<T>::T2 V2;
    V2 q[WRAP_CAP];        // inverted offsets
    int id[WRAP_CAP];      // slot (build) or index (repair); negative: virtual corner
    float2 w[32];          // circles of the ring (2 x centre)
    float d[32];           // their diameters, rounded up
    unsigned char ring[32];
    int row[32];           // per non-empty range of the rows at hand: first slot less its place in the sequence
};

// floats ordered as unsigned integers
__device__ __forceinline__ unsigned ordered(float x)
{
    const unsigned b = __float_as_uint(x);
    return b ^ ((unsigned)((int)b >> 31) | 0x80000000u);
}
__device__ __forceinline__ float unordered(unsigned k)
{
    return __uint_as_float(k & 0x80000000u ? k ^ 0x80000000u : ~k);
}
__device__ __forceinline__ float warp_min(float x) { return unordered(__reduce_min_sync(FULL, ordered(x))); }
__device__ __forceinline__ float warp_max(float x) { return unordered(__reduce_max_sync(FULL, ordered(x))); }

// W_HEAVY: not done because its scan would be too large here too
enum { W_OK = 0, W_FAIL = 1, W_HEAVY = 2 };

template <typename T, bool IDX, bool GEN>
struct Wrap {
    typedef Prec<T> PR;
    typedef typename PR::T2 V2;
    const RingArgs &A;
    const SetDesc &S;
    WrapMem<T> &M;
    const int lane;
    const double2 p;
    const int self;
    int ocx, ocy;
    float fx, fy, skin;
    int n = 0, m = 0;
    unsigned cand = 0, tests = 0, u32 = 0, u64 = 0, ins = 0, mism = 0, cells = 0;

    __device__ __forceinline__ Wrap(const RingArgs &a, const SetDesc &s, WrapMem<T> &mm, int ln, double2 pp, int self_)
        : A(a), S(s), M(mm), lane(ln), p(pp), self(self_)
    {
        const double2 f = cell_pos<GEN>(S, p);
        ocx = min(max((int)floor(f.x), 0), S.xsize - 1);
        ocy = min(max((int)floor(f.y), 0), S.ysize - 1);
        fx = (float)(f.x - (double)ocx);
        fy = (float)(f.y - (double)ocy);
        skin = A.skin ? *A.skin : 0.0f;
    }

    // the columns [a, b] of `row` that the circles reach (relative to the own cell), within [x0, x1]
    __device__ __forceinline__ void row_reach(int row, int &a, int &b) const
    {
        const float mg = skin + 1e-3f;
        const float ylo = ((float)row - fy - mg) * (float)S.ch, yhi = ((float)(row + 1) - fy + mg) * (float)S.ch;
        float lo = 3e38f, hi = -3e38f;
        for (int k = 0; k < m; ++k) {
            const float2 w = M.w[k];
            const float cy = 0.5f * w.y, r = 0.5f * M.d[k];
            const float dy = fmaxf(fmaxf(ylo - cy, cy - yhi), 0.0f);
            const float h2 = (r - dy) * (r + dy);
            if (h2 >= 0.0f) {
                const float h = sqrt_over(h2);
                lo = fminf(lo, 0.5f * w.x - h);
                hi = fmaxf(hi, 0.5f * w.x + h);
            }
        }
        const float icw = (float)S.icw;
        const float la = fx + lo * icw, lb = fx + hi * icw;
        const float slack = mg + 1e-6f * (fabsf(la) + fabsf(lb));
        // (compared as floats: the extents may be far outside the integers)
        if (la - slack > (float)a) a = la - slack > (float)b ? b + 1 : (int)floorf(la - slack);
        if (lb + slack < (float)(b + 1)) b = lb + slack < (float)a ? a - 1 : (int)floorf(lb + slack);
    }

    // candidates of the window's cells behind the n already there; r2: largest |d|^2 taken; filter:
    // only those that may lie in one of the m circles.  False when they do not all fit (or `most`
    // candidates were in the window)
    __device__ __forceinline__ bool gather(int x0, int x1, int y0, int y1, T r2, bool filter, int most)
    {
        const bool seam = ocx + x0 < 0 || ocx + x1 >= S.xsize;
        const int per = seam ? 16 : 32;   // rows a turn: a row over the edge has two parts
        // (a window over a whole axis takes every cell: a row or column of it stands for two distances
        // from the point, the one it is listed at and the nearest, which candidates are taken at)
        const bool tight = !GEN && filter && y1 - y0 >= 8 && y1 - y0 + 1 < S.ysize && x1 - x0 + 1 < S.xsize;
        const int known = n;
        bool odd = false;
        for (int r0 = y0; r0 <= y1; r0 += per) {
            const int row = r0 + (seam ? lane >> 1 : lane);
            int start = 0, cnt = 0;
            if (row <= y1) {
                int a = x0, b = x1;
                if (tight) row_reach(row, a, b);
                int ca = ocx + a, cb = ocx + b;
                if (seam && (lane & 1)) {
                    // the part on the other side of the box's edge
                    if (ocx + x0 < 0) {
                        cb = min(cb, -1) + S.xsize;
                        ca += S.xsize;
                    } else {
                        ca = max(ca, S.xsize) - S.xsize;
                        cb -= S.xsize;
                    }
                } else {
                    ca = max(ca, 0);
                    cb = min(cb, S.xsize - 1);
                }
                if (ca <= cb) {
                    const int base = S.cell_base + wrapi(ocy + row, S.ysize) * S.xsize;
                    start = __ldg(&A.cstart[base + ca]);
                    cnt = __ldg(&A.cstart[base + cb + 1]) - start;
                }
            }
            int incl = cnt;
            for (int o = 1; o < 32; o <<= 1) {
                const int v = __shfl_up_sync(FULL, incl, o);
                if (lane >= o) incl += v;
            }
            const int total = __shfl_sync(FULL, incl, 31), excl = incl - cnt;
            cand += (unsigned)total;
            if (total > most) return false;
            most -= total;
            // candidate j of the sequence belongs to the last non-empty range that begins at or before
            // it: the ranges' offsets in a table, the beginnings within 32 candidates as bits
            const unsigned filled = __ballot_sync(FULL, cnt > 0);
            __syncwarp();
            if (cnt > 0) M.row[__popc(filled & ((1u << lane) - 1u))] = start - excl;
            __syncwarp();
            for (int base = 0; base < total; base += 32) {
                const int j = base + lane, at0 = excl - base;
                const unsigned begins = __reduce_or_sync(FULL, cnt > 0 && (unsigned)at0 < 32u ? 1u << at0 : 0u);
                const int before = base == 0 ? 0 : __popc(__ballot_sync(FULL, cnt > 0 && at0 < 0));
                const int rank = before - 1 + __popc(begins & (FULL >> (31 - lane)));
                int id = M.row[rank] + j;
                bool keep = j < total;
                T dx = (T)0, dy = (T)0, nd = (T)1;
                if (keep) {
                    if (IDX) id = __ldg(&A.sidx[id]);
                    const double2 c = __ldg(IDX ? &A.pos[id] : &A.spos[id]);
                    double2 d;
                    if (GEN) {
                        d = gen_off(c, p, S);
                    } else {
                        // (wrap_off with one comparison in the common case)
                        d = make_double2(__dsub_rn(c.x, p.x), __dsub_rn(c.y, p.y));
                        if (fabs(d.x) > S.hLx) d.x = wrap_off(c.x, p.x, S.Lx, S.hLx);
                        if (fabs(d.y) > S.hLy) d.y = wrap_off(c.y, p.y, S.Ly, S.hLy);
                    }
                    dx = PR::from64(d.x);
                    dy = PR::from64(d.y);
                    nd = dx * dx + dy * dy;
                    keep = id != self && nd <= r2;
                    // outside the safe range of squares and reciprocals nothing is certain here
                    // (except that a coincident point is no neighbour)
                    if (keep && !(nd > (T)1e-30 && nd < (T)1e30)) {
                        odd |= d.x != 0.0 || d.y != 0.0;
                        keep = false;
                    }
                }
                if (filter && keep) {
                    const T l1 = fabs(dx) + fabs(dy);
                    keep = false;
                    for (int k = 0; k < m; ++k) {
                        const float2 w = M.w[k];
                        keep |= dx * (T)w.x + dy * (T)w.y - nd > -l1 * (T)M.d[k] * (T)0.00390625;
                    }
                }
                if (keep)
                    for (int k = 0; k < known; ++k) keep &= M.id[k] != id;
                const unsigned got = __ballot_sync(FULL, keep);
                if (got) {
                    const int at = n + __popc(got & ((1u << lane) - 1u));
                    if (keep && at < WRAP_CAP) {
                        const T iv = rcp_fast(nd);
                        M.q[at] = PR::mk2(dx * iv, dy * iv);
                        M.id[at] = id;
                    }
                    n += __popc(got);
                    if (n > WRAP_CAP) {
                        n = __any_sync(FULL, odd) ? WRAP_CAP + 1 : WRAP_CAP;
                        return false;
                    }
                }
            }
        }
        if (__any_sync(FULL, odd)) n = WRAP_CAP + 1;
        return true;
    }

    // +1 left, -1 right, 0 on the circle
    __device__ __forceinline__ int recheck(int ka, int kb, int kc) const
    {
        return star_recheck<GEN, true>(IDX ? A.pos : A.spos, &S, p, M.id[ka], M.id[kb], M.id[kc]);
    }

    // the hull of the n <= 32 K candidates: M.ring[0 .. m).  1: done, 0: open, -1: not decided
    // here.  (A form for two candidates a lane and one for four: with the places beyond n skipped
    // at run time 10,000 points took 50 us, the compiler predicates them.)
    template <int K>
    __device__ __forceinline__ int walk()
    {
        V2 c[K];
        T ec[K];
        unsigned far = 0;
        int first = 0;
#pragma unroll
        for (int j = 0; j < K; ++j) {
            const int k = lane + 32 * j;
            c[j] = k < n ? M.q[k] : PR::mk2((T)0, (T)0);
            ec[j] = err1<T>(c[j]);
            const unsigned l = __float_as_uint((float)(c[j].x * c[j].x + c[j].y * c[j].y));
            if (l > far) {
                far = l;
                first = k;
            }
        }
        const unsigned most = __reduce_max_sync(FULL, far);
        first = __shfl_sync(FULL, first, __ffs(__ballot_sync(FULL, far == most)) - 1);
        int ka = first;
        const bool check = A.check != 0;
        m = 0;
        for (int guard = 0; guard < 2 * WRAP_CAP; ++guard) {
            const V2 a = M.q[ka];
            const T ea = err1<T>(a);
            // slope of a' -> c' in the frame (tangent, inward) of a'; only directions within half a
            // turn ahead (not the vertex itself, nor the origin that stands in for places without a
            // candidate: fused, their tangent parts are rounding errors of either sign)
            float best = 3e38f;
            int kb = -1;
            V2 v[K];
#pragma unroll
            for (int j = 0; j < K; ++j) {
                v[j] = PR::mk2(c[j].x - a.x, c[j].y - a.y);
                const float u = (float)(a.x * v[j].y - a.y * v[j].x);
                const float slope = -(float)(a.x * v[j].x + a.y * v[j].y) * rcp_fast(u);
                const int k = lane + 32 * j;
                if (u > 0.0f && slope < best && k != ka && k < n) {
                    best = slope;
                    kb = k;
                }
            }
            const unsigned key = kb >= 0 ? ordered(best) : FULL, least = __reduce_min_sync(FULL, key);
            if (least == FULL) return 0;
            const unsigned who = __ballot_sync(FULL, key == least);
            kb = __shfl_sync(FULL, kb, __ffs(who) - 1);
            // every other candidate to the left of the edge
            for (;;) {
                const V2 b = M.q[kb];
                const T eb = err1<T>(b), ux = b.x - a.x, uy = b.y - a.y;
                const T lu = fabs(ux) + fabs(uy), eab = ea + eb;
                unsigned open = 0;
#pragma unroll
                for (int j = 0; j < K; ++j) {
                    // (turn() with the differences at hand)
                    const int k = lane + 32 * j;
                    const T o = ux * v[j].y - uy * v[j].x;
                    const T bnd = (fabs(v[j].x) + fabs(v[j].y)) * eab + (lu * (ea + ec[j]) + PR::tiny());
                    open |= (unsigned)(k < n && k != ka && k != kb && (!(o > bnd) || check)) << j;
                }
                ++tests;
                unsigned lanes = __ballot_sync(FULL, open != 0);
                int right = -1;   // a candidate to the right
                while (lanes) {
                    const int src = __ffs(lanes) - 1;
                    const unsigned oj = __shfl_sync(FULL, open, src);
                    const int kc = src + 32 * (__ffs(oj) - 1);
                    const V2 cc = M.q[kc];
                    T o, bnd;
                    turn<T>(a, b, cc, ea, eb, err1<T>(cc), o, bnd);
                    const int e = recheck(ka, kb, kc);
                    if (o > bnd) {   // (check mode)
                        mism += lane == 0 && e < 0;
                    } else {
                        u32 += lane == 0;
                        if (e == 0) {
                            u64 += lane == 0;
                            return -1;
                        }
                        if (e < 0) {
                            right = kc;
                            break;
                        }
                    }
                    if (lane == src) open &= open - 1u;
                    lanes = __ballot_sync(FULL, open != 0);
                }
                if (right < 0) break;
                kb = right;
                if (++guard >= 2 * WRAP_CAP) return -1;
            }
            if (lane == 0) M.ring[m] = (unsigned char)ka;
            ++m;
            ka = kb;
            if (ka == first) {
                __syncwarp();
                return m >= 3 ? 1 : 0;
            }
            if (m >= 32) return -1;
        }
        return -1;
    }

    // the whole construction; W_OK: lane k < m holds the ring's k-th entry in `out`
    __device__ __forceinline__ int run(int &out)
    {
        // first window: about WRAP_TARGET candidates at the set's mean density, fewer cells and a
        // radius cut where the density is higher
        const int lim = min(S.xsize, S.ysize) - 1;
        int W = min(max((int)sqrtf(WRAP_TARGET / S.per_cell), 3), min(lim, 31));
        if (W < 3) return W_FAIL;
        const T cell_area = GEN ? (T)fabs(S.m11 * S.m22 - S.m12 * S.m21) / ((T)S.xsize * (T)S.ysize) : (T)(S.cw * S.ch);
        T r2 = PR::inf();
        int x0, x1, y0, y1;
        auto window = [&]() {
            const int h = (W - 1) >> 1;
            const bool even = (W & 1) == 0;
            x0 = -h - (even && fx < 0.5f ? 1 : 0);
            x1 = x0 + W - 1;
            y0 = -h - (even && fy < 0.5f ? 1 : 0);
            y1 = y0 + W - 1;
        };
        window();
        bool first = true;      // still choosing the first window
        bool filter = false;    // the ring's circles are known and bounded
        bool full = false;      // the window holds all of them
        for (int pass = 0; pass < WRAP_PASSES; ++pass) {
            // what is there already: nothing, or the ring
            n = first ? 0 : m;
            const unsigned seen = cand;
            // (a window of three cells may scan WRAP_WORK candidates: dense cells, as of a clustered set at
            // the mean spacing, 5,850 a point: 1M points 62 ms in the incremental kernels, 37 ms here)
            const bool fits = gather(x0, x1, y0, y1, r2, filter, first && W > 3 ? 8 * WRAP_CAP : (int)WRAP_WORK);
            if (n > WRAP_CAP) return W_FAIL;
            if (cand > WRAP_WORK) return W_HEAVY;
            if (first && !fits) {
                // denser here: the smallest window that holds a disc of WRAP_TARGET candidates at the
                // local density, cut to that disc; then half as many
                if (r2 == PR::inf()) r2 = (T)(WRAP_TARGET * (float)(W * W) / (3.14159265f * (float)(cand - seen))) * cell_area;
                else r2 *= (T)0.5;
                if (W == 3 && cand - seen > WRAP_WORK) return W_HEAVY;
                const float reach = sqrtf((float)(r2 / cell_area));   // in cells
                W = min(W, max(3, (int)ceilf(1.0f + 2.0f * reach)));
                window();
                continue;
            }
            cells += (unsigned)((x1 - x0 + 1) * (y1 - y0 + 1));
            // every candidate of the window that matters is there: the ring is the window's
            const bool complete = fits && r2 == PR::inf();
            __syncwarp();
            int r;
            for (bool corners = false;; corners = true) {
                r = n < 3 ? 0 : (n <= 64 ? walk<2>() : walk<WRAP_K>());
                if (r != 0 || corners) break;
                // open: with the virtual corners
                if (n + 4 > WRAP_CAP || !first) return W_FAIL;
                if (lane < 4) {
                    const double v = (double)S.V;
                    const T x = (T)((lane == 0 || lane == 3) ? v : -v), y = (T)(lane < 2 ? v : -v);
                    const T iv = rcp_fast(x * x + y * y);
                    M.q[n + lane] = PR::mk2(x * iv, y * iv);
                    M.id[n + lane] = -1 - lane;
                }
                n += 4;
                __syncwarp();
            }
            if (r != 1) return W_FAIL;
            // one lane per edge: its circle
            const int ka = lane < m ? M.ring[lane] : 0, kb = lane < m ? M.ring[lane + 1 < m ? lane + 1 : 0] : 0;
            const V2 a = M.q[ka], b = M.q[kb];
            const int id = lane < m ? M.id[ka] : 0;
            const T g = a.x * b.y - a.y * b.x;
            // (conditions and margins as in dgt_star.cu)
            bool good = g > ((T)0.001953125 / ((T)256 * PR::u() * PR::u())) * err1<T>(a) * err1<T>(b);
            const T ig = rcp_fast(g);
            float wx = (float)((b.y - a.y) * ig), wy = (float)((a.x - b.x) * ig);
            float hw = sqrt_over(wx * wx + wy * wy) * 1.00390625f;
            good = good && hw < 1e15f;
            const bool in = lane < m;
            if (in && !good) {
                // a sliver: its circle in double
                const double2 *P = IDX ? A.pos : A.spos;
                const double2 oa = star_off<GEN>(P, &S, p, id), ob = star_off<GEN>(P, &S, p, M.id[kb]);
                const double4 c = make_circ<double>(oa.x, oa.y, ob.x, ob.y);
                wx = (float)c.x;
                wy = (float)c.y;
                hw = (float)(2.0 * c.w) * 1.00390625f;
                good = c.w < 5e14;
            }
            const bool all_good = __all_sync(FULL, !in || good);
            const bool real = __all_sync(FULL, !in || id >= 0);
            float u0 = 3e38f, u1 = -3e38f, v0 = 3e38f, v1 = -3e38f;
            if (in) {
                const float uc = GEN ? (float)S.g11 * wx + (float)S.g12 * wy : wx * (float)S.icw;
                const float vc = GEN ? (float)S.g21 * wx + (float)S.g22 * wy : wy * (float)S.ich;
                const float hu = hw * (float)(GEN ? S.gnx : S.icw), hv = hw * (float)(GEN ? S.gny : S.ich);
                u0 = 0.5f * (uc - hu);
                u1 = 0.5f * (uc + hu);
                v0 = 0.5f * (vc - hv);
                v1 = 0.5f * (vc + hv);
            }
            u0 = warp_min(u0);
            u1 = warp_max(u1);
            v0 = warp_min(v0);
            v1 = warp_max(v1);
            const float hx = 0.5f * (float)S.xsize, hy = 0.5f * (float)S.ysize;
            const bool inside = all_good && real && u0 >= -hx && u1 <= hx && v0 >= -hy && v1 <= hy;
            // cells reached, widened far beyond rounding
            const float mg = 2e-4f + skin;
            const float a0 = fx + u0 - mg - 4e-7f * fabsf(u0), a1 = fx + u1 + mg + 4e-7f * fabsf(u1);
            const float b0 = fy + v0 - mg - 4e-7f * fabsf(v0), b1 = fy + v1 + mg + 4e-7f * fabsf(v1);
            const bool holds = a0 >= (float)x0 && a1 <= (float)(x1 + 1) && b0 >= (float)y0 && b1 <= (float)(y1 + 1);
            const float big = warp_max(in ? hw : 0.0f);
            // final: all candidates of the circles it began with were taken, or the circles lie in a
            // complete window, or within the first one's cut
            if ((fits && full) || (complete && holds) || (first && holds && (T)big * (T)big <= r2)) {
                out = id;
                return inside ? W_OK : W_FAIL;
            }
            // the next window: the cells the circles reach, at most three times the present extent
            // and never more than the whole axis
            const int ex = x1 - x0 + 1, ey = y1 - y0 + 1;
            full = true;
            auto grow = [&](int lo, int hi, float need_lo, float need_hi, int e, int size, int &g0, int &g1) {
                // (an unbounded circle needs everything)
                const bool in0 = all_good && need_lo >= (float)(lo - e), in1 = all_good && need_hi < (float)(hi + e + 1);
                g0 = in0 ? (int)floorf(need_lo) : lo - e;
                g1 = in1 ? (int)floorf(need_hi) : hi + e;
                if (g1 - g0 + 1 >= size) {
                    g0 = -(size >> 1);
                    g1 = g0 + size - 1;
                } else {
                    full &= in0 && in1;
                }
            };
            int gx0, gx1, gy0, gy1;
            grow(x0, x1, a0, a1, ex, S.xsize, gx0, gx1);
            grow(y0, y1, b0, b1, ey, S.ysize, gy0, gy1);
            // (unbounded in the whole box)
            if (!all_good && gx0 == x0 && gx1 == x1 && gy0 == y0 && gy1 == y1) return W_FAIL;
            if (gx1 - gx0 >= WRAP_REACH || gy1 - gy0 >= WRAP_REACH) return W_HEAVY;
            x0 = gx0, x1 = gx1, y0 = gy0, y1 = gy1;
            // the ring to the front, its circles beside it
            __syncwarp();
            if (in) {
                M.q[lane] = a;
                M.id[lane] = id;
                M.w[lane] = make_float2(wx, wy);
                M.d[lane] = hw;
            }
            __syncwarp();
            first = false;
            filter = all_good;
            r2 = PR::inf();
        }
        return W_FAIL;
    }
};

// repair: what the rebuilt ring contradicts is queued (finish_repair of dgt_builder.cuh, a lane
// per neighbour)
__device__ __forceinline__ void warp_finish_repair(const RingArgs &A, int pid, int id, int m, int lane)
{
    const int ebase = *A.epoch_ptr + 1, ep = ebase + A.round;
    const int *row = A.tri + (size_t)pid * A.stride;
    const int om = A.nn[pid];
    const int olen = om >= 1 && om <= A.stride ? om : 0;
    for (int k0 = 0; k0 < olen; k0 += 32) {
        const int o = k0 + lane < olen ? row[k0 + lane] : -1;
        bool kept = false;
        for (int j = 0; j < m; ++j) kept |= __shfl_sync(FULL, id, j) == o;
        if (!kept && o >= 0 && o < A.npoints) enqueue_next(A, ebase, ep, o);
    }
    const int pred = __shfl_sync(FULL, id, lane == 0 ? m - 1 : lane - 1);
    const int succ = __shfl_sync(FULL, id, lane + 1 < m ? lane + 1 : 0);
    if (lane < m && A.mark[id] < ebase) {
        const int mn = A.nn[id];
        bool ok = mn >= 3 && mn <= A.stride;
        const int *rr = A.tri + (size_t)id * A.stride;
        if (ok && mn <= RR) {
            Ring16 rn;
            row_load(rr, A.stride, rn);
            int pr, sc;
            ok = ring_find(rn, mn, pid, pr, sc) >= 0 && pr == succ && sc == pred;
        } else if (ok) {
            int pos = -1;
            for (int t = 0; t < mn; ++t)
                if (rr[t] == pid) pos = t;
            ok = pos >= 0 && rr[pos == 0 ? mn - 1 : pos - 1] == succ && rr[pos + 1 == mn ? 0 : pos + 1] == pred;
        }
        if (!ok) enqueue_next(A, ebase, ep, id);
    }
}

// the ring (lane k < m: its k-th entry), rotated to its smallest index, into row pid
__device__ __forceinline__ void warp_store_ring(const RingArgs &A, int pid, int id, int m, int lane, int &maxr)
{
    maxr = max(maxr, m);
    if (m > A.stride) {
        if (lane == 0) {
            atomicMax(&A.st->need_stride, m);
            A.nn[pid] = 0;   // row left unwritten: mark the ring invalid
        }
        return;
    }
    const unsigned key = lane < m ? (unsigned)id : FULL;
    const unsigned least = __reduce_min_sync(FULL, key);
    const int at = __ffs(__ballot_sync(FULL, key == least)) - 1;
    if (lane < m) A.tri[(size_t)pid * A.stride + (lane >= at ? lane - at : lane - at + m)] = id;
    if (lane == 0) A.nn[pid] = m;
}

// WRAP_HANDED: the points of A.star_list (those the thread-per-point stage could not finish);
// WRAP_OWN: A's own items; WRAP_REPAIR: its own if there are at most A.wrap_items (the
// thread-per-point stage then leaves them), else the list
template <typename T, bool IDX, bool GEN>
__global__ void __launch_bounds__(WRAP_WARPS * 32) k_wrap(RingArgs A)
{
    __shared__ WrapMem<T> mem[WRAP_WARPS];
    const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
    WrapMem<T> &M = mem[wib];
    Ctr ctr = { 0, 0, 0, 0, 0, 0, 0 };
    unsigned pts = 0, heavy = 0;
    int maxr = 0;
    const bool handed = A.wrap_mode == WRAP_HANDED || (A.wrap_mode == WRAP_REPAIR && item_count(A) > A.wrap_items);
    const int n = handed ? min(*A.star_count, A.n_items) : item_count(A);
    if (A.count_round && blockIdx.x == 0 && threadIdx.x == 0 && n > 0) {
        atomicAdd(&A.st->repaired, (unsigned long long)n);
        atomicMax(&A.st->rounds, A.round + 1);
    }
    if ((int)blockIdx.x * WRAP_WARPS >= n) return;
    for (int item = blockIdx.x * WRAP_WARPS + wib; item < n; item += gridDim.x * WRAP_WARPS) {
        int pid, slot = 0;
        if (handed || IDX) {
            pid = handed ? A.star_list[item] : A.worklist[item];
            if (!IDX) slot = A.slot_of[pid];
        } else {
            slot = A.item_base + item;
            pid = __ldg(&A.sidx[slot]);
        }
        const SetDesc &S = A.sets[A.set_of ? __ldg(&A.set_of[pid]) : 0];
        const double2 p = __ldg(IDX ? &A.pos[pid] : &A.spos[slot]);
        Wrap<T, IDX, GEN> b(A, S, M, lane, p, IDX ? pid : slot);
        int id = -1;
        const int r = b.run(id);
        // more than a thread may scan (counted; complemented in the deferred list)
        const bool over = r == W_HEAVY || b.cells + b.cand > (unsigned)A.work_budget;
        if (r == W_OK) {
            ++pts;
            heavy += over;
            if (!IDX && lane < b.m) id = __ldg(&A.sidx[id]);
            if (IDX) {
                warp_finish_repair(A, pid, id, b.m, lane);
                __syncwarp();
            }
            warp_store_ring(A, pid, id, b.m, lane, maxr);
        } else if (lane == 0) {
            A.defer_list[atomicAdd(A.defer_count, 1)] = over ? ~pid : pid;
        }
        if (lane == 0) {
            ctr.cand += b.cand;
            ctr.tests += b.tests * (unsigned)b.n;
            ctr.ins += b.m;
            ctr.cells += b.cells;
        }
        ctr.u32 += b.u32;
        ctr.u64 += b.u64;
        ctr.mism += b.mism;
        __syncwarp();
    }
    if (lane == 0 && heavy) atomicAdd(&A.st->heavy_points, (unsigned long long)heavy);
    flush_counters(A, ctr, lane == 0 ? pts : 0, maxr);
}

template <typename T, bool IDX, bool GEN>
cudaError_t launch_wrap_t(const RingArgs &a, int sms, cudaStream_t s)
{
    int blocks = (a.n_items + WRAP_WARPS - 1) / WRAP_WARPS;
    const int most = sms * 6;
    if (blocks > most) blocks = most;
    k_wrap<T, IDX, GEN><<<blocks, WRAP_WARPS * 32, 0, s>>>(a);
    return cudaGetLastError();
}

}  // namespace

cudaError_t launch_wrap(const RingArgs &a, int mode, int sms, cudaStream_t s)
{
    if (a.n_items <= 0) return cudaSuccess;
    const bool idx = a.cand_by_index != 0;
    if (a.general) {
        if (mode == MODE_F64) return idx ? launch_wrap_t<double, true, true>(a, sms, s) : launch_wrap_t<double, false, true>(a, sms, s);
        return idx ? launch_wrap_t<float, true, true>(a, sms, s) : launch_wrap_t<float, false, true>(a, sms, s);
    }
    if (mode == MODE_F64) return idx ? launch_wrap_t<double, true, false>(a, sms, s) : launch_wrap_t<double, false, false>(a, sms, s);
    return idx ? launch_wrap_t<float, true, false>(a, sms, s) : launch_wrap_t<float, false, false>(a, sms, s);
}

}  // namespace dgt
