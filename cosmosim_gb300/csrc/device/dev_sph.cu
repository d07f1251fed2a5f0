// dev_sph.cu — SPH density/pressure and forces on the shared octree
// (reference src/sph.c:45-196) and the neighbour query of
// src/octree.c:236-318.
//
// Neighbour order matters: the reference keeps the first 128 bodies within
// the radius in depth-first octant order (src/octree.c:260-277, sph.h:9), and
// the cap binds often. The sorted order of a tree built here is that order; in
// a caller's pool the preorder cells meet the leaves in it. Each pass runs in
// two kernels: the walk records every gas body's capped list, then a pair
// kernel sums over the lists in that order — the FP64 pair arithmetic then
// runs densely, one lane per gas body, instead of once per walk step for
// whichever lanes found a neighbour. Lanes are the gas bodies in key order.
// Its divisions and square roots (about ten FP64 operations each with the
// compiler's operators, on a GPU whose FP64 rate is 1/64 of FP32) run on the
// integer pipes (div_rn, sqrt_rn): correctly rounded, so bit-identical.
//
// Compiled with -fmad=false, with the reference's operation order, so for the
// same inputs every sum rounds as the reference's does.
#include "dev_fpint.cuh"
#include "dev_internal.cuh"

namespace {

constexpr int SPH_THREADS = 128;
constexpr double GAMMA = 5.0 / 3.0;
constexpr double PI_D = 3.14159265358979323846;

// The pair kernels are bound by the FP64 pipe, on which comparisons run too:
// these compare (and halve and double) by the bits, with the same results.
constexpr long long ONE_BITS = 0x3ff0000000000000ll, INF_BITS = 0x7ff0000000000000ll;

// q > 1 for q that is not negative (false for NaN, as the comparison).
__device__ __forceinline__ bool above_one(double q)
{
    const unsigned long long b = (unsigned long long)__double_as_longlong(q);
    return b - (unsigned long long)(ONE_BITS + 1) < (unsigned long long)(INF_BITS - ONE_BITS);
}
// q <= 0.5 for q that is not negative (false for NaN).
__device__ __forceinline__ bool at_most_half(double q)
{
    return (unsigned long long)__double_as_longlong(q) <= (unsigned long long)(ONE_BITS - (1ll << 52));
}
// v < 0 (false for -0 and NaN).
__device__ __forceinline__ bool negative(double v)
{
    const unsigned long long b = (unsigned long long)__double_as_longlong(v);
    return b - ((1ull << 63) + 1ull) < (unsigned long long)INF_BITS;
}
// r < 1e-15 for r that is not negative.
__device__ __forceinline__ bool tiny(double r)
{
    return (unsigned long long)__double_as_longlong(r) <
           (unsigned long long)__double_as_longlong(1e-15);
}
// 0.5 v and 2 v: an exponent step unless a result could be subnormal or infinite.
__device__ __forceinline__ double half_of(double v)
{
    const long long b = __double_as_longlong(v);
    if ((unsigned)((int)(b >> 52) & 0x7ff) - 2u < 2045u)
        return __longlong_as_double(b - (1ll << 52));
    return 0.5 * v;
}
__device__ __forceinline__ double twice(double v)
{
    const long long b = __double_as_longlong(v);
    if ((unsigned)((int)(b >> 52) & 0x7ff) - 1u < 2045u)
        return __longlong_as_double(b + (1ll << 52));
    return 2.0 * v;
}

// M4 cubic spline W(r, h), src/sph.c:11-25, with its normalisation 8/(pi h^3)
// computed by the caller once per gas body (the same expression, so the same
// value): one division fewer per pair.
__device__ __forceinline__ double kernel_W_norm(double r, double h, double norm)
{
    if (h < 1e-10)
        return 0.0;
    double q = div_rn(r, h);
    if (above_one(q))
        return 0.0;
    // norm (1 - a + a q), a = 6 q q, or 2 norm t t t, t = 1 - q: three of the
    // multiplications are shared
    const bool in = at_most_half(q);
    const double t = 1.0 - q, u = in ? q : t;
    const double a = (in ? 6.0 : twice(norm)) * u * u, w = a * u;
    return in ? norm * (1.0 - a + w) : w;
}

__device__ __forceinline__ double kernel_norm(double h) { return div_rn(8.0, PI_D * h * h * h); }

// the kernel's radial derivative dW/dr(r, h), src/sph.c:27-41; its two
// branches, -12 q + 18 q q and -6 t t (t = 1 - q), share their operations
// (adding -0 changes nothing)
__device__ __forceinline__ double kernel_dWdr(double r, double h)
{
    if (h < 1e-10)
        return 0.0;
    const Divisor by_h = divisor(h); // one reciprocal for both quotients
    double q = div_rn(r, by_h);
    if (above_one(q) || tiny(r))
        return 0.0;
    double norm = div_rn(8.0, PI_D * h * h * h);
    const bool in = at_most_half(q);
    const double t = 1.0 - q, u = in ? q : t;
    const double linear = in ? -12.0 * q : -0.0;
    return div_rn(norm * (linear + (in ? 18.0 : -6.0) * u * u), by_h);
}

struct SphArgs {
    const int *gas;
    const double *x, *y, *z, *vx, *vy, *vz, *m;
    const int *type;
    double *h, *rho, *P, *u;
    double *ax, *ay, *az;
    const double4_32a *geo;
    const NodeS32 *s32;
    const NodeW64 *w64;
    const NodeLink *link;
    const int *child;
    const DevRoot *root;
    const float4 *sp, *box, *sbox; // sorted records, their boxes by 32 and by 1024 (k_sph_sort)
    DevScalars *sc;
    int *nb;       // neighbour lists, slot-major
    int *nb_count; // neighbours per gas body
    int *relist;   // per gas body: the density pass changed h (search again)
    int reuse;     // force pass: keep the density lists of bodies with relist 0
    int density;   // density pass (the lists also store 8/(pi h^3) in pr2)
    double *pr2, *cs; // per-body force terms (k_sph_body_terms)
    double *sum;      // force sums of the gas bodies, 3 x stride
    int n, node_cap, stride;
};

// ---- neighbour lists: one warp per query ----------------------------------
//
// The warp scans the preorder cells 32 at a time. Lane k tests cell cur+k
// against the query sphere (the reference's box test, src/octree.c:250-256).
// A cell is reached only if no ancestor failed; inside the window an
// ancestor u of v satisfies u < v < next(u), so "v lies under a failed cell"
// is an exclusive prefix-max over lanes of next(u) of failed cells, compared
// with v. Reached leaves whose body lies within the radius are neighbours,
// taken in lane (= depth-first) order up to the cap. The cursor then moves
// past the window and past every failed cell's subtree.
//
// Tests run in FP32 with a bound on their rounding: a decision is taken in
// FP32 only when the FP32 value clears the threshold by more than that bound
// (position errors <= 8 ulp of the largest magnitude involved per axis, plus
// 2^-18 relative on the squared sums); otherwise the reference's own FP64
// expression decides. So every decision equals the reference's.

constexpr float FP32_EPS_POS = 0x1p-21f; // 8 x 2^-24 per axis
constexpr float FP32_EPS_SUM = 0x1p-18f;

// Box test of src/octree.c:250-256: true when the cell may hold neighbours.
__device__ __forceinline__ bool box_reaches(const NodeS32 &c, float qx, float qy, float qz,
                                            float mq, float r2f, const SphArgs &a, int cell,
                                            double px, double py, double pz, double r2)
{
    const float e = (mq + c.cmax) * FP32_EPS_POS;
    const float dx = fmaxf(0.0f, fabsf(qx - c.cx) - c.hs);
    const float dy = fmaxf(0.0f, fabsf(qy - c.cy) - c.hs);
    const float dz = fmaxf(0.0f, fabsf(qz - c.cz) - c.hs);
    const float lx = fmaxf(0.0f, dx - e), ly = fmaxf(0.0f, dy - e), lz = fmaxf(0.0f, dz - e);
    const float lo = lx * lx + ly * ly + lz * lz;
    if (lo > r2f * (1.0f + FP32_EPS_SUM))
        return false;
    const float hx = dx + e, hy = dy + e, hz = dz + e;
    const float hi = hx * hx + hy * hy + hz * hz;
    if (hi < r2f * (1.0f - FP32_EPS_SUM))
        return true;
    const double4_32a g = a.geo[cell]; // too close to call in FP32
    double gx = fmax(0.0, fabs(px - g.x) - g.w);
    double gy = fmax(0.0, fabs(py - g.y) - g.w);
    double gz = fmax(0.0, fabs(pz - g.z) - g.w);
    return !(gx * gx + gy * gy + gz * gz > r2);
}

// Leaf test of src/octree.c:262-272: body within the radius.
__device__ __forceinline__ bool leaf_within(const NodeS32 &c, float qx, float qy, float qz,
                                            float mq, float r2f, const SphArgs &a, double px,
                                            double py, double pz, double r2)
{
    const float mb = fmaxf(fabsf(c.bx), fmaxf(fabsf(c.by), fabsf(c.bz)));
    const float e = (mq + mb) * FP32_EPS_POS;
    const float dx = fabsf(c.bx - qx), dy = fabsf(c.by - qy), dz = fabsf(c.bz - qz);
    const float hx = dx + e, hy = dy + e, hz = dz + e;
    const float hi = hx * hx + hy * hy + hz * hz;
    if (hi < r2f * (1.0f - FP32_EPS_SUM))
        return true;
    const float lx = fmaxf(0.0f, dx - e), ly = fmaxf(0.0f, dy - e), lz = fmaxf(0.0f, dz - e);
    const float lo = lx * lx + ly * ly + lz * lz;
    if (lo > r2f * (1.0f + FP32_EPS_SUM))
        return false;
    const int j = c.body;
    double bx = a.x[j] - px;
    double by = a.y[j] - py;
    double bz = a.z[j] - pz;
    return bx * bx + by * by + bz * bz <= r2;
}

__device__ __forceinline__ int warp_excl_max(int v)
{
    const int lane = threadIdx.x & 31;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        int t = __shfl_up_sync(0xffffffffu, v, o);
        if (lane >= o)
            v = max(v, t);
    }
    int ex = __shfl_up_sync(0xffffffffu, v, 1);
    return lane == 0 ? INT_MIN : ex;
}

// Lists: gas body gas[k] gets its first CSG_SPH_MAX_NEIGHBORS neighbours within
// its current smoothing length, in depth-first order, slot-major
// (nb[slot * stride + k]) for coalesced reads in the pair kernels. The density
// pass uses h before its update (src/sph.c:53-63), the force pass after it
// (src/sph.c:112-126): each pass builds its list from the h it sees.
//
// On a tree built here the bodies' sorted order is the depth-first order of
// their leaves, so a list needs no tree: the sorted positions are kept as
// float4 records with the box of every 32 (a chunk) and of every 1024 (a
// super-chunk), made by k_sph_sort, and a warp tests super-chunk boxes, then
// the chunk boxes of those the query sphere meets, then the bodies of those
// chunks, 32 at a time and always in sorted order. Per query this reads about
// 25 chunks where the walk over preorder cells below read over a hundred
// windows of 48-byte records: 105 -> 34 us a pass for the 100k merger's 10,000
// gas bodies. A caller's pool (no sorted order) keeps that walk.
//
// A body whose FP32 distance is too close to the radius to call is decided by
// the reference's expressions: its own distance, and the box test of every cell
// on its path (which could reject it only within rounding).

// Sorted records, chunk boxes and the gas bodies' list (in sorted order up to
// the order in which warps count themselves in; nothing depends on it).
constexpr int SORT_THREADS = 1024; // one super-chunk per block

__global__ void __launch_bounds__(SORT_THREADS) k_sph_sort(
    DevScalars *sc, const int *__restrict__ perm, const double *__restrict__ x,
    const double *__restrict__ y, const double *__restrict__ z, const int *__restrict__ type,
    const signed char *__restrict__ lcp, float4 *__restrict__ sp, float4 *__restrict__ box,
    float4 *__restrict__ sbox, int *__restrict__ gas)
{
    __shared__ float4 s_lo[CSG_WARP], s_hi[CSG_WARP];
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    const int p = blockIdx.x * SORT_THREADS + threadIdx.x, na = sc->n_alive;
    if (blockIdx.x * SORT_THREADS >= na)
        return; // the whole block
    const float inf = __int_as_float(0x7f800000);
    float4 lo = make_float4(inf, inf, inf, 0.0f), hi = make_float4(-inf, -inf, -inf, 0.0f);
    bool is_gas = false;
    int b = -1;
    if (p < na) {
        b = perm[p];
        const float fx = (float)x[b], fy = (float)y[b], fz = (float)z[b];
        // bodies equal to depth 64 after the first share its leaf, which names
        // the first only
        const bool own = p == 0 || lcp[p - 1] < CSG_MAX_LEVEL;
        sp[p] = make_float4(fx, fy, fz, __int_as_float(own ? b : -1));
        lo = make_float4(fx, fy, fz, fmaxf(fabsf(fx), fmaxf(fabsf(fy), fabsf(fz))));
        hi = make_float4(fx, fy, fz, 0.0f);
        is_gas = type[b] == BODY_GAS;
    }
    const unsigned g = __ballot_sync(0xffffffffu, is_gas);
    int k = 0;
    if (lane == 0 && g)
        k = atomicAdd(&sc->n_gas, __popc(g));
    k = __shfl_sync(0xffffffffu, k, 0);
    if (is_gas)
        gas[k + __popc(g & ((1u << lane) - 1u))] = b;
    auto join = [](float4 &l, float4 &h) {
#pragma unroll
        for (int o = 16; o; o >>= 1) {
            l.x = fminf(l.x, __shfl_xor_sync(0xffffffffu, l.x, o));
            l.y = fminf(l.y, __shfl_xor_sync(0xffffffffu, l.y, o));
            l.z = fminf(l.z, __shfl_xor_sync(0xffffffffu, l.z, o));
            l.w = fmaxf(l.w, __shfl_xor_sync(0xffffffffu, l.w, o));
            h.x = fmaxf(h.x, __shfl_xor_sync(0xffffffffu, h.x, o));
            h.y = fmaxf(h.y, __shfl_xor_sync(0xffffffffu, h.y, o));
            h.z = fmaxf(h.z, __shfl_xor_sync(0xffffffffu, h.z, o));
        }
    };
    join(lo, hi);
    if (lane == 0) {
        const int c = blockIdx.x * CSG_WARP + wid;
        box[2 * c] = lo;
        box[2 * c + 1] = hi;
        s_lo[wid] = lo;
        s_hi[wid] = hi;
    }
    __syncthreads();
    if (wid == 0) {
        lo = s_lo[lane];
        hi = s_hi[lane];
        join(lo, hi);
        if (lane == 0) {
            sbox[2 * blockIdx.x] = lo;
            sbox[2 * blockIdx.x + 1] = hi;
        }
    }
}

struct Query {
    double px, py, pz, r2;
    float qx, qy, qz, mq, r2f;
};

// Whether a box of sorted bodies may hold one within the radius: never false
// for one that does.
__device__ __forceinline__ bool chunk_meets(const float4 *box, int c, const Query &q)
{
    const float4 lo = __ldg(&box[2 * c]), hi = __ldg(&box[2 * c + 1]);
    const float e = (q.mq + lo.w) * FP32_EPS_POS;
    const float dx = fmaxf(0.0f, fmaxf(lo.x - q.qx, q.qx - hi.x) - e);
    const float dy = fmaxf(0.0f, fmaxf(lo.y - q.qy, q.qy - hi.y) - e);
    const float dz = fmaxf(0.0f, fmaxf(lo.z - q.qz, q.qz - hi.z) - e);
    return dx * dx + dy * dy + dz * dz <= q.r2f * (1.0f + FP32_EPS_SUM);
}

// The reference's own tests of the body at sorted position p (src/octree.c:
// 250-272): every cell on its path, then its distance.
__device__ __noinline__ bool exact_within(const SphArgs &a, int p, int j, double px, double py,
                                          double pz, double r2)
{
    double bx = a.x[j] - px;
    double by = a.y[j] - py;
    double bz = a.z[j] - pz;
    const double d2 = bx * bx + by * by + bz * bz;
    if (!(d2 <= r2))
        return false;
    // a cell on the path lies no further than the body, but for the rounding of
    // its centre and of the differences (a few ulp of the root's extent)
    const DevRoot &root = *a.root;
    const double R = fabs(root.c0[0]) + fabs(root.c0[1]) + fabs(root.c0[2]) + root.hs0 + fabs(px) +
                     fabs(py) + fabs(pz);
    const double slack = 1e-14 * R;
    if (d2 + slack * (slack + 4.0 * sqrt(r2)) < r2 * (1.0 - 1e-14))
        return true;
    const int nn = a.sc->n_nodes;
    for (int cell = 0, level = 0; level <= CSG_MAX_LEVEL; level++) {
        const double4_32a g = a.geo[cell];
        double gx = fmax(0.0, fabs(px - g.x) - g.w);
        double gy = fmax(0.0, fabs(py - g.y) - g.w);
        double gz = fmax(0.0, fabs(pz - g.z) - g.w);
        if (gx * gx + gy * gy + gz * gz > r2)
            return false;
        int next = -1;
        for (int o = 0; o < 8; o++) { // the child whose bodies include position p
            const int c = a.child[8 * (size_t)cell + o];
            if (c > cell && c < nn && a.link[c].first <= p && p < a.link[c].first + a.link[c].count)
                next = c;
        }
        if (next < 0)
            return true; // the leaf
        cell = next;
    }
    return true;
}

__device__ __forceinline__ bool body_within(const SphArgs &a, const Query &q, const float4 &v, int p)
{
    const int j = __float_as_int(v.w);
    if (j < 0)
        return false;
    const float mb = fmaxf(fabsf(v.x), fmaxf(fabsf(v.y), fabsf(v.z)));
    const float e = (q.mq + mb) * FP32_EPS_POS;
    const float dx = fabsf(v.x - q.qx), dy = fabsf(v.y - q.qy), dz = fabsf(v.z - q.qz);
    const float hx = dx + e, hy = dy + e, hz = dz + e;
    if (hx * hx + hy * hy + hz * hz < q.r2f * (1.0f - FP32_EPS_SUM))
        return true;
    const float lx = fmaxf(0.0f, dx - e), ly = fmaxf(0.0f, dy - e), lz = fmaxf(0.0f, dz - e);
    if (lx * lx + ly * ly + lz * lz > q.r2f * (1.0f + FP32_EPS_SUM))
        return false;
    return exact_within(a, p, j, q.px, q.py, q.pz, q.r2);
}

__device__ __forceinline__ void list_sorted(const SphArgs &a, int k, int lane)
{
    const int na = (a.sc->n_nodes > a.node_cap) ? 0 : a.sc->n_alive;
    const int chunks = (na + CSG_WARP - 1) / CSG_WARP, supers = (chunks + CSG_WARP - 1) / CSG_WARP;
    const int i = a.gas[k];
    const double h = a.h[i];
    Query q;
    q.px = a.x[i];
    q.py = a.y[i];
    q.pz = a.z[i];
    q.r2 = h * h;
    q.qx = (float)q.px;
    q.qy = (float)q.py;
    q.qz = (float)q.pz;
    q.mq = fmaxf(fabsf(q.qx), fmaxf(fabsf(q.qy), fabsf(q.qz)));
    q.r2f = (float)q.r2;
    const unsigned lt = (1u << lane) - 1u;
    const size_t stride = (size_t)a.stride;
    int found = 0;
    for (int s0 = 0; s0 < supers && found < CSG_SPH_MAX_NEIGHBORS; s0 += CSG_WARP) {
        const int s = s0 + lane;
        unsigned ms = __ballot_sync(0xffffffffu, s < supers && chunk_meets(a.sbox, s, q));
        while (ms && found < CSG_SPH_MAX_NEIGHBORS) {
            const int c0 = (s0 + __ffs((int)ms) - 1) * CSG_WARP;
            ms &= ms - 1u;
            unsigned mc = __ballot_sync(0xffffffffu,
                                        c0 + lane < chunks && chunk_meets(a.box, c0 + lane, q));
            if (!mc)
                continue;
            const float4 none = make_float4(0.0f, 0.0f, 0.0f, __int_as_float(-1));
            int p = (c0 + __ffs((int)mc) - 1) * CSG_WARP + lane;
            mc &= mc - 1u;
            float4 v = p < na ? __ldg(&a.sp[p]) : none;
            for (;;) {
                // the next chunk's bodies are on their way during this one's tests
                const bool more = mc != 0u;
                int pn = 0;
                float4 vn = none;
                if (more) {
                    pn = (c0 + __ffs((int)mc) - 1) * CSG_WARP + lane;
                    mc &= mc - 1u;
                    vn = pn < na ? __ldg(&a.sp[pn]) : none;
                }
                const bool cand = body_within(a, q, v, p);
                const unsigned m = __ballot_sync(0xffffffffu, cand);
                if (cand) {
                    const int slot = found + __popc(m & lt);
                    if (slot < CSG_SPH_MAX_NEIGHBORS)
                        a.nb[stride * slot + k] = __float_as_int(v.w);
                }
                found = min(CSG_SPH_MAX_NEIGHBORS, found + __popc(m));
                if (!more || found == CSG_SPH_MAX_NEIGHBORS)
                    break;
                p = pn;
                v = vn;
            }
        }
    }
    if (lane == 0) {
        a.nb_count[k] = found;
        if (a.density) // its pairs need 8/(pi h^3) of this body
            a.pr2[i] = h < 1e-10 ? 0.0 : kernel_norm(h);
    }
}

// The same on a caller's pool.
__device__ __forceinline__ void list_one(const SphArgs &a, int k, int lane)
{
    const int nnodes = (a.sc->n_nodes > a.node_cap) ? 0 : a.sc->n_nodes;
    const int i = a.gas[k];
    const double px = a.x[i], py = a.y[i], pz = a.z[i];
    const double h = a.h[i];
    const double r2 = h * h;
    const float qx = (float)px, qy = (float)py, qz = (float)pz;
    const float mq = fmaxf(fabsf(qx), fmaxf(fabsf(qy), fabsf(qz)));
    const float r2f = (float)r2;
    const unsigned lt = (1u << lane) - 1u;
    const size_t stride = (size_t)a.stride;
    int found = 0;
    int cur = 0;
    while (cur < nnodes && found < CSG_SPH_MAX_NEIGHBORS) {
        const int v = cur + lane;
        const bool valid = v < nnodes;
        NodeS32 c;
        bool reach = false;
        int fail_next = 0;
        if (valid) {
            c = a.s32[v];
            reach = box_reaches(c, qx, qy, qz, mq, r2f, a, v, px, py, pz, r2);
            if (!reach)
                fail_next = c.next;
            if (c.next <= v)
                dev_fail(a.sc, CSG_ERR_WALK_LIMIT);
        }
        const int above = warp_excl_max(fail_next);
        bool cand = false;
        if (valid && reach && above <= v && c.body != -1) {
            if (c.body == -3)
                dev_fail(a.sc, CSG_ERR_BAD_POOL);
            else if (c.body >= 0)
                cand = leaf_within(c, qx, qy, qz, mq, r2f, a, px, py, pz, r2);
        }
        const unsigned m = __ballot_sync(0xffffffffu, cand);
        if (cand) {
            const int slot = found + __popc(m & lt);
            if (slot < CSG_SPH_MAX_NEIGHBORS)
                a.nb[stride * slot + k] = c.body;
        }
        found = min(CSG_SPH_MAX_NEIGHBORS, found + __popc(m));
        // skip past the window and past every failed subtree
        const int jump = __reduce_max_sync(0xffffffffu, (unsigned)max(fail_next, 0));
        cur = max(cur + CSG_WARP, jump); // strictly increases: the loop ends
    }
    if (lane == 0) {
        a.nb_count[k] = found;
        if (a.density) // its pairs need 8/(pi h^3) of this body
            a.pr2[i] = h < 1e-10 ? 0.0 : kernel_norm(h);
    }
}

template <bool SORTED>
__global__ void __launch_bounds__(SPH_THREADS) k_sph_lists(SphArgs a)
{
    const int lane = threadIdx.x & 31;
    const int n_gas = a.sc->n_gas;
    const int nwarps = (int)((gridDim.x * (long long)SPH_THREADS) >> 5);
    for (int k = (int)(((long long)blockIdx.x * SPH_THREADS + threadIdx.x) >> 5); k < n_gas;
         k += nwarps) // warp-uniform
        if (!a.reuse || a.relist[k]) {
            if (SORTED)
                list_sorted(a, k, lane);
            else
                list_one(a, k, lane);
        }
}

// Pair kernels. A block takes a group of up to 32 gas bodies; its pair threads
// compute the group's (list slot, body) terms into shared memory, PAIR_TERMS at
// a time, and its sum warps, one lane per body and one warp per component, add
// the terms of the slots before in list order: the reference's order, with the
// same operations, so the sums are the reference's bit for bit (a skipped pair
// stores 0, and x - 0 == x for every x). Two buffers, one barrier per step: the
// long dependent chains of the sums run beside the pairs. The FP64 pipe bounds
// both kernels, and an instruction holds it for a whole warp however few lanes
// are active: hence a lane per body in the sums, and groups of one size, so
// that every block gets as many bodies. For the 100k merger's 10,000 gas bodies
// density takes 69 us and forces 174 us (the pipe busy for 3/4 of both); with
// the terms in global memory, a second kernel for the sums and every quotient
// with its own reciprocal 93 and 232 us, the substep 802 us instead of 865.
// Blocks of 128, 192 or 384 pair threads (6, 4, 2 per SM): within 1%.
constexpr int PAIR_THREADS = 256;
constexpr int PAIR_BLOCKS = 3; // per SM
constexpr int PAIR_TERMS = 3 * PAIR_THREADS;
constexpr int PAIR_GROUP = CSG_WARP;
constexpr int PAIR_SLOTS = 64; // most list slots per step
constexpr int DENSITY_THREADS = PAIR_THREADS + CSG_WARP;
constexpr int FORCE_THREADS = PAIR_THREADS + 3 * CSG_WARP;
constexpr int SUM_THREADS = 64;

// One step: slots first .. first + slots of the group's bodies k0 .. k0 + count.
struct PairStep {
    int buf, k0, count, first, slots;
    bool last;
};

// The groups of a block: fn pairs(step) on the pair threads, then fn sums(step)
// on the sum threads, a step behind.
template <class Pairs, class Sums>
__device__ __forceinline__ void for_groups(int n_gas, const int *__restrict__ nb_count, Pairs pairs,
                                           Sums sums)
{
    const int grid = (int)gridDim.x, lane = threadIdx.x & 31;
    const int rounds = (n_gas + PAIR_GROUP * grid - 1) / (PAIR_GROUP * grid);
    const int B = rounds > 0 ? (n_gas + rounds * grid - 1) / (rounds * grid) : 1;
    const int most_slots = min(PAIR_SLOTS, PAIR_TERMS / B);
    PairStep before;
    before.count = 0;
    int buf = 0;
    for (int round = 0; round <= rounds; round++) { // the last one: sums alone
        PairStep now;
        now.k0 = (round * grid + (int)blockIdx.x) * B;
        now.count = round < rounds ? max(0, min(B, n_gas - now.k0)) : 0;
        const int most =
            __reduce_max_sync(0xffffffffu, lane < now.count ? nb_count[now.k0 + lane] : 0);
        now.first = 0;
        do {
            now.buf = buf;
            now.slots = min(most_slots, most - now.first);
            now.last = now.first + most_slots >= most;
            if (threadIdx.x < PAIR_THREADS) {
                if (now.count > 0)
                    pairs(now);
            } else if (before.count > 0) {
                sums(before);
            }
            __syncthreads();
            before = now;
            buf ^= 1;
            now.first += most_slots;
        } while (!before.last);
    }
}

// fn pair(p, slot, body of the group) for the pairs of a step
template <class Pair>
__device__ __forceinline__ void for_pairs(const PairStep &st, const int *nn, Pair pair)
{
    const int B = st.count, ds = PAIR_THREADS / B, db = PAIR_THREADS - ds * B;
    int s = threadIdx.x / B, b = threadIdx.x - s * B;
    for (int p = threadIdx.x; s < st.slots; p += PAIR_THREADS) {
        if (st.first + s < nn[b])
            pair(p, st.first + s, b);
        s += ds;
        b += db;
        if (b >= B) {
            b -= B;
            s++;
        }
    }
}

__device__ __forceinline__ void pair_threads_sync()
{
    asm volatile("bar.sync 1, %0;" ::"n"(PAIR_THREADS) : "memory");
}

// P/(rho^2 + 1e-15) and the sound speed sqrt(gamma P/(rho + 1e-15)) of one gas
// body (src/sph.c:112, :153-154, :170-171): the force pairs need them for both
// bodies, computed once each they are the reference's per-pair values.
__device__ __forceinline__ void body_terms(const SphArgs &a, int j, double rho, double P)
{
    a.pr2[j] = div_rn(P, rho * rho + 1e-15);
    a.cs[j] = sqrt_rn(div_rn(GAMMA * P, rho + 1e-15));
}

// Density, adaptive h and pressure, src/sph.c:45-97 (terms m_j W(r, h_i)), and
// the body's force terms.
__global__ void __launch_bounds__(DENSITY_THREADS, PAIR_BLOCKS) k_sph_density(SphArgs a)
{
    __shared__ double term[2][PAIR_TERMS];
    __shared__ double sx[PAIR_GROUP], sy[PAIR_GROUP], sz[PAIR_GROUP], sh[PAIR_GROUP],
        snorm[PAIR_GROUP];
    __shared__ int snn[PAIR_GROUP];
    const int n_gas = a.sc->n_gas;
    const size_t stride = (size_t)a.stride;
    double rho = 0.0;
    for_groups(
        n_gas, a.nb_count,
        [&](const PairStep &st) {
            if (st.first == 0) {
                const int t = threadIdx.x;
                if (t < st.count) {
                    const int i = a.gas[st.k0 + t];
                    sx[t] = a.x[i];
                    sy[t] = a.y[i];
                    sz[t] = a.z[i];
                    sh[t] = a.h[i];
                    snorm[t] = a.pr2[i];
                    snn[t] = a.nb_count[st.k0 + t];
                }
                pair_threads_sync();
            }
            for_pairs(st, snn, [&](int p, int slot, int b) {
                const int j = a.nb[stride * slot + st.k0 + b];
                double dx = sx[b] - a.x[j];
                double dy = sy[b] - a.y[j];
                double dz = sz[b] - a.z[j];
                double r = sqrt_rn(dx * dx + dy * dy + dz * dz);
                term[st.buf][p] = a.m[j] * kernel_W_norm(r, sh[b], snorm[b]);
            });
        },
        [&](const PairStep &st) {
            const int b = threadIdx.x - PAIR_THREADS, k = st.k0 + b;
            if (b >= st.count)
                return;
            if (st.first == 0)
                rho = 0.0;
            const int nn = a.nb_count[k], end = min(nn - st.first, st.slots);
            for (int s = 0; s < end; s++)
                rho += term[st.buf][s * st.count + b];
            if (!st.last)
                return;
            const int i = a.gas[k];
            const double hi = a.h[i];
            int relist = 1;
            if (nn < 20 && hi < 50.0)
                a.h[i] = hi * 1.2;
            else if (nn > 48 && hi > 0.1)
                a.h[i] = hi * 0.8;
            else
                relist = 0;
            a.relist[k] = relist;
            if (rho < 1e-15 || isnan(rho))
                rho = 1e-15;
            a.rho[i] = rho;
            double u = a.u[i];
            if (u < 1e-15)
                u = 1e-15;
            const double P = (GAMMA - 1.0) * rho * u;
            a.P[i] = P;
            body_terms(a, i, rho, P);
        });
}

// The body terms alone, for a force pass that no density pass preceded.
__global__ void __launch_bounds__(SUM_THREADS) k_sph_body_terms(SphArgs a)
{
    const int k = blockIdx.x * SUM_THREADS + threadIdx.x;
    if (k >= a.sc->n_gas)
        return;
    const int j = a.gas[k];
    body_terms(a, j, a.rho[j], a.P[j]);
}

// Pressure gradient + Monaghan viscosity, src/sph.c:126-196: the bodies' sums
// (k_sph_force_add adds them to the accelerations).
__global__ void __launch_bounds__(FORCE_THREADS, PAIR_BLOCKS) k_sph_force(SphArgs a)
{
    __shared__ double term[2][3][PAIR_TERMS];
    __shared__ double sx[PAIR_GROUP], sy[PAIR_GROUP], sz[PAIR_GROUP], svx[PAIR_GROUP],
        svy[PAIR_GROUP], svz[PAIR_GROUP], sh[PAIR_GROUP], srho[PAIR_GROUP], spr2[PAIR_GROUP],
        scs[PAIR_GROUP];
    __shared__ int snn[PAIR_GROUP], si[PAIR_GROUP];
    const int n_gas = a.sc->n_gas;
    const size_t stride = (size_t)a.stride;
    double sum = 0.0;
    for_groups(
        n_gas, a.nb_count,
        [&](const PairStep &st) {
            if (st.first == 0) {
                const int t = threadIdx.x;
                if (t < st.count) {
                    const int i = a.gas[st.k0 + t];
                    si[t] = i;
                    sx[t] = a.x[i];
                    sy[t] = a.y[i];
                    sz[t] = a.z[i];
                    svx[t] = a.vx[i];
                    svy[t] = a.vy[i];
                    svz[t] = a.vz[i];
                    sh[t] = a.h[i];
                    srho[t] = a.rho[i];
                    spr2[t] = a.pr2[i];
                    scs[t] = a.cs[i];
                    snn[t] = a.nb_count[st.k0 + t];
                }
                pair_threads_sync();
            }
            for_pairs(st, snn, [&](int p, int slot, int b) {
                const int j = a.nb[stride * slot + st.k0 + b];
                double tx = 0.0, ty = 0.0, tz = 0.0;
                if (j != si[b] && a.type[j] == BODY_GAS) {
                    double dx = sx[b] - a.x[j];
                    double dy = sy[b] - a.y[j];
                    double dz = sz[b] - a.z[j];
                    double r = sqrt_rn(dx * dx + dy * dy + dz * dz);
                    if (!tiny(r)) {
                        double h_avg = half_of(sh[b] + a.h[j]);
                        double rho_j = a.rho[j];
                        double dvx = svx[b] - a.vx[j];
                        double dvy = svy[b] - a.vy[j];
                        double dvz = svz[b] - a.vz[j];
                        double vr = dvx * dx + dvy * dy + dvz * dz;
                        double visc = 0.0;
                        if (negative(vr)) {
                            double mu = div_rn(h_avg * vr, r * r + 0.01 * h_avg * h_avg);
                            double c_avg = half_of(scs[b] + a.cs[j]);
                            double rho_avg = half_of(srho[b] + rho_j);
                            visc = div_rn(-c_avg * mu + twice(mu) * mu, rho_avg + 1e-15);
                        }
                        double g = kernel_dWdr(r, h_avg);
                        const Divisor by_r = divisor(r); // one reciprocal for the three
                        double gx = div_rn(g * dx, by_r);
                        double gy = div_rn(g * dy, by_r);
                        double gz = div_rn(g * dz, by_r);
                        double f = a.m[j] * (spr2[b] + a.pr2[j] + visc);
                        tx = f * gx;
                        ty = f * gy;
                        tz = f * gz;
                    }
                }
                term[st.buf][0][p] = tx;
                term[st.buf][1][p] = ty;
                term[st.buf][2][p] = tz;
            });
        },
        [&](const PairStep &st) {
            const int t = threadIdx.x - PAIR_THREADS, b = t & 31, c = t >> 5, k = st.k0 + b;
            if (b >= st.count)
                return;
            if (st.first == 0)
                sum = 0.0;
            const int end = min(a.nb_count[k] - st.first, st.slots);
            for (int s = 0; s < end; s++)
                sum -= term[st.buf][c][s * st.count + b];
            if (st.last)
                a.sum[stride * c + k] = isnan(sum) ? 0.0 : sum;
        });
}

__global__ void __launch_bounds__(SUM_THREADS) k_sph_force_add(SphArgs a)
{
    const int k = blockIdx.x * SUM_THREADS + threadIdx.x;
    if (k >= a.sc->n_gas)
        return;
    const int i = a.gas[k];
    const size_t stride = (size_t)a.stride;
    a.ax[i] += a.sum[k] * 0.1;
    a.ay[i] += a.sum[stride + k] * 0.1;
    a.az[i] += a.sum[2 * stride + k] * 0.1;
}

// One query, one thread: src/octree.c:293-318.
__global__ void k_find_one(SphArgs a, double cx, double cy, double cz, double radius, int cap,
                           int *__restrict__ buf, int *__restrict__ count)
{
    const int nn = (a.sc->n_nodes > a.node_cap) ? 0 : a.sc->n_nodes;
    const double r2 = radius * radius;
    int c = 0, cur = 0;
    while (cur < nn && c < cap) {
        const double4_32a g = a.geo[cur];
        const int next = a.w64[cur].next, body = a.w64[cur].body;
        if (next <= cur) {
            dev_fail(a.sc, CSG_ERR_WALK_LIMIT);
            break;
        }
        double gx = fmax(0.0, fabs(cx - g.x) - g.w);
        double gy = fmax(0.0, fabs(cy - g.y) - g.w);
        double gz = fmax(0.0, fabs(cz - g.z) - g.w);
        if (gx * gx + gy * gy + gz * gz > r2) {
            cur = next;
            continue;
        }
        if (body >= 0) {
            if (body >= a.n) {
                dev_fail(a.sc, CSG_ERR_BAD_POOL);
            } else if (!(a.m[body] <= 0.0)) {
                double bx = a.x[body] - cx;
                double by = a.y[body] - cy;
                double bz = a.z[body] - cz;
                if (bx * bx + by * by + bz * bz <= r2)
                    buf[c++] = body;
            }
        }
        cur = cur + 1;
    }
    *count = c;
}

// Sorted records are held for whole super-chunks.
size_t sorted_cap(const csgd_t *d)
{
    return ((size_t)(d->cap > 0 ? d->cap : 1) + SORT_THREADS - 1) / SORT_THREADS * SORT_THREADS;
}

SphArgs make_args(csgd_t *d)
{
    SphArgs a;
    a.gas = d->gas;
    a.x = d->x;
    a.y = d->y;
    a.z = d->z;
    a.vx = d->vx;
    a.vy = d->vy;
    a.vz = d->vz;
    a.m = d->m;
    a.type = d->type;
    a.h = d->h;
    a.rho = d->rho;
    a.P = d->P;
    a.u = d->u;
    a.ax = d->ax;
    a.ay = d->ay;
    a.az = d->az;
    a.geo = d->geo;
    a.s32 = d->s32;
    a.w64 = d->w64;
    a.link = d->link;
    a.child = d->child;
    a.root = d->roots;
    a.sp = d->sph_sorted;
    a.box = a.sp + sorted_cap(d);
    a.sbox = a.box + 2 * (sorted_cap(d) / CSG_WARP);
    a.sc = d->sc;
    a.nb = d->nb;
    a.nb_count = d->nb_count;
    a.relist = d->sph_relist;
    a.reuse = 0;
    a.density = 0;
    a.pr2 = d->pr2;
    a.cs = d->cs;
    a.sum = d->sph_sum;
    a.n = d->n;
    a.node_cap = d->node_cap;
    a.stride = d->cap;
    return a;
}

// Caller-index order, for trees imported from a caller pool (no key order).
__global__ void k_gas_flags_idx(int n, const double *__restrict__ m, const int *__restrict__ type,
                                int *__restrict__ flag)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n)
        return;
    flag[i] = (type[i] == BODY_GAS && !(m[i] <= 0.0)) ? 1 : 0;
}

__global__ void k_gas_scatter_idx(DevScalars *sc, int n, const int *__restrict__ flag,
                                  const int *__restrict__ base, int *__restrict__ gas)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i == 0)
        sc->n_gas = base[n];
    if (i < n && flag[i])
        gas[base[i]] = i;
}

int gas_list(csgd_t *d)
{
    if (d->gas_valid)
        return CSG_OK;
    const int n = d->n;
    const int g = csgd_grid(n, 256);
    if (!d->imported) {
        float4 *sp = d->sph_sorted;
        float4 *box = sp + sorted_cap(d), *sbox = box + 2 * (sorted_cap(d) / CSG_WARP);
        if (!d->gas_zero) // the build's first kernel cleared it, unless it was counted since
            cudaMemsetAsync(&d->sc->n_gas, 0, sizeof(int), d->stream);
        d->gas_zero = 0;
        { k_sph_sort<<<csgd_grid(n, SORT_THREADS), SORT_THREADS, 0, d->stream>>>(d->sc, d->perm, d->x, d->y, d->z, d->type, d->lcp, sp, box, sbox, d->gas); d->launches++; }
    } else {
        { k_gas_flags_idx<<<g, 256, 0, d->stream>>>(n, d->m, d->type, d->cnt); d->launches++; }
        int rc = csg_scan_exclusive(d, d->cnt, d->base, n, nullptr);
        if (rc)
            return rc;
        { k_gas_scatter_idx<<<g, 256, 0, d->stream>>>(d->sc, n, d->cnt, d->base, d->gas); d->launches++; }
    }
    d->gas_valid = 1;
    return csgd_check(d, cudaGetLastError());
}

} // namespace

// Lists live in device memory sized for every body being gas (128 ints each),
// allocated on first SPH use.
static int ensure_lists(csgd_t *d)
{
    int rc = csgd_ensure_tree_extras(d, 1, 0); // SPH walks the cell geometry
    if (rc)
        return rc;
    if (d->nb && d->nb_cap >= d->cap)
        return CSG_OK;
    if (d->nb)
        cudaFree(d->nb);
    if (d->nb_count)
        cudaFree(d->nb_count);
    if (d->pr2)
        cudaFree(d->pr2);
    if (d->cs)
        cudaFree(d->cs);
    if (d->sph_sum)
        cudaFree(d->sph_sum);
    if (d->sph_relist)
        cudaFree(d->sph_relist);
    if (d->sph_sorted)
        cudaFree(d->sph_sorted);
    d->sph_sorted = nullptr;
    d->nb = nullptr;
    d->nb_count = d->sph_relist = nullptr;
    d->pr2 = d->cs = d->sph_sum = nullptr;
    size_t c = (size_t)(d->cap > 0 ? d->cap : 1);
    if (csgd_malloc((void **)&d->nb, sizeof(int) * CSG_SPH_MAX_NEIGHBORS * c) != cudaSuccess ||
        csgd_malloc((void **)&d->nb_count, sizeof(int) * c) != cudaSuccess ||
        csgd_malloc((void **)&d->sph_relist, sizeof(int) * c) != cudaSuccess ||
        // records, 2 words a chunk, 2 a super-chunk
        csgd_malloc((void **)&d->sph_sorted,
                    sizeof(float4) * (sorted_cap(d) + sorted_cap(d) / 16 + sorted_cap(d) / 512)) !=
            cudaSuccess ||
        csgd_malloc((void **)&d->pr2, sizeof(double) * c) != cudaSuccess ||
        csgd_malloc((void **)&d->cs, sizeof(double) * c) != cudaSuccess ||
        csgd_malloc((void **)&d->sph_sum, sizeof(double) * 3 * c) != cudaSuccess) {
        cudaGetLastError();
        csgd_set_err(d, CSG_ERR_NOMEM);
        return CSG_ERR_NOMEM;
    }
    d->nb_cap = d->cap;
    return CSG_OK;
}

static int sph_pass(csgd_t *d, int forces, bool sums = true, bool reuse = false)
{
    if (d->n_gal > 1) { // one system only (see csgd_set_systems)
        return CSG_ERR_UNSUPPORTED;
    }
    if (d->n <= 0)
        return CSG_OK;
    if (!d->geometry_valid) {
        return CSG_ERR_BAD_ARG;
    }
    int rc = ensure_lists(d);
    if (!rc)
        rc = gas_list(d);
    if (rc)
        return rc;
    SphArgs a = make_args(d);
    a.reuse = (forces && reuse) ? 1 : 0;
    a.density = forces ? 0 : 1;
    const int g = csgd_grid(d->n, SUM_THREADS);
    // one warp per gas body for the lists, warps striding over the gas bodies
    int gl = csgd_grid((long long)d->n * CSG_WARP, SPH_THREADS);
    if (gl > d->num_sms * 16)
        gl = d->num_sms * 16;
    if (d->imported)
        k_sph_lists<false><<<gl, SPH_THREADS, 0, d->stream>>>(a);
    else
        k_sph_lists<true><<<gl, SPH_THREADS, 0, d->stream>>>(a);
    d->launches++;
    // the gas count is known on the device only: the groups stride over the grid
    const int gp = d->num_sms * PAIR_BLOCKS;
    if (forces) {
        if (!a.reuse)
            { k_sph_body_terms<<<g, SUM_THREADS, 0, d->stream>>>(a); d->launches++; }
        { k_sph_force<<<gp, FORCE_THREADS, 0, d->stream>>>(a); d->launches++; }
        if (sums)
            { k_sph_force_add<<<g, SUM_THREADS, 0, d->stream>>>(a); d->launches++; }
    } else {
        { k_sph_density<<<gp, DENSITY_THREADS, 0, d->stream>>>(a); d->launches++; }
    }
    return csgd_check(d, cudaGetLastError());
}

extern "C" int csgd_sph_density(csgd_t *d) { return sph_pass(d, 0); }

extern "C" int csgd_prepare_sph(csgd_t *d) { return ensure_lists(d); }

extern "C" int csgd_sph_forces(csgd_t *d, int reuse_lists)
{
    return sph_pass(d, 1, true, reuse_lists != 0);
}

extern "C" int csgd_sph_force_terms(csgd_t *d, int reuse_lists)
{
    return sph_pass(d, 1, false, reuse_lists != 0);
}

extern "C" int csgd_sph_force_sums(csgd_t *d)
{
    if (d->n <= 0)
        return CSG_OK;
    SphArgs a = make_args(d);
    { k_sph_force_add<<<csgd_grid(d->n, SUM_THREADS), SUM_THREADS, 0, d->stream>>>(a); d->launches++; }
    return csgd_check(d, cudaGetLastError());
}

extern "C" int csgd_find_neighbors(csgd_t *d, double cx, double cy, double cz, double radius,
                                   int *buf, int cap, int *count_out)
{
    if (d->n_gal > 1) { // one system only (see csgd_set_systems)
        return CSG_ERR_UNSUPPORTED;
    }
    *count_out = 0;
    if (cap <= 0)
        return CSG_OK;
    if (!d->geometry_valid) {
        return CSG_ERR_BAD_ARG;
    }
    // scratch: the export rank buffer holds the result (node_cap >= cap is not
    // guaranteed, so cap is clamped to the buffer)
    if (cap > d->node_cap)
        cap = d->node_cap;
    int *dbuf = d->rank;
    int *dcount = d->ord_id;
    SphArgs a = make_args(d);
    { k_find_one<<<1, 1, 0, d->stream>>>(a, cx, cy, cz, radius, cap, dbuf, dcount); d->launches++; }
    int c = 0;
    cudaMemcpyAsync(&c, dcount, sizeof(int), cudaMemcpyDeviceToHost, d->stream);
    int rc = csgd_sync(d);
    if (rc)
        return rc;
    if (c > 0) {
        cudaMemcpyAsync(buf, dbuf, sizeof(int) * (size_t)c, cudaMemcpyDeviceToHost, d->stream);
        rc = csgd_sync(d);
    }
    *count_out = c;
    return rc;
}
