// dev_walk.cu — Barnes-Hut gravity walks (reference src/octree.c:171-234).
//
// Both walks give every body exactly the reference's interaction set: the
// cells it accepts by the monopole test (s*s)/d^2 < theta^2 with d^2 > 0, or
// reaches as leaves other than itself, in depth-first octant order.
//
// Traversal: one warp walks the tree for 32 bodies that are neighbours in key
// order, up to 32 cells a round (see "traversal in rounds" below).
//
// FP64 walk: the drop-in precision (k_walk64ws). Openings decided as in the
//   FP32 walk (equal to the reference's FP64 rounding); interactions queued
//   and evaluated densely in FP64 by a second warp per task, with 1/r^3 from
//   an FP32 rsqrt seed by integer arithmetic (one rounding), summed per child
//   subtree of the root as the FP32 walk does; small systems split the same
//   way (k_walk64ws_units), with the same bits. k_walk64_exact instead
//   uses the reference's own operation sequence per step (1/(r2*sqrt(r2)),
//   no fused multiply-add) — bit-identical results on the reference's own
//   tree; used by parity tests. It alone walks cell by cell: one cursor over
//   the preorder ids, each lane sleeping below an index `skip` (it accepted an
//   ancestor), the next 32 cells staged per warp in shared memory.
// FP32-mixed walk: positions and centres as float hi/lo pairs (differences
//   keep ~48 bits), rsqrt/products in FP32, Kahan-compensated FP32 sums per
//   body (small systems: per child subtree of the root, added in FP64).
//   Openings within the FP32 error band of the threshold are decided in FP64,
//   so the interaction set equals the FP64 walk's. Small systems with few
//   tasks for the GPU are walked by eight warps per task, one per root child
//   (k_walk32_units), with the same bits as one warp per task (k_walk32).
#include "dev_internal.cuh"

namespace {

struct WalkArgs {
    const int *perm;
    const double *x, *y, *z;
    const NodeW64 *w64;
    const NodeW32 *w32;
    const int *child; // 8 ids per cell
    const WalkTask *tasks;
    const DevRoot *roots;
    DevScalars *sc;
    double *ax, *ay, *az;
    double G, eps2, theta2, t2lo, t2hi;
    float Gf, eps2f;
    // FP32 opening test: accept when s^2 acc_k < d^2, open when s^2 opn_k > d^2
    // (acc_k, opn_k = (1 +- g) / theta^2); in between, |theta^2 d^2 - s^2| is
    // inside the FP32 error band g s^2 and the FP64 test decides
    float acc_k, opn_k;
    int node_cap;
    int group; // 0: one warp per task; g > 0: take g tasks at a time from a counter
    int wait_polls; // producer/consumer waits give up after this many polls
    double *part;   // split walks: segment partials, part[(3 * k + d) * pstride + body]
    long long pstride;
    // systems of at most split_max bodies (sys_n[gal] each in an ensemble,
    // n_bodies for one system) sum by the root's children; the FP64 whole-task
    // walk leaves them out when skip_small is set
    const int *sys_n;
    int n_bodies, split_max, skip_small;
};

// Work distribution shared by the walks. A task is up to 32 consecutive
// sorted bodies of one system. With group == 0 warp w of the grid walks task
// w; otherwise (persistent launch, a few blocks per SM) each warp takes the
// next `group` tasks from sc->task_next until none are left. Every take
// advances the counter, so the loop ends after at most n_tasks/group + 1
// takes per warp.
__device__ __forceinline__ int take_tasks(const WalkArgs &a)
{
    int v = 0;
    if ((threadIdx.x & 31) == 0)
        v = atomicAdd(&a.sc->task_next, a.group);
    return __shfl_sync(0xffffffffu, v, 0);
}

// Walk statistics: interactions, warp steps and lane-steps of lanes that
// had not finished (lane utilisation = active / (32 steps)).
struct WalkStats {
    unsigned long long hits = 0, steps = 0, active = 0;
};

// Validated task: bodies [pos0, pos0+count) and the system's cells [root, end).
struct TaskRange {
    int pos0, count, root, end;
    bool small; // its system has at most split_max bodies
};

__device__ __forceinline__ bool small_system(const WalkArgs &a, int gal)
{
    return (a.sys_n ? a.sys_n[gal] : a.n_bodies) <= a.split_max;
}

template <int WARPS, bool PERSIST, typename Fn>
__device__ __forceinline__ void for_each_task(const WalkArgs &a, Fn fn)
{
    const int nn = a.sc->n_nodes;
    if (nn > a.node_cap || nn < 1)
        return; // no valid tree (capacity error already recorded)
    const int nt = a.sc->n_tasks;
    auto run = [&](int t) {
        const WalkTask w = a.tasks[t];
        const DevRoot &r = a.roots[w.gal];
        const TaskRange tr{w.pos0, w.count, r.root, r.end, small_system(a, w.gal)};
        if (tr.root < 0 || tr.end > nn || tr.root >= tr.end)
            dev_fail(a.sc, CSG_ERR_WALK_LIMIT);
        else
            fn(tr);
    };
    if (!PERSIST) {
        const int t = blockIdx.x * WARPS + (threadIdx.x >> 5);
        if (t < nt)
            run(t);
        return;
    }
    int t = take_tasks(a), tend = t + a.group;
    while (t < nt) {
        run(t);
        if (++t >= tend) {
            t = take_tasks(a);
            tend = t + a.group;
        }
    }
}

// Reference opening decision fl(s2/d2) < theta2 (src/octree.c:202-203),
// without a division unless s2 is within 2^-50 of theta2*d2.
__device__ __forceinline__ bool accept64(double s2, double d2, const WalkArgs &a)
{
    if (!(d2 > 0.0))
        return false;
    if (s2 < a.t2lo * d2)
        return true;
    if (s2 > a.t2hi * d2)
        return false;
    return __ddiv_rn(s2, d2) < a.theta2;
}

// The reference's own FP64 operation sequence per step, one warp per task,
// no fused multiply-add: bit-identical accelerations on the reference's tree.
template <bool STATS>
__device__ __forceinline__ void walk64_exact_task(const WalkArgs &a, NodeW64 *win,
                                                  const TaskRange &tr, WalkStats &st)
{
    const int lane = threadIdx.x & 31;
    const int nn = tr.end;
    const bool valid = lane < tr.count;
    const int me = valid ? a.perm[tr.pos0 + lane] : -1;
    const double px = valid ? a.x[me] : 0.0, py = valid ? a.y[me] : 0.0,
                 pz = valid ? a.z[me] : 0.0;
    double sx = 0.0, sy = 0.0, sz = 0.0;
    int skip = valid ? 0 : INT_MAX;
    int cur = tr.root, wbase = INT_MIN / 2;
    while (cur < nn) {
        if (cur - wbase >= CSG_WARP) {
            wbase = cur;
            __syncwarp();
            if (wbase + lane < nn)
                win[lane] = a.w64[wbase + lane];
            __syncwarp();
        }
        const NodeW64 c = win[cur - wbase];
        bool open = false;
        if (STATS) {
            st.steps++;
            st.active += (cur >= skip);
        }
        if (cur >= skip) {
            if (c.m == 0.0) { // empty cell: reference returns at once (src/octree.c:181-182)
                skip = c.next;
            } else {
                const double dx = __dsub_rn(c.cx, px);
                const double dy = __dsub_rn(c.cy, py);
                const double dz = __dsub_rn(c.cz, pz);
                const double d2 = __dadd_rn(__dadd_rn(__dmul_rn(dx, dx), __dmul_rn(dy, dy)),
                                            __dmul_rn(dz, dz));
                bool take;
                if (c.body >= 0) {
                    take = (c.body != me);
                } else {
                    take = d2 > 0.0 && __ddiv_rn(c.s2, d2) < a.theta2;
                    if (take)
                        skip = c.next;
                    else
                        open = true;
                }
                if (take) {
                    const double r2 = __dadd_rn(d2, a.eps2);
                    const double inv = __ddiv_rn(1.0, __dmul_rn(r2, __dsqrt_rn(r2)));
                    const double gm = __dmul_rn(a.G, c.m);
                    sx = __dadd_rn(sx, __dmul_rn(__dmul_rn(gm, dx), inv));
                    sy = __dadd_rn(sy, __dmul_rn(__dmul_rn(gm, dy), inv));
                    sz = __dadd_rn(sz, __dmul_rn(__dmul_rn(gm, dz), inv));
                    if (STATS)
                        st.hits++;
                }
            }
        }
        const int nxt = __any_sync(0xffffffffu, open) ? cur + 1 : c.next;
        if (nxt <= cur) { // a malformed tree must not loop
            dev_fail(a.sc, CSG_ERR_WALK_LIMIT);
            break;
        }
        cur = nxt;
    }
    if (valid) {
        a.ax[me] = sx;
        a.ay[me] = sy;
        a.az[me] = sz;
    }
}

__device__ __forceinline__ void add_hits(const WalkArgs &a, const WalkStats &w)
{
    unsigned int h = __reduce_add_sync(0xffffffffu, (unsigned int)w.hits);
    unsigned int ac = __reduce_add_sync(0xffffffffu, (unsigned int)w.active);
    if ((threadIdx.x & 31) == 0) {
        if (h)
            atomicAdd(&a.sc->interactions, (unsigned long long)h);
        atomicAdd(&a.sc->walk_steps, w.steps);
        atomicAdd(&a.sc->walk_active, (unsigned long long)ac);
    }
}

template <bool STATS>
__global__ void __launch_bounds__(8 * CSG_WARP) k_walk64_exact(WalkArgs a)
{
    __shared__ NodeW64 win_all[8][CSG_WARP];
    NodeW64 *win = win_all[threadIdx.x >> 5];
    WalkStats st;
    for_each_task<8, false>(a, [&](const TaskRange &tr) { walk64_exact_task<STATS>(a, win, tr, st); });
    if (STATS)
        add_hits(a, st);
}

// m/r^3 for the queued FP64 walk without FP64 operations (the FP64 pipe is
// the walk's bottleneck on this GPU): from the FP32 rsqrt seed y0 (rel.
// error < 2^-21) by integer arithmetic (m_r3_from_seed: the series of
// (1-e)^-3/2, e = 1 - r2 y0^2, one rounding). The seed's conversion is a bit
// operation. Range checks on the exponents (2^-99 <= r2 < 2^100,
// 2^-863 <= m < 2^865) keep every integer step in range; outside them (and
// for m = 0) the plain expression.
__device__ __forceinline__ double m_inv_r3_q(double m, double r2)
{
    const long long bits = __double_as_longlong(r2);
    const long long mb = __double_as_longlong(m);
    if ((unsigned long long)((bits >> 52) - 924) <= 198ull && // sign clear, exponent 924..1122
        (unsigned long long)((mb >> 52) - 160) < 1728ull)     // sign clear, exponent 160..1887
        return m_r3_from_seed(bits, mb, rsqrtf(f32_from_f64_bits(bits)));
    return m / (r2 * sqrt(r2));
}

// ---- traversal in rounds ----------------------------------------------------
//
// A warp walks the tree for its 32 bodies from a stack of (cell, lanes that
// reached it) in shared memory, up to 32 cells a round. First every lane takes
// one cell and compares it with the box of the 32 bodies: a cell whose
// opening test must come out the same for every point of the box (and every
// leaf) is settled for all lanes at once; only the rest ("undecided", 15% of
// the cells at 1M bodies, theta 0.5, 25% in the 100k merger) is tested lane by lane. The round then
// hands the accepted cells to the warp's sink, tests the undecided ones, and
// pushes the children of opened cells with the lanes that opened them. So
// every body meets exactly the cells that the reference's walk accepts for it.
//
// Why: visiting one cell per warp step with all lanes took about 66
// instructions a step (3574 steps per 32 bodies at 1M, theta 0.5), of which
// the pair term was a fifth, and 32 dependent steps where a round has one.
// Classifying 32 cells with one instruction stream and evaluating without a
// decision per step takes about 25 a cell. FP32-mixed walk, alone, per cell step
// before -> in rounds: 1M 8.43 -> 4.03 ms, 100k merger 0.66 -> 0.30 ms, 64
// galaxies 3.40 -> 2.48 ms; 10k-body interaction lists 0.25 -> 0.13 ms. It is
// bound by instruction issue (67% busy at 1M); 42% of the lane slots idle in
// cells that only some lanes reach. Measured and not used: starting the next
// round's loads before this round's evaluations (12 more live registers: 1M
// 4.28-4.5 ms), 24 resident warps per SM (more spills: 4.31 ms).
//
// Children come from the child table (8 ids per cell), loaded before the
// round's evaluations and used after them. Opened cells whose children find no
// room on the stack go back on it themselves, marked; if not one cell's
// children fit (deeper than any tree built here, but a caller's pool may have
// thousands of levels) that cell's subtree is walked stackless, cell by cell.
constexpr int RND_STACK = 384; // 1M, theta 0.5: fits all but rare rounds (256: 6% slower)
constexpr int RND_PAIRS = 17;  // accepted cells from pair 0, undecided from the next pair on
constexpr int RND_REC = 20;    // words per staged pair
constexpr unsigned RND_OPEN = 0x80000000u; // stack entry: known open, children not pushed yet

typedef unsigned long long u64;

struct __align__(16) RoundShared {
    float4 box[2];                  // centre and half extents (rounded up) of the 32 bodies
    float rec[RND_PAIRS * RND_REC]; // staged cells, two per record: word 2 k + half of field k
    uint2 stk[RND_STACK];           // cell, lanes
    unsigned open[CSG_WARP];        // lanes that opened undecided cell e
};

// Packed FP32 pairs (two lanes of one 64-bit register): each half rounds as
// the scalar operation does.
__device__ __forceinline__ u64 pack2(float lo, float hi)
{
    return (u64)__float_as_uint(lo) | ((u64)__float_as_uint(hi) << 32);
}
__device__ __forceinline__ float lo2(u64 v) { return __uint_as_float((unsigned)v); }
__device__ __forceinline__ float hi2(u64 v) { return __uint_as_float((unsigned)(v >> 32)); }
__device__ __forceinline__ u64 add2(u64 a, u64 b)
{
    u64 d;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
    return d;
}
__device__ __forceinline__ u64 mul2(u64 a, u64 b)
{
    u64 d;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
    return d;
}
__device__ __forceinline__ u64 fma2(u64 a, u64 b, u64 c)
{
    u64 d;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
    return d;
}
__device__ __forceinline__ u64 sub2(u64 a, u64 b) // a - b: -1 b + a rounds once
{
    return fma2(b, pack2(-1.0f, -1.0f), a);
}

// A lane's body: its index and the FP32 high and low parts of its position.
struct LaneBody {
    bool valid;
    int me;
    int pos0; // the task's first sorted position
    unsigned bit;
    float hx, hy, hz, lx, ly, lz;
};

__device__ __forceinline__ float warp_minf(float v)
{
#pragma unroll
    for (int o = 16; o; o >>= 1)
        v = fminf(v, __shfl_xor_sync(0xffffffffu, v, o));
    return v;
}
__device__ __forceinline__ float warp_maxf(float v)
{
#pragma unroll
    for (int o = 16; o; o >>= 1)
        v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
    return v;
}

__device__ __forceinline__ LaneBody lane_body(const WalkArgs &a, RoundShared &sh,
                                              const TaskRange &tr)
{
    LaneBody L;
    const int lane = threadIdx.x & 31;
    L.valid = lane < tr.count;
    L.bit = 1u << lane;
    L.pos0 = tr.pos0;
    // lanes without a body stand at the first body (they widen no box)
    const int b = a.perm[tr.pos0 + (L.valid ? lane : 0)];
    L.me = L.valid ? b : -1;
    const double px = a.x[b], py = a.y[b], pz = a.z[b];
    L.hx = (float)px;
    L.hy = (float)py;
    L.hz = (float)pz;
    L.lx = (float)(px - (double)L.hx);
    L.ly = (float)(py - (double)L.hy);
    L.lz = (float)(pz - (double)L.hz);
    const float bx = 0.5f * (warp_minf(L.hx) + warp_maxf(L.hx));
    const float by = 0.5f * (warp_minf(L.hy) + warp_maxf(L.hy));
    const float bz = 0.5f * (warp_minf(L.hz) + warp_maxf(L.hz));
    const float ex = warp_maxf(fabsf((L.hx - bx) + L.lx)) * (1.0f + 0x1p-20f);
    const float ey = warp_maxf(fabsf((L.hy - by) + L.ly)) * (1.0f + 0x1p-20f);
    const float ez = warp_maxf(fabsf((L.hz - bz) + L.lz)) * (1.0f + 0x1p-20f);
    if (lane == 0) { // in shared memory: the registers stay with the sums
        sh.box[0] = make_float4(bx, by, bz, 0.0f);
        sh.box[1] = make_float4(ex, ey, ez, 0.0f);
    }
    __syncwarp();
    return L;
}

// The reference's FP64 opening test, for the rare cell inside the FP32 band.
__device__ __noinline__ bool decide64(const WalkArgs &a, int cell, int me)
{
    const NodeW64 e = a.w64[cell];
    const double ex = e.cx - a.x[me], ey = e.cy - a.y[me], ez = e.cz - a.z[me];
    return accept64(e.s2, ex * ex + ey * ey + ez * ez, a);
}

__device__ __forceinline__ void stage_cell(float *rec, int e, const float4 &A, const float4 &B,
                                           unsigned mask, int cell)
{
    float *r = rec + (e >> 1) * RND_REC + (e & 1);
    r[0] = A.x;
    r[2] = A.y;
    r[4] = A.z;
    r[6] = A.w;
    r[8] = B.x;
    r[10] = B.y;
    r[12] = B.z;
    r[14] = B.w;
    r[16] = __uint_as_float(mask);
    r[18] = __int_as_float(cell);
}

// The second half of an odd pair: no lane takes it (its other words are stale
// but finite).
__device__ __forceinline__ void stage_none(float *rec, int e)
{
    rec[(e >> 1) * RND_REC + (e & 1) + 16] = 0.0f;
}

__device__ __forceinline__ unsigned staged_mask(const float *rec, int e)
{
    return __float_as_uint(rec[(e >> 1) * RND_REC + (e & 1) + 16]);
}
__device__ __forceinline__ int staged_cell(const float *rec, int e)
{
    return __float_as_int(rec[(e >> 1) * RND_REC + (e & 1) + 18]);
}

// What every sink knows of its lane: the body, its lane bit and minus its
// position in FP32 parts, duplicated for packed use.
struct LanePos {
    u64 nhx, nhy, nhz, nlx, nly, nlz;
    unsigned bit;
    int me;

    __device__ __forceinline__ explicit LanePos(const LaneBody &L)
        : nhx(pack2(-L.hx, -L.hx)), nhy(pack2(-L.hy, -L.hy)), nhz(pack2(-L.hz, -L.hz)),
          nlx(pack2(-L.lx, -L.lx)), nly(pack2(-L.ly, -L.ly)), nlz(pack2(-L.lz, -L.lz)),
          bit(L.bit), me(L.me)
    {
    }
};

// The sink's view of a round:
//   accept(rec, n)  n accepted cells staged from rec, with the lanes that take
//                   each (the lanes that reached it, less a leaf's own body)
//   terms(...)      two undecided cells: differences, d^2, masses, whether
//                   this lane takes each, and their ids
//
// A cell tested by every lane for itself, outside a round (the root; cells of
// a subtree walked stackless). Sets take/open for the lane.
template <class Sink>
__device__ __forceinline__ void lane_test(const WalkArgs &a, const LaneBody &L, int cell,
                                          bool active, int &next, bool &take, bool &open,
                                          Sink &sink)
{
    const float4 *w = (const float4 *)(a.w32 + cell);
    const float4 A = __ldg(w), B = __ldg(w + 1);
    const int2 nb = __ldg((const int2 *)(w + 2));
    next = nb.x;
    const float dx = (A.x - L.hx) + (B.x - L.lx);
    const float dy = (A.y - L.hy) + (B.y - L.ly);
    const float dz = (A.z - L.hz) + (B.z - L.lz);
    const float d2 = fmaf(dx, dx, fmaf(dy, dy, dz * dz));
    take = open = false;
    if (A.w == 0.0f && a.w64[cell].m == 0.0) // empty (src/octree.c:181-182): nothing below counts
        return;
    if (nb.y >= 0) {
        take = active && nb.y != L.me;
    } else if (active) {
        take = B.w * a.acc_k < d2;
        if (!take && !(B.w * a.opn_k > d2))
            take = decide64(a, cell, L.me);
        open = !take;
    }
    sink.terms(pack2(dx, dx), pack2(dy, dy), pack2(dz, dz), pack2(d2, d2), pack2(A.w, A.w), take,
               false, cell, cell);
}

// The subtree of `top` for the lanes of `mask`, one cell per step in preorder
// (no stack: a lane sleeps below `skip`).
template <bool STATS, class Sink>
__device__ __forceinline__ void walk_stackless(const WalkArgs &a, const LaneBody &L, int top,
                                               unsigned mask, Sink &sink, WalkStats &st)
{
    const int end = max(top + 1, __ldg(&a.w32[top].next));
    int skip = (mask & L.bit) ? top : INT_MAX;
    for (int cur = top; cur < end;) {
        const bool active = cur >= skip;
        int next;
        bool take, open;
        if (STATS) {
            st.steps++;
            st.active += active;
        }
        lane_test(a, L, cur, active, next, take, open, sink);
        if (STATS)
            st.hits += take;
        if (active && !open)
            skip = next;
        cur = max(__any_sync(0xffffffffu, open) ? cur + 1 : next, cur + 1);
    }
}

// One lane's cell of a round.
struct RoundCell {
    int cell;
    unsigned mask; // lanes that reached it (0: no cell)
    bool again;    // opened in an earlier round, its children had no room
    float4 A, B;   // hi centre of mass, mass; lo centre of mass, s^2
    int first, body;
};

// Takes up to 32 cells off the stack, one per lane, and starts their loads.
__device__ __forceinline__ RoundCell round_pop(const WalkArgs &a, const RoundShared &sh, int &sp)
{
    const int lane = threadIdx.x & 31;
    const int k = min(CSG_WARP, sp);
    sp -= k;
    const uint2 ent = sh.stk[sp + (lane < k ? lane : 0)];
    RoundCell c;
    c.cell = (int)(ent.x & ~RND_OPEN);
    c.mask = lane < k ? ent.y : 0u;
    c.again = lane < k && (ent.x & RND_OPEN);
    const float4 *w = (const float4 *)(a.w32 + c.cell);
    c.A = __ldg(w);
    c.B = __ldg(w + 1);
    const int4 n = __ldg((const int4 *)(w + 2));
    c.body = n.y;
    c.first = n.w;
    return c;
}

// Walks the stack's cells (sp of them) and everything below them.
template <bool STATS, class Sink>
__device__ __forceinline__ void walk_rounds(const WalkArgs &a, RoundShared &sh, const LaneBody &L,
                                            int sp, Sink &sink, WalkStats &st)
{
    const int lane = threadIdx.x & 31;
    const unsigned lt = L.bit - 1u;
    while (sp > 0) {
        const RoundCell c = round_pop(a, sh, sp);
        const float4 bc = sh.box[0], be = sh.box[1];
        if (STATS) {
            st.steps += __popc(__ballot_sync(0xffffffffu, c.mask && !c.again));
            st.active += c.again ? 0 : __popc(c.mask);
        }
        // the box's nearest and farthest point, in FP32 with the rounding of
        // the differences (2^-22) covered by 2^-20, so that a cell called
        // accepted (opened) is accepted (opened) by every lane's own test
        const float dx = fabsf((c.A.x - bc.x) + c.B.x), dy = fabsf((c.A.y - bc.y) + c.B.y),
                    dz = fabsf((c.A.z - bc.z) + c.B.z);
        const float nx = fmaxf(fmaf(dx, 1.0f - 0x1p-20f, -be.x), 0.0f),
                    ny = fmaxf(fmaf(dy, 1.0f - 0x1p-20f, -be.y), 0.0f),
                    nz = fmaxf(fmaf(dz, 1.0f - 0x1p-20f, -be.z), 0.0f);
        const float fx = fmaf(dx, 1.0f + 0x1p-20f, be.x), fy = fmaf(dy, 1.0f + 0x1p-20f, be.y),
                    fz = fmaf(dz, 1.0f + 0x1p-20f, be.z);
        bool live = c.mask != 0u && !c.again;
        if (c.A.w == 0.0f && live && a.w64[c.cell].m == 0.0)
            live = false; // empty cell of a caller's pool
        const bool acc =
            live && (c.body >= 0 || c.B.w * a.acc_k < fmaf(nx, nx, fmaf(ny, ny, nz * nz)));
        const bool opn =
            c.again || (live && !acc && c.B.w * a.opn_k > fmaf(fx, fx, fmaf(fy, fy, fz * fz)));
        const bool und = live && !acc && !opn;
        const unsigned bacc = __ballot_sync(0xffffffffu, acc);
        const unsigned bund = __ballot_sync(0xffffffffu, und);
        int4 c03 = make_int4(-1, -1, -1, -1), c47 = c03;
        if (opn || und) { // used after the undecided cells' tests
            const int4 *cp = (const int4 *)(a.child + 8 * (size_t)c.cell);
            c03 = __ldg(cp);
            c47 = __ldg(cp + 1);
        }
        const int na = __popc(bacc), nu = __popc(bund);
        const int ub = (na + 1) & ~1; // place of the first undecided cell
        const int place = acc ? __popc(bacc & lt) : ub + __popc(bund & lt);
        unsigned tm = c.mask; // lanes that take an accepted cell: a leaf's own body does not
        if (c.body >= 0 && (unsigned)(c.first - L.pos0) < CSG_WARP)
            tm &= ~(1u << (c.first - L.pos0));
        if (acc || und)
            stage_cell(sh.rec, place, c.A, c.B, tm, c.cell);
        if (lane == 0 && (na & 1))
            stage_none(sh.rec, na);
        if (lane == 1 && (nu & 1))
            stage_none(sh.rec, ub + nu);
        __syncwarp();
        if (STATS)
            for (int e = 0; e < na; e++)
                st.hits += (staged_mask(sh.rec, e) & L.bit) != 0u;
        const u64 acck = pack2(a.acc_k, a.acc_k), opnk = pack2(a.opn_k, a.opn_k);
        for (int e = 0; e < nu; e += 2) {
            const ulonglong2 *r = (const ulonglong2 *)(sh.rec + ((ub + e) >> 1) * RND_REC);
            const ulonglong2 q0 = r[0], q1 = r[1], q2 = r[2], q3 = r[3];
            const int4 t = *(const int4 *)(r + 4); // masks, cells
            const u64 ux = add2(add2(q0.x, sink.nhx), add2(q2.x, sink.nlx));
            const u64 uy = add2(add2(q0.y, sink.nhy), add2(q2.y, sink.nly));
            const u64 uz = add2(add2(q1.x, sink.nhz), add2(q3.x, sink.nlz));
            const u64 d2 = fma2(ux, ux, fma2(uy, uy, mul2(uz, uz)));
            const u64 sa = mul2(q3.y, acck), so = mul2(q3.y, opnk);
            const bool act0 = t.x & L.bit, act1 = t.y & L.bit;
            bool acc0 = lo2(sa) < lo2(d2), acc1 = hi2(sa) < hi2(d2); // implies d2 > 0
            const bool amb0 = act0 && !acc0 && !(lo2(so) > lo2(d2));
            const bool amb1 = act1 && !acc1 && !(hi2(so) > hi2(d2));
            if (amb0 || amb1) { // inside the FP32 band: rare
                if (amb0)
                    acc0 = decide64(a, t.z, L.me);
                if (amb1)
                    acc1 = decide64(a, t.w, L.me);
            }
            const bool take0 = act0 && acc0, take1 = act1 && acc1;
            const unsigned o0 = __ballot_sync(0xffffffffu, act0 && !acc0);
            const unsigned o1 = __ballot_sync(0xffffffffu, act1 && !acc1);
            if (lane == 0)
                *(uint2 *)&sh.open[e] = make_uint2(o0, o1);
            if (STATS)
                st.hits += take0 + take1;
            sink.terms(ux, uy, uz, d2, q1.y, take0, take1, t.z, t.w);
        }
        __syncwarp();
        const unsigned om = opn ? c.mask : und ? sh.open[place - ub] : 0u;
        const int ch[8] = {c03.x, c03.y, c03.z, c03.w, c47.x, c47.y, c47.z, c47.w};
        int cnt = 0;
        if (om) {
#pragma unroll
            for (int q = 0; q < 8; q++)
                cnt += ch[q] > c.cell; // preorder: a child's id is above its parent's
        }
        int at = cnt;
#pragma unroll
        for (int o = 1; o < CSG_WARP; o <<= 1) {
            const int v = __shfl_up_sync(0xffffffffu, at, o);
            if (lane >= o)
                at += v;
        }
        int total = __shfl_sync(0xffffffffu, at, 31);
        if (total > RND_STACK - sp) { // warp-uniform; at least one place per cell is free
            const unsigned bo = __ballot_sync(0xffffffffu, cnt > 0);
            // children of the first cells, as far as every later cell keeps a place
            const bool fits = at + __popc(bo & ~lt & ~L.bit) <= RND_STACK - sp;
            unsigned keep = __ballot_sync(0xffffffffu, cnt > 0 && !fits);
            const int f = __ffs(keep) - 1;
            total = __shfl_sync(0xffffffffu, at - cnt, f);
            if (keep == bo) { // not even one: walk the first cell's subtree without the stack
                walk_stackless<STATS>(a, L, __shfl_sync(0xffffffffu, c.cell, f),
                                      __shfl_sync(0xffffffffu, om, f), sink, st);
                if (lane == f)
                    cnt = 0;
                keep &= keep - 1u;
            }
            if (keep & L.bit) {
                sh.stk[sp + __popc(keep & lt)] = make_uint2((unsigned)c.cell | RND_OPEN, om);
                cnt = 0;
            }
            sp += __popc(keep);
        }
        at += sp - cnt;
        if (cnt > 0) {
#pragma unroll
            for (int q = 0; q < 8; q++)
                if (ch[q] > c.cell)
                    sh.stk[at++] = make_uint2((unsigned)ch[q], om);
        }
        sp += total;
        __syncwarp();
        sink.accept(sh.rec, na);
        __syncwarp(); // records read before they are staged again
    }
}

// The walk of one cell's subtree for the lanes of `mask`.
template <bool STATS, class Sink>
__device__ __forceinline__ void walk_subtree(const WalkArgs &a, RoundShared &sh, const LaneBody &L,
                                             int cell, unsigned mask, Sink &sink, WalkStats &st)
{
    if ((threadIdx.x & 31) == 0)
        sh.stk[0] = make_uint2((unsigned)cell, mask);
    __syncwarp();
    walk_rounds<STATS>(a, sh, L, 1, sink, st);
}

// The k-th existing child of a cell, or -1.
__device__ __forceinline__ int nth_child(const WalkArgs &a, int cell, int k)
{
    int found = -1;
    for (int q = 0; q < 8; q++) {
        const int c = __ldg(&a.child[8 * (size_t)cell + q]);
        if (c > cell && k-- == 0)
            found = c;
    }
    return found;
}

__device__ __forceinline__ void kahan_add2(u64 &s, u64 &c, u64 v)
{
    const u64 y = sub2(v, c);
    const u64 t = add2(s, y);
    c = sub2(sub2(t, s), y);
    s = t;
}

// FP32-mixed sums: pair terms in FP32 from ~48-bit position differences, two
// cells at a time in packed arithmetic; the terms of a round (at most 17 per
// half, 8 on average) are added with Kahan compensation (per-body compensated
// FP32 summation); G applied once. Lanes that do not take a cell add zero.
//
// A large system's task sums the whole tree in one go. A small system's
// (split_max bodies or fewer) closes its sums into double partials: first the
// root's own term, then one per child subtree of the system's root
// ("segment" k < 8, in child order); the body's acceleration is G times the
// sum of the partials in that order. Its tasks can so be walked by one warp
// (all segments in turn) or by eight (one segment each; unit 0 also takes the
// root's term, and 0 + root is the root exactly; the partials added by
// k_walk_sum) with the same bits; the launch picks by the tasks it has. Which
// sum a system gets depends on its own size only, so that it comes out the
// same alone and in an ensemble.
constexpr int WSEGS = 8;

struct Sum32 : LanePos {
    u64 eps2;
    u64 bx, by, bz;             // current block
    u64 sx, sy, sz, cx, cy, cz; // compensated sums

    __device__ __forceinline__ Sum32(const WalkArgs &a, const LaneBody &L)
        : LanePos(L), eps2(pack2(a.eps2f, a.eps2f))
    {
        clear();
    }
    __device__ __forceinline__ void clear()
    {
        bx = by = bz = sx = sy = sz = cx = cy = cz = 0ull;
    }
    __device__ __forceinline__ void fold()
    {
        kahan_add2(sx, cx, bx);
        kahan_add2(sy, cy, by);
        kahan_add2(sz, cz, bz);
        bx = by = bz = 0ull;
    }
    static __device__ __forceinline__ float rsq(float r2) // r2 >= eps2f, a normal number
    {
        float y;
        asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(r2));
        return y;
    }
    __device__ __forceinline__ void pair(u64 dx, u64 dy, u64 dz, u64 r2, u64 m, bool t0, bool t1)
    {
        const u64 y = pack2(rsq(lo2(r2)), rsq(hi2(r2)));
        const u64 f0 = mul2(m, mul2(y, mul2(y, y)));
        const u64 f = pack2(t0 ? lo2(f0) : 0.0f, t1 ? hi2(f0) : 0.0f);
        bx = fma2(f, dx, bx);
        by = fma2(f, dy, by);
        bz = fma2(f, dz, bz);
    }
    __device__ __forceinline__ void accept(const float *rec, int n)
    {
#pragma unroll 2
        for (int e = 0; e < n; e += 2) {
            const ulonglong2 *r = (const ulonglong2 *)(rec + (e >> 1) * RND_REC);
            const ulonglong2 q0 = r[0], q1 = r[1], q2 = r[2], q3 = r[3];
            const uint2 t = *(const uint2 *)(r + 4); // masks
            const u64 dx = add2(add2(q0.x, nhx), add2(q2.x, nlx));
            const u64 dy = add2(add2(q0.y, nhy), add2(q2.y, nly));
            const u64 dz = add2(add2(q1.x, nhz), add2(q3.x, nlz));
            const u64 r2 = fma2(dx, dx, fma2(dy, dy, fma2(dz, dz, eps2)));
            pair(dx, dy, dz, r2, q1.y, t.x & bit, t.y & bit);
        }
        fold();
    }
    __device__ __forceinline__ void terms(u64 dx, u64 dy, u64 dz, u64 d2, u64 m, bool t0, bool t1,
                                          int, int)
    {
        pair(dx, dy, dz, add2(d2, eps2), m, t0, t1);
    }
    // one component's halves as a double: the FP32 sum of the two, its
    // rounding error (two-sum) joining the compensations
    static __device__ __forceinline__ double join(u64 s, u64 c)
    {
        const float p = lo2(s), q = hi2(s), t = p + q, w = t - p;
        const float e = (p - (t - w)) + (q - w);
        return (double)t - (double)((lo2(c) + hi2(c)) - e);
    }
    // the sums so far as doubles; starts the next segment
    __device__ __forceinline__ void close(double &x, double &y, double &z)
    {
        fold();
        x = join(sx, cx);
        y = join(sy, cy);
        z = join(sz, cz);
        clear();
    }
};

// Per-warp shared memory of the FP32 walk: the round's and the double sums
// (3 x 32, here so that the registers stay with the traversal). Staged words
// start finite: the second half of an odd pair may be read before it is
// written (its term is discarded, but zero times a NaN would not be zero).
struct __align__(16) Walk32Shared {
    RoundShared r;
    double g[3 * CSG_WARP];
};

__device__ __forceinline__ void clear_rec(RoundShared &sh)
{
    for (int i = threadIdx.x & 31; i < RND_PAIRS * RND_REC; i += CSG_WARP)
        sh.rec[i] = 0.0f;
    __syncwarp();
}

// The root: taken or opened lane by lane; returns the lanes that open it.
// count: this warp's takes count (one of a split task's units counts them).
template <bool STATS, class Sink>
__device__ __forceinline__ unsigned walk_root(const WalkArgs &a, const LaneBody &L,
                                              const TaskRange &tr, Sink &sink, WalkStats &st,
                                              bool count = true)
{
    int next;
    bool take, open;
    if (STATS) {
        st.steps++;
        st.active += L.valid;
    }
    lane_test(a, L, tr.root, L.valid, next, take, open, sink);
    if (STATS)
        st.hits += count && take;
    return __ballot_sync(0xffffffffu, open);
}

// The whole task by one warp: a large system's tree from the root; a small
// system's root, then each child subtree of it as a segment, every one closed
// into the double sum g.
template <bool STATS>
__device__ __forceinline__ void walk32_task(const WalkArgs &a, Walk32Shared &sh,
                                            const TaskRange &tr, WalkStats &st)
{
    const int lane = threadIdx.x & 31;
    double *g = sh.g + lane;
    clear_rec(sh.r);
    const LaneBody L = lane_body(a, sh.r, tr);
    Sum32 sum(a, L);
    double x = 0.0, y = 0.0, z = 0.0;
    unsigned go = __ballot_sync(0xffffffffu, L.valid);
    int q = -1; // whole: one subtree, the root's; else the root's children
    if (tr.small) {
        go = walk_root<STATS>(a, L, tr, sum, st);
        sum.close(x, y, z);
        q = 0;
    }
    g[0] = x;
    g[CSG_WARP] = y;
    g[2 * CSG_WARP] = z;
    const int qend = tr.small ? (go ? 8 : 0) : 0;
    for (; q < qend; q++) {
        const int c = q < 0 ? tr.root : __ldg(&a.child[8 * (size_t)tr.root + q]);
        if (q >= 0 && c <= tr.root)
            continue;
        walk_subtree<STATS>(a, sh.r, L, c, go, sum, st);
        sum.close(x, y, z);
        g[0] += x;
        g[CSG_WARP] += y;
        g[2 * CSG_WARP] += z;
    }
    if (L.valid) {
        a.ax[L.me] = a.G * g[0];
        a.ay[L.me] = a.G * g[CSG_WARP];
        a.az[L.me] = a.G * g[2 * CSG_WARP];
    }
}

// Segment k < 8 of a task by one warp; its partial into part[k] (3 x pstride),
// segment 0's with the root's term added first (as the whole walk adds them:
// 0 + root is the root exactly). The root step runs for every k: it sets
// which lanes go on.
__device__ __forceinline__ void walk32_unit(const WalkArgs &a, Walk32Shared &sh,
                                            const TaskRange &tr, int k, double *part,
                                            long long pstride)
{
    WalkStats st;
    clear_rec(sh.r);
    const LaneBody L = lane_body(a, sh.r, tr);
    Sum32 sum(a, L);
    const unsigned open = walk_root<false>(a, L, tr, sum, st);
    double rx, ry, rz, x = 0.0, y = 0.0, z = 0.0;
    sum.close(rx, ry, rz);
    double *g = sh.g + (threadIdx.x & 31);
    g[0] = rx;
    g[CSG_WARP] = ry;
    g[2 * CSG_WARP] = rz;
    const int c = nth_child(a, tr.root, k);
    if (open && c >= 0) {
        walk_subtree<false>(a, sh.r, L, c, open, sum, st);
        sum.close(x, y, z);
    }
    if (L.valid) {
        part[(3 * k + 0) * pstride + L.me] = k == 0 ? g[0] + x : x;
        part[(3 * k + 1) * pstride + L.me] = k == 0 ? g[CSG_WARP] + y : y;
        part[(3 * k + 2) * pstride + L.me] = k == 0 ? g[2 * CSG_WARP] + z : z;
    }
}

// a = G (part[0] + ... + part[7]) for every live body, in child order: the
// whole walk's own sum.
// With sys_n (an ensemble's FP64 walk): only bodies of systems of at most
// split_max bodies, the ones the split walk covered.
__global__ void k_walk_sum(const double *__restrict__ part, long long pstride,
                             const double *__restrict__ m, int n, double G, double *ax,
                             double *ay, double *az, const int *__restrict__ gid,
                             const int *__restrict__ sys_n, int split_max)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n || m[i] <= 0.0)
        return;
    if (sys_n && sys_n[gid[i]] > split_max)
        return; // walked whole, written by that walk
    double s[3] = {0.0, 0.0, 0.0};
#pragma unroll
    for (int k = 0; k < WSEGS; k++)
#pragma unroll
        for (int d = 0; d < 3; d++)
            s[d] += part[(3 * k + d) * pstride + i];
    ax[i] = G * s[0];
    ay[i] = G * s[1];
    az[i] = G * s[2];
}

// Resident warps per SM the FP32 walks' registers are sized for.
constexpr int WALK32_RES = 20;

// One warp per (task, segment): unit u walks segment u % 8 of task u / 8.
__global__ void __launch_bounds__(4 * CSG_WARP, WALK32_RES / 4) k_walk32_units(WalkArgs a, double *part,
                                                                   long long pstride)
{
    __shared__ Walk32Shared sh_all[4];
    const int nn = a.sc->n_nodes;
    if (nn > a.node_cap || nn < 1)
        return;
    const int u = blockIdx.x * 4 + (threadIdx.x >> 5);
    if (u >= a.sc->n_tasks * WSEGS)
        return;
    const WalkTask w = a.tasks[u / WSEGS];
    const DevRoot &r = a.roots[w.gal];
    const TaskRange tr{w.pos0, w.count, r.root, r.end, small_system(a, w.gal)};
    if (tr.root < 0 || tr.end > nn || tr.root >= tr.end)
        dev_fail(a.sc, CSG_ERR_WALK_LIMIT);
    else
        walk32_unit(a, sh_all[threadIdx.x >> 5], tr, u % WSEGS, part, pstride);
}

template <bool STATS, int WARPS, bool PERSIST>
__global__ void __launch_bounds__(WARPS * CSG_WARP, WALK32_RES / WARPS) k_walk32(WalkArgs a)
{
    __shared__ Walk32Shared sh_all[WARPS];
    Walk32Shared &sh = sh_all[threadIdx.x >> 5];
    WalkStats st;
    for_each_task<WARPS, PERSIST>(a, [&](const TaskRange &tr) { walk32_task<STATS>(a, sh, tr, st); });
    if (STATS)
        add_hits(a, st);
}

// FP64 evaluation: accepted cells are queued per lane in shared memory and
// evaluated in FP64 in batches where every lane has work, in the order they
// were accepted (the reference's depth-first order). The FP64 pipe then does
// useful work on (almost) every lane instead of once per traversal step for
// the few lanes that interact at that step.

// Loads queued entry s of the lane (its cell's centre of mass and mass), or
// zeros when s >= count (no queue read, no cell read). With MARK a negative
// entry is a segment marker (mk; nothing loaded).
template <int Q64, bool MARK>
__device__ __forceinline__ void q64_load(const WalkArgs &a, const int *q, int lane, int head, int s,
                                         int count, double2 &p01, double2 &p23, bool &mk)
{
    p01 = make_double2(0.0, 0.0);
    p23 = p01;
    mk = false;
    if (s < count) {
        const int c = q[((head + s) & (Q64 - 1)) * CSG_WARP + lane];
        if (MARK)
            mk = c < 0;
        if (!MARK || !mk) {
            p01 = __ldg((const double2 *)&a.w64[c]);     // cx, cy
            p23 = __ldg((const double2 *)&a.w64[c] + 1); // cz, m
        }
    }
}

__device__ __forceinline__ void q64_term(const WalkArgs &a, const double2 &p01, const double2 &p23,
                                         double px, double py, double pz, double &sx, double &sy,
                                         double &sz)
{
    const double dx = p01.x - px, dy = p01.y - py, dz = p23.x - pz;
    const double r2 = fma(dx, dx, fma(dy, dy, fma(dz, dz, a.eps2)));
    const double f = m_inv_r3_q(p23.y, r2);
    sx = fma(f, dx, sx);
    sy = fma(f, dy, sy);
    sz = fma(f, dz, sz);
}

// A unit's segment partials: part[(3 * k + d) * pstride + body].
__device__ __forceinline__ void put_partial(const WalkArgs &a, int k, int me, double sx, double sy,
                                            double sz)
{
    a.part[(3 * k + 0) * a.pstride + me] = sx;
    a.part[(3 * k + 1) * a.pstride + me] = sy;
    a.part[(3 * k + 2) * a.pstride + me] = sz;
}

// Evaluates the lane's next `count` queued entries (count >= 0; lanes without
// a body pass 0 and never read their queue), two at a time in queue order.
// The next two cells' loads are in flight while the current two are
// evaluated (few consumer warps per SM at small N, each waiting on its
// loads). MARK: a marker closes segment kc (its partial written, the sum
// restarted).
template <int Q64, bool MARK>
__device__ __forceinline__ void q64_eval(const WalkArgs &a, const int *q, int lane, int &head,
                                         int count, double px, double py, double pz,
                                         double &sx, double &sy, double &sz, int me, int &kc)
{
    count = max(count, 0);
    const int kmax = (int)__reduce_max_sync(0xffffffffu, (unsigned)count);
    double2 a01, a23, b01, b23;
    bool ma, mb;
    q64_load<Q64, MARK>(a, q, lane, head, 0, count, a01, a23, ma);
    q64_load<Q64, MARK>(a, q, lane, head, 1, count, b01, b23, mb);
    for (int s = 0; s < kmax; s += 2) {
        double2 c01, c23, d01, d23;
        bool mc, md;
        q64_load<Q64, MARK>(a, q, lane, head, s + 2, count, c01, c23, mc);
        q64_load<Q64, MARK>(a, q, lane, head, s + 3, count, d01, d23, md);
        if (s < count) {
            if (MARK && ma) { // rare
                put_partial(a, kc++, me, sx, sy, sz);
                sx = sy = sz = 0.0;
            } else {
                q64_term(a, a01, a23, px, py, pz, sx, sy, sz);
            }
        }
        if (s + 1 < count) {
            if (MARK && mb) {
                put_partial(a, kc++, me, sx, sy, sz);
                sx = sy = sz = 0.0;
            } else {
                q64_term(a, b01, b23, px, py, pz, sx, sy, sz);
            }
        }
        a01 = c01;
        a23 = c23;
        b01 = d01;
        b23 = d23;
        ma = mc;
        mb = md;
    }
    head += count;
}

// FP64 walk, producer/consumer form. Each task has two warps: the producer
// walks the tree (in rounds, the FP32 decisions) and appends each lane's
// accepted cells to that lane's ring in shared memory; the consumer evaluates
// the rings in FP64, in the order the cells were accepted. The traversal
// (FP32/ALU pipes) and the evaluation (FP64 pipe) then overlap on every SM
// instead of alternating in one warp. The warps hand over through per-lane
// head and tail counters in shared memory; every wait polls with a sleep and
// gives up after a.wait_polls polls (recording CSG_ERR_DEVICE_WAIT, then both
// warps leave the task). A pair of the split form (G > 0) walks G segments
// of a task: the root step, then the subtrees of the root's children k0 ..
// k0 + G - 1, with a marker (-1) queued on every lane between two segments.
constexpr int WS_RING = 128;   // ring slots per lane (power of two)
constexpr int WS_BATCH = 8;    // dense batch the consumer waits for; fewer entries a lane once
                               // some lane's ring is half full (at 3/4: 1% slower at 1M; the
                               // producer needs room for a round, 32 entries, on every lane)

struct WsShared {
    int ring[WS_RING * CSG_WARP]; // slot-major: ring[slot * 32 + lane]
    int tail[CSG_WARP];           // published by the producer
    int head[CSG_WARP];           // published by the consumer
    int done;                     // producer finished (tails final)
    int broken;                   // a wait gave up: both warps leave
};

__device__ __forceinline__ int ws_load(const volatile int *p) { return *p; }

// The producer's sink: every taken cell goes to the lane's ring.
struct PushQueue : LanePos {
    WsShared &sh;
    DevScalars *sc;
    int wait_polls;
    int tail, head_seen, pairs;
    bool mute, broken;

    __device__ __forceinline__ PushQueue(const WalkArgs &a, const LaneBody &L, WsShared &s)
        : LanePos(L), sh(s), sc(a.sc), wait_polls(a.wait_polls), tail(0), head_seen(0), pairs(0),
          mute(false), broken(false)
    {
    }
    __device__ __forceinline__ void publish()
    {
        __threadfence_block(); // ring entries before the tail
        ((volatile int *)sh.tail)[threadIdx.x & 31] = tail;
    }
    // waits (warp-uniform) until every lane's ring has room for n entries
    __device__ __forceinline__ void room(int n)
    {
        bool full = tail - head_seen + n > WS_RING;
        if (!__any_sync(0xffffffffu, full) || broken)
            return;
        publish();
        for (int i = 0; i < wait_polls; i++) {
            head_seen = ws_load(&sh.head[threadIdx.x & 31]);
            full = tail - head_seen + n > WS_RING;
            if (!__any_sync(0xffffffffu, full) || ws_load(&sh.broken))
                break;
            __nanosleep(64);
        }
        __threadfence_block(); // heads read before slots are overwritten
        if (__any_sync(0xffffffffu, full)) { // gave up (or the consumer did)
            if ((threadIdx.x & 31) == 0) {
                dev_fail(sc, CSG_ERR_DEVICE_WAIT);
                ((volatile int *)&sh.broken)[0] = 1;
            }
            broken = true;
        }
    }
    __device__ __forceinline__ void put(bool want, int value) // after room()
    {
        if (want && !broken) {
            sh.ring[(tail & (WS_RING - 1)) * CSG_WARP + (threadIdx.x & 31)] = value;
            tail++;
        }
    }
    __device__ __forceinline__ void accept(const float *rec, int n)
    {
        room(n);
        for (int e = 0; e < n; e++) {
            put(staged_mask(rec, e) & bit, staged_cell(rec, e));
        }
        publish();
    }
    __device__ __forceinline__ void terms(u64, u64, u64, u64, u64, bool t0, bool t1, int c0, int c1)
    {
        room(2);
        put(t0 && !mute, c0);
        put(t1 && !mute, c1);
        if ((++pairs & 3) == 0)
            publish();
    }
};

template <bool STATS, int G>
__device__ __forceinline__ void ws_produce(const WalkArgs &a, RoundShared &rs, WsShared &sh,
                                           const TaskRange &tr, int k0, WalkStats &st)
{
    const LaneBody L = lane_body(a, rs, tr);
    PushQueue q(a, L, sh);
    q.mute = G > 0 && k0 != 0; // the root's terms are segment 0's
    const unsigned open = walk_root<STATS>(a, L, tr, q, st, !q.mute);
    q.mute = false;
    int k = 0; // child (segment) number
    for (int o = 0; o < 8 && open; o++) {
        const int c = __ldg(&a.child[8 * (size_t)tr.root + o]);
        if (c <= tr.root)
            continue;
        if (G == 0 || (k >= k0 && k < k0 + G)) {
            if (G > 0 && k > k0) { // a segment marker
                q.room(1);
                q.put(L.valid, -1);
            }
            walk_subtree<STATS>(a, rs, L, c, open, q, st);
        }
        k++;
    }
    q.publish();
    __syncwarp();
    if ((threadIdx.x & 31) == 0)
        ((volatile int *)&sh.done)[0] = 1; // after every lane's final tail (fenced above)
}

template <int G>
__device__ __forceinline__ void ws_consume(const WalkArgs &a, WsShared &sh, const TaskRange &tr,
                                           int k0)
{
    const int lane = threadIdx.x & 31;
    const bool valid = lane < tr.count;
    const int me = valid ? a.perm[tr.pos0 + lane] : -1;
    const double px = valid ? a.x[me] : 0.0, py = valid ? a.y[me] : 0.0,
                 pz = valid ? a.z[me] : 0.0;
    double sx = 0.0, sy = 0.0, sz = 0.0;
    int head = 0, polls = 0, kc = k0; // kc: the segment being summed (split form)
    while (true) {
        const bool done = ws_load(&sh.done) != 0; // read before the tails: they are final then
        __threadfence_block();
        const int tail = ws_load(&sh.tail[lane]);
        __threadfence_block(); // the tail before the entries it covers
        const int avail = valid ? tail - head : 0;
        const int amin = (int)__reduce_min_sync(0xffffffffu, (unsigned)(valid ? avail : INT_MAX));
        const int amax = (int)__reduce_max_sync(0xffffffffu, (unsigned)avail);
        int take = 0;
        if (amin >= WS_BATCH)
            take = amin; // dense: every lane has work
        else if (done || amax >= WS_RING / 2)
            take = -1; // the rest (done), or relief for a lane without room for a round's entries
        if (take != 0) {
            const int n = take > 0 ? (valid ? take : 0) : min(avail, done ? avail : WS_BATCH);
            q64_eval<WS_RING, (G > 1)>(a, sh.ring, lane, head, n, px, py, pz, sx, sy, sz, me, kc);
            __threadfence_block(); // entries read before the head is published
            ((volatile int *)sh.head)[lane] = head;
            polls = 0;
            if (done && __all_sync(0xffffffffu, !valid || head == tail))
                break;
            continue;
        }
        if (ws_load(&sh.broken))
            return;
        if (++polls >= a.wait_polls) {
            if (lane == 0) {
                dev_fail(a.sc, CSG_ERR_DEVICE_WAIT);
                ((volatile int *)&sh.broken)[0] = 1;
            }
            return;
        }
        __nanosleep(64);
    }
    if (valid && G > 0) { // the last segment's partial (segment 0's with the root's term),
        put_partial(a, kc, me, sx, sy, sz); // zeros for segments the walk did not reach
        for (int kk = kc + 1; kk < k0 + G; kk++)
            put_partial(a, kk, me, 0.0, 0.0, 0.0);
    } else if (valid) {
        a.ax[me] = a.G * sx;
        a.ay[me] = a.G * sy;
        a.az[me] = a.G * sz;
    }
}

// PAIRS producer/consumer pairs per block (task t of the grid is pair
// t % PAIRS of block t / PAIRS), 10 pairs per SM either way (shared memory): one pair for
// launches of few tasks (finer blocks balance better over the SMs), two
// otherwise (measured faster from ~100k bodies on).
// One producer/consumer pair per task (G == 0) or per unit of G segments,
// u = (8 / G) * task + k0 / G (partials into a.part).
template <bool STATS, int PAIRS, int G>
__device__ __forceinline__ void walk64ws_body(const WalkArgs &a)
{
    __shared__ WsShared sh_all[PAIRS];
    __shared__ RoundShared rs_all[PAIRS];
    const int warp = threadIdx.x >> 5, pair = warp >> 1, lane = threadIdx.x & 31;
    WsShared &sh = sh_all[pair];
    const int nn = a.sc->n_nodes;
    if (nn > a.node_cap || nn < 1)
        return;
    const int u = blockIdx.x * PAIRS + pair;
    const int t = G > 0 ? u / (8 / G) : u, k0 = G > 0 ? (u % (8 / G)) * G : 0;
    TaskRange tr{0, 0, 0, 0, false};
    bool ok = t < a.sc->n_tasks;
    if (ok) {
        const WalkTask w = a.tasks[t];
        const DevRoot &r = a.roots[w.gal];
        tr = TaskRange{w.pos0, w.count, r.root, r.end, small_system(a, w.gal)};
        if (G > 0 ? !tr.small : (tr.small && a.skip_small)) {
            ok = false; // the other form walks this system
        } else if (tr.root < 0 || tr.end > nn || tr.root >= tr.end) {
            if ((warp & 1) == 0 && lane == 0)
                dev_fail(a.sc, CSG_ERR_WALK_LIMIT);
            ok = false;
        }
    }
    if (ok && (warp & 1) == 0) {
        sh.tail[lane] = 0;
        sh.head[lane] = 0;
        if (lane == 0) {
            sh.done = 0;
            sh.broken = 0;
        }
    }
    __syncthreads(); // every thread: counters set before either warp of any pair starts
    if (!ok)
        return; // both warps of the pair
    WalkStats st;
    if ((warp & 1) == 0)
        ws_produce<STATS, G>(a, rs_all[pair], sh, tr, k0, st);
    else
        ws_consume<G>(a, sh, tr, k0);
    if (STATS && (warp & 1) == 0)
        add_hits(a, st);
}

template <bool STATS, int PAIRS>
__global__ void __launch_bounds__(2 * PAIRS * CSG_WARP, 20 / (2 * PAIRS)) k_walk64ws(WalkArgs a)
{
    walk64ws_body<STATS, PAIRS, 0>(a);
}

// The FP64 walk split by the root's children (trees built here, few tasks
// for the GPU): partials into a.part, summed by k_walk_sum; the same bits as
// k_walk64ws.
template <bool STATS, int PAIRS, int G>
__global__ void __launch_bounds__(2 * PAIRS * CSG_WARP, 20 / (2 * PAIRS)) k_walk64ws_units(WalkArgs a)
{
    walk64ws_body<STATS, PAIRS, G>(a);
}

// Dead bodies get a = 0 (src/octree.c:226-230); alive ones are overwritten by
// the walk.
// Also rewinds the task counter of the persistent walks.
__global__ void k_zero_acc(const double *__restrict__ m, double *ax, double *ay, double *az, int n,
                           DevScalars *sc)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i == 0)
        sc->task_next = 0;
    if (i >= n)
        return;
    if (m[i] <= 0.0) {
        ax[i] = 0.0;
        ay[i] = 0.0;
        az[i] = 0.0;
    }
}

// Interaction lists: the cells each alive body interacts with (the FP64 walk's
// interaction set, in the order the walk meets them), written per caller
// index: ids[offs[i] .. offs[i] + counts[i]). FILL = false counts, FILL = true
// writes (offs from an exclusive scan of the counts).
template <bool FILL>
struct ListSink : LanePos {
    int *ids;
    int k, lim;

    __device__ __forceinline__ ListSink(const LaneBody &L) : LanePos(L), ids(nullptr), k(0), lim(0) {}
    __device__ __forceinline__ void put(bool want, int cell)
    {
        if (want) {
            if (FILL && k < lim)
                ids[k] = cell;
            k++;
        }
    }
    __device__ __forceinline__ void accept(const float *rec, int n)
    {
        for (int e = 0; e < n; e++) {
            put(staged_mask(rec, e) & bit, staged_cell(rec, e));
        }
    }
    __device__ __forceinline__ void terms(u64, u64, u64, u64, u64, bool t0, bool t1, int c0, int c1)
    {
        put(t0, c0);
        put(t1, c1);
    }
};

template <bool FILL, int WARPS>
__global__ void __launch_bounds__(WARPS * CSG_WARP) k_walk_lists(WalkArgs a, int *counts,
                                                             const int *offs, int *ids, int cap)
{
    __shared__ RoundShared rs_all[WARPS];
    RoundShared &rs = rs_all[threadIdx.x >> 5];
    for_each_task<WARPS, false>(a, [&](const TaskRange &tr) {
        const LaneBody L = lane_body(a, rs, tr);
        ListSink<FILL> q(L);
        if (FILL && L.valid) {
            const int base = offs[L.me];
            q.ids = ids + base;
            q.lim = min(counts[L.me], cap - base);
        }
        WalkStats st;
        walk_subtree<false>(a, rs, L, tr.root, __ballot_sync(0xffffffffu, L.valid), q, st);
        if (!FILL && L.valid)
            counts[L.me] = q.k;
    });
}

} // namespace

// ---- host side -------------------------------------------------------------

namespace {

WalkArgs walk_args(csgd_t *d, const csgd_force_params *p)
{
    WalkArgs a;
    a.perm = d->perm;
    a.x = d->x;
    a.y = d->y;
    a.z = d->z;
    a.w64 = d->w64;
    a.w32 = d->w32;
    a.child = d->child;
    a.tasks = d->tasks;
    a.roots = d->roots;
    a.sc = d->sc;
    a.wait_polls = csgd_wait_polls(d);
    a.ax = d->ax;
    a.ay = d->ay;
    a.az = d->az;
    a.G = p->G;
    a.eps2 = p->softening * p->softening;
    a.theta2 = p->theta * p->theta;
    a.t2lo = a.theta2 * (1.0 - 0x1p-50);
    a.t2hi = a.theta2 * (1.0 + 0x1p-50);
    a.Gf = (float)p->G;
    // at least the smallest normal number: no sum of squares below 2e-31
    // changes, and under that y^3 of the pair term overflows to inf either way
    a.eps2f = fmaxf((float)a.eps2, 1.17549435e-38f);
    // FP32 error band: |d| is exact to ~2^-46 |coordinates| (hi/lo pairs), d^2
    // to a few FP32 ulps, each product below to 2^-23; g = 2^-19 (1 + theta^2)
    // relative covers them with a wide margin. theta = 0 gives acc_k = opn_k =
    // inf: nothing is accepted, every cell with d^2 > 0 opens.
    const double g = 0x1p-19 * (1.0 + a.theta2);
    a.acc_k = (float)((1.0 + g) / a.theta2);
    a.opn_k = (float)((1.0 - g) / a.theta2);
    a.node_cap = d->node_cap;
    a.group = d->walk_group;
    a.sys_n = d->n_gal > 1 ? d->sys_n : nullptr;
    a.n_bodies = d->n;
    a.split_max = (int)csgd_split_max_bodies(d);
    a.skip_small = 0;
    return a;
}

// Kernel variant by (stats, persistent).
#define CSG_LAUNCH_WALK(K, W, grid, s, a)                                                  \
    do {                                                                                    \
        if (persist && stats)                                                               \
            K<true, W, true><<<grid, W * CSG_WARP, 0, s>>>(a);                              \
        else if (persist)                                                                   \
            K<false, W, true><<<grid, W * CSG_WARP, 0, s>>>(a);                             \
        else if (stats)                                                                     \
            K<true, W, false><<<grid, W * CSG_WARP, 0, s>>>(a);                             \
        else                                                                                \
            K<false, W, false><<<grid, W * CSG_WARP, 0, s>>>(a);                            \
    } while (0)


// One walk launch with the state's launch shape.
void launch_walk(csgd_t *d, const WalkArgs &a, int precision, int exact)
{
    cudaStream_t s = d->stream;
    const int W = d->walk_warps == 4 ? 4 : 8;
    const bool stats = d->stats != 0;
    const bool persist = a.group > 0 && !exact;
    WalkArgs b = a;
    if (!persist)
        b.group = 0;
    int grid;
    if (persist) {
        grid = d->num_sms * d->walk_bps;
    } else {
        const long long tasks = (long long)d->n / CSG_WARP + d->n_gal + 1; // >= n_tasks
        grid = (int)((tasks + W - 1) / W);
    }
    if (grid < 1)
        grid = 1;
    if (exact) {
        if (stats)
            k_walk64_exact<true><<<grid, 8 * CSG_WARP, 0, s>>>(b);
        else
            k_walk64_exact<false><<<grid, 8 * CSG_WARP, 0, s>>>(b);
    } else if (precision == CSG_PREC_FP32_MIXED && !stats && csgd_walk_split(d) &&
               d->wpart && d->wpart_cap >= d->n) {
        // few tasks for the GPU: eight warps per task, one per root child,
        // then the partials added in child order (the same bits as below)
        const long long units = ((long long)d->n / CSG_WARP + d->n_gal + 1) * WSEGS;
        k_walk32_units<<<(int)((units + 3) / 4), 4 * CSG_WARP, 0, s>>>(b, d->wpart,
                                                                       (long long)d->wpart_cap);
        d->launches++;
        k_walk_sum<<<csgd_grid(d->n, 256), 256, 0, s>>>(d->wpart, (long long)d->wpart_cap, d->m,
                                                          d->n, b.G, d->ax, d->ay, d->az, nullptr,
                                                          nullptr, 0);
    } else if (precision == CSG_PREC_FP32_MIXED) {
        if (W == 4)
            CSG_LAUNCH_WALK(k_walk32, 4, grid, s, b);
        else
            CSG_LAUNCH_WALK(k_walk32, 8, grid, s, b);
    } else { // FP64: producer/consumer pairs (the task group applies to FP32 only)
        // small systems (split_max bodies or fewer): pairs per (task, root
        // children), partials added by k_walk_sum; the rest a pair per task
        const bool units = d->wpart && d->wpart_cap >= d->n &&
                           csgd_sys_min_n(d) <= b.split_max;
        b.skip_small = units;
        if (units) {
            // G segments per pair: one while the units fit about four waves of
            // pairs (about 12 per SM), more (with markers between them) for larger launches
            const long long tasks = (long long)d->n / CSG_WARP + d->n_gal + 1;
            int g = 1;
            while (g < WSEGS && tasks * (WSEGS / g) > 4LL * 12 * d->num_sms)
                g *= 2;
            const long long nu = tasks * (WSEGS / g);
            const int pairs = nu > 8LL * d->num_sms ? 2 : 1;
            const int gw = (int)((nu + pairs - 1) / pairs);
            b.part = d->wpart;
            b.pstride = d->wpart_cap;
#define CSG_U(ST, P, GG) k_walk64ws_units<ST, P, GG><<<gw, 2 * P * CSG_WARP, 0, s>>>(b)
#define CSG_UG(ST, P)                                                                              \
    do {                                                                                          \
        if (g == 1)                                                                               \
            CSG_U(ST, P, 1);                                                                      \
        else if (g == 2)                                                                          \
            CSG_U(ST, P, 2);                                                                      \
        else if (g == 4)                                                                          \
            CSG_U(ST, P, 4);                                                                      \
        else                                                                                      \
            CSG_U(ST, P, 8);                                                                      \
    } while (0)
            if (pairs == 2 && stats)
                CSG_UG(true, 2);
            else if (pairs == 2)
                CSG_UG(false, 2);
            else if (stats)
                CSG_UG(true, 1);
            else
                CSG_UG(false, 1);
#undef CSG_UG
#undef CSG_U
            k_walk_sum<<<csgd_grid(d->n, 256), 256, 0, s>>>(d->wpart, (long long)d->wpart_cap,
                                                              d->m, d->n, b.G, d->ax, d->ay, d->az,
                                                              d->gid, b.sys_n, b.split_max);
            d->launches += 2;
            if (csgd_sys_max_n(d) <= b.split_max)
                return; // every system is small
        }
        const long long tasks = (long long)d->n / CSG_WARP + d->n_gal + 1; // >= n_tasks
        const int pairs = tasks > 8LL * d->num_sms ? 2 : 1;
        const int gw = (int)((tasks + pairs - 1) / pairs);
        const int threads = 2 * pairs * CSG_WARP;
        if (pairs == 2 && stats)
            k_walk64ws<true, 2><<<gw, threads, 0, s>>>(b);
        else if (pairs == 2)
            k_walk64ws<false, 2><<<gw, threads, 0, s>>>(b);
        else if (stats)
            k_walk64ws<true, 1><<<gw, threads, 0, s>>>(b);
        else
            k_walk64ws<false, 1><<<gw, threads, 0, s>>>(b);
    }
    d->launches++;
}

} // namespace

extern "C" int csgd_gravity_ex(csgd_t *d, const csgd_force_params *p, int exact)
{
    const int n = d->n;
    if (n <= 0)
        return CSG_OK;
    WalkArgs a = walk_args(d, p);
    if (exact) // the parity walk keeps one warp per task, 8 warps per block
        a.group = 0;
    cudaStream_t s = d->stream;
    cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
    if (cudaStreamIsCapturing(s, &cap) == cudaSuccess && cap == cudaStreamCaptureStatusNone) {
        const int rc = csgd_prepare_walk(d, p->precision); // a capture prepared it before
        if (rc)
            return rc;
    }
    { k_zero_acc<<<csgd_grid(n, 256), 256, 0, s>>>(d->m, d->ax, d->ay, d->az, n, d->sc); d->launches++; }
    if (exact) {
        const int saved = d->walk_warps;
        d->walk_warps = 8;
        launch_walk(d, a, p->precision, 1);
        d->walk_warps = saved;
    } else {
        launch_walk(d, a, p->precision, 0);
    }
    return csgd_check(d, cudaGetLastError());
}

extern "C" int csgd_gravity(csgd_t *d, const csgd_force_params *p)
{
    return csgd_gravity_ex(d, p, 0);
}

extern "C" int csgd_walk_lists(csgd_t *d, const csgd_force_params *p, int *counts,
                               const int *offs, int *ids, int cap, int fill)
{
    const int n = d->n;
    if (n <= 0)
        return CSG_OK;
    if (d->imported) { // lists are defined on trees built here
        return CSG_ERR_UNSUPPORTED;
    }
    WalkArgs a = walk_args(d, p);
    a.group = 0;
    const long long tasks = (long long)n / CSG_WARP + d->n_gal + 1;
    // few tasks (the adjoint's 10k bodies are ~313): 2-warp blocks spread them
    // over every SM instead of crowding 8 per SM on a quarter of the GPU
    if (tasks < 8LL * d->num_sms) {
        const int grid = (int)((tasks + 1) / 2);
        if (fill)
            { k_walk_lists<true, 2><<<grid, 2 * CSG_WARP, 0, d->stream>>>(a, counts, offs, ids, cap); d->launches++; }
        else
            { k_walk_lists<false, 2><<<grid, 2 * CSG_WARP, 0, d->stream>>>(a, counts, offs, ids, cap); d->launches++; }
    } else {
        const int grid = (int)((tasks + 7) / 8);
        if (fill)
            { k_walk_lists<true, 8><<<grid, 8 * CSG_WARP, 0, d->stream>>>(a, counts, offs, ids, cap); d->launches++; }
        else
            { k_walk_lists<false, 8><<<grid, 8 * CSG_WARP, 0, d->stream>>>(a, counts, offs, ids, cap); d->launches++; }
    }
    return csgd_check(d, cudaGetLastError());
}

// ---- launch shape and its autotuner ------------------------------------------

extern "C" int csgd_set_walk_shape(csgd_t *d, const CsgWalkShape *w)
{
    if (!w || (w->warps_per_block != 4 && w->warps_per_block != 8) || w->task_group < 0 ||
        w->task_group > 64 || (w->task_group > 0 && (w->blocks_per_sm < 1 || w->blocks_per_sm > 32))) {
        return CSG_ERR_BAD_ARG;
    }
    if (d->walk_warps != w->warps_per_block || d->walk_group != w->task_group ||
        d->walk_bps != w->blocks_per_sm)
        csgd_drop_graph(d); // the captured walk launch changes
    d->walk_warps = w->warps_per_block;
    d->walk_group = w->task_group;
    d->walk_bps = w->task_group > 0 ? w->blocks_per_sm : 0;
    return CSG_OK;
}

extern "C" void csgd_get_walk_shape(const csgd_t *d, CsgWalkShape *w)
{
    w->warps_per_block = d->walk_warps;
    w->task_group = d->walk_group;
    w->blocks_per_sm = d->walk_bps;
    w->ms = 0.0f;
}

// Times every candidate launch shape on the current tree (reps walks each,
// the median kept) and keeps the fastest. The walk's results do not depend on
// the shape: every body's sum is formed by one lane in the same order.
extern "C" int csgd_autotune_walk(csgd_t *d, const csgd_force_params *p, int reps,
                                  CsgWalkShape *out, CsgWalkShape *all, int all_cap,
                                  int *n_all)
{
    if (reps < 1 || reps > 64) {
        return CSG_ERR_BAD_ARG;
    }
    // persistent candidates: 8, 16 or 24 resident warps per SM (24 is what
    // their register allocation allows), task groups of 1, 2 or 4
    static const int groups[] = {1, 2, 4};
    static const int resident[] = {8, 16, 24};
    CsgWalkShape cand[2 * (1 + 9)];
    int nc = 0;
    for (int w = 4; w <= 8; w += 4) {
        cand[nc++] = CsgWalkShape{w, 0, 0, 0.0f};
        for (int g : groups)
            for (int rw : resident)
                cand[nc++] = CsgWalkShape{w, g, rw / w, 0.0f};
    }
    CsgWalkShape saved;
    csgd_get_walk_shape(d, &saved);
    cudaEvent_t e0, e1;
    if (cudaEventCreate(&e0) != cudaSuccess)
        return csgd_check(d, cudaGetLastError());
    if (cudaEventCreate(&e1) != cudaSuccess) {
        cudaEventDestroy(e0);
        return csgd_check(d, cudaGetLastError());
    }
    int rc = CSG_OK;
    int best = -1;
    for (int c = 0; c < nc && rc == CSG_OK; c++) {
        d->walk_warps = cand[c].warps_per_block;
        d->walk_group = cand[c].task_group;
        d->walk_bps = cand[c].blocks_per_sm;
        float t[64];
        for (int r = 0; r <= reps && rc == CSG_OK; r++) { // first run warms up
            cudaEventRecord(e0, d->stream);
            rc = csgd_gravity(d, p);
            cudaEventRecord(e1, d->stream);
            if (rc == CSG_OK)
                rc = csgd_sync(d);
            if (rc == CSG_OK && r > 0)
                cudaEventElapsedTime(&t[r - 1], e0, e1);
        }
        if (rc != CSG_OK)
            break;
        for (int i = 1; i < reps; i++) // insertion sort for the median
            for (int j = i; j > 0 && t[j] < t[j - 1]; j--) {
                float x = t[j];
                t[j] = t[j - 1];
                t[j - 1] = x;
            }
        cand[c].ms = t[reps / 2];
        if (best < 0 || cand[c].ms < cand[best].ms)
            best = c;
    }
    cudaEventDestroy(e0);
    cudaEventDestroy(e1);
    d->walk_warps = saved.warps_per_block;
    d->walk_group = saved.task_group;
    d->walk_bps = saved.blocks_per_sm;
    if (rc != CSG_OK)
        return rc;
    if (n_all)
        *n_all = nc;
    for (int c = 0; all && c < nc && c < all_cap; c++)
        all[c] = cand[c];
    rc = csgd_set_walk_shape(d, &cand[best]);
    if (out)
        *out = cand[best];
    return rc;
}
