// dev_walk.cu — Barnes-Hut gravity walks (reference src/octree.c:171-234).
//
// Both walks give every body exactly the reference's interaction set: the
// cells it accepts by the monopole test (s*s)/d^2 < theta^2 with d^2 > 0, or
// reaches as leaves other than itself (in the order of the rounds, not the
// reference's depth-first one).
//
// Traversal: one warp walks the tree for 32 bodies that are neighbours in key
// order, up to 32 cells a round (see "traversal in rounds" below).
//
// FP64 walk: the drop-in precision (k_walk64ws). Openings decided as in the
//   FP32 walk (equal to the reference's FP64 rounding); interactions queued
//   and evaluated densely by two further warps per task, differences and sums
//   in FP64 and m/r^3 by integers (dev_fixpair.cuh), small systems split by
//   child subtrees as in the FP32 walk (k_walk64ws_units). k_walk64_exact instead
//   uses the reference's own operation sequence per step (1/(r2*sqrt(r2)),
//   no fused multiply-add) — bit-identical results on the reference's own
//   tree; used by parity tests. It alone walks cell by cell: one cursor over
//   the preorder ids, each lane sleeping below an index `skip` (it accepted an
//   ancestor), the next 32 cells staged per warp in shared memory.
// FP32-mixed walk: positions and centres as float hi/lo pairs (differences
//   keep ~48 bits), rsqrt/products in FP32, Kahan-compensated FP32 sums per
//   body (small systems: per child subtree of the split cell, mostly the root,
//   added in FP64).
//   Openings within the FP32 error band of the threshold are decided in FP64,
//   so the interaction set equals the FP64 walk's. Small systems with few
//   tasks for the GPU are walked by eight warps per task, one per child
//   subtree (k_walk32_units), with the same bits as one warp per task (k_walk32).
#include "dev_fixpair.cuh"
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
    float eps2f;
    PairEps eps; // FP64 walk
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
    // n_bodies for one system) sum by the split cell's children; the FP64 whole-task
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
    int split;  // its children are the segments of a small system
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
        const TaskRange tr{w.pos0, w.count, r.root, r.end, r.split, small_system(a, w.gal)};
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
// decision per step takes about 25 a cell. FP32-mixed walk inside the substep, cell
// by cell -> in rounds: 1M 8.43 -> 4.17 ms, 100k merger 0.83 -> 0.35 ms, 64
// galaxies 3.40 -> 2.36 ms; 10k-body interaction lists 0.25 -> 0.13 ms. It is
// bound by instruction issue (67% busy at 1M); 42% of the lane slots idle in
// cells that only some lanes reach. Measured and not used: starting the next
// round's loads before the same round's evaluations (12 more live registers: 1M
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
constexpr int SUM_BLOCK = 16;  // undecided cells a block of uncompensated terms
constexpr unsigned RND_OPEN = 0x80000000u; // stack entry: known open, children not pushed yet

typedef unsigned long long u64;

struct __align__(16) RoundShared {
    float4 box[2];                  // centre and half extents (rounded up) of the 32 bodies
    float rec[RND_PAIRS * RND_REC]; // staged cells, two per record: word 2 k + half of field k
    uint2 stk[RND_STACK];           // cell, lanes
    uint2 open[CSG_WARP];           // lanes that opened, and that take, undecided cell e
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

// The sink's view of a round, by its kind:
//   pair terms (BLOCKS false)
//     accept(rec, n)  n accepted cells staged from rec, with the lanes that take
//                     each (the lanes that reached it, less a leaf's own body)
//     terms(...)      two undecided cells: differences, d^2, masses, whether
//                     this lane takes each
//     fold()          ends a block of uncompensated terms
//   interaction lists (BLOCKS true)
//     block(cell, w)  the round's cells, one per lane, and the lane's own takes:
//                     bit j for lane j's cell
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
    if constexpr (Sink::BLOCKS)
        sink.block(cell, take ? 1u : 0u);
    else
        sink.terms(pack2(dx, dx), pack2(dy, dy), pack2(dz, dz), pack2(d2, d2), pack2(A.w, A.w),
                   take, false);
}

// 32 x 32 bit transpose across the warp: bit l of lane j's x becomes bit j of
// lane l's result.
__device__ __forceinline__ unsigned warp_transpose(unsigned x)
{
    const int lane = threadIdx.x & 31;
    unsigned m = 0x0000ffffu; // bits whose index has no 'k'
#pragma unroll
    for (int k = 16; k; k >>= 1) {
        const unsigned y = __shfl_xor_sync(0xffffffffu, x, k);
        x = (lane & k) ? (x & ~m) | ((y & ~m) >> k) : (x & m) | ((y & m) << k);
        m ^= m << (k >> 1);
    }
    return x;
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
        if constexpr (!Sink::BLOCKS)
            sink.fold();
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
        // place of the first undecided cell (a list needs no accepted cell staged)
        const int ub = Sink::BLOCKS ? 0 : (na + 1) & ~1;
        const int place = acc ? __popc(bacc & lt) : ub + __popc(bund & lt);
        unsigned tm = c.mask; // lanes that take an accepted cell: a leaf's own body does not
        if (c.body >= 0 && (unsigned)(c.first - L.pos0) < CSG_WARP)
            tm &= ~(1u << (c.first - L.pos0));
        if ((acc && !Sink::BLOCKS) || und)
            stage_cell(sh.rec, place, c.A, c.B, tm, c.cell);
        if (!Sink::BLOCKS && lane == 0 && (na & 1))
            stage_none(sh.rec, na);
        if (lane == 1 && (nu & 1))
            stage_none(sh.rec, ub + nu);
        __syncwarp();
        if (STATS && acc)
            st.hits += __popc(tm);
        const u64 acck = pack2(a.acc_k, a.acc_k), opnk = pack2(a.opn_k, a.opn_k);
        for (int e = 0; e < nu;) {
            for (const int stop = Sink::BLOCKS ? nu : min(nu, e + SUM_BLOCK); e < stop; e += 2) {
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
                if constexpr (Sink::BLOCKS) {
                    const unsigned t0 = __ballot_sync(0xffffffffu, take0);
                    const unsigned t1 = __ballot_sync(0xffffffffu, take1);
                    if (lane == 0)
                        *(uint4 *)&sh.open[e] = make_uint4(o0, t0, o1, t1);
                } else {
                    if (lane == 0) {
                        sh.open[e].x = o0;
                        sh.open[e + 1].x = o1;
                    }
                    sink.terms(ux, uy, uz, d2, q1.y, take0, take1);
                }
                if (STATS)
                    st.hits += take0 + take1;
            }
            if constexpr (!Sink::BLOCKS)
                sink.fold();
        }
        __syncwarp();
        const unsigned om = opn ? c.mask : und ? sh.open[place - ub].x : 0u;
        if constexpr (Sink::BLOCKS)
            sink.block(c.cell, warp_transpose(acc ? tm : und ? sh.open[place].y : 0u));
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
        if constexpr (!Sink::BLOCKS)
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
// cells at a time in packed arithmetic; blocks of them are added with Kahan
// compensation (per-body compensated FP32 summation); G applied once. Lanes
// that do not take a cell add zero. A block is a chain of at most 8 additions per
// half: 8 undecided pairs, or a round's accepted pairs (16 at most), two by two.
// One block a round, its up to 17 terms one after the other, was 1-4% faster (1M
// 4.12 ms against 4.17, 100k merger 0.342 and 0.354) and 5-9% less exact in the
// median, 25% at 1M in the largest error; chains of 8 single terms throughout
// cost a second or third block a round: 1M 4.42-4.59 ms.
//
// A large system's task sums the whole tree in one go. A small system's
// (split_max bodies or fewer) closes its sums into double partials: first the
// terms of the root (and of what walk_top walks), then one per child subtree
// of the system's split cell, mostly the root ("segment" k < 8, in child order); the body's acceleration is G times the
// sum of the partials in that order. Its tasks can so be walked by one warp
// (all segments in turn) or by eight (one segment each; unit 0 also takes the
// root's term, and 0 + root is the root exactly; the partials added by
// k_walk_sum) with the same bits; the launch picks by the tasks it has. Which
// sum a system gets depends on its own size only, so that it comes out the
// same alone and in an ensemble.
constexpr int WSEGS = 8;

struct Sum32 : LanePos {
    static constexpr bool BLOCKS = false;
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
    static __device__ __forceinline__ u64 factor(u64 r2, u64 m, bool t0, bool t1)
    {
        const u64 y = pack2(rsq(lo2(r2)), rsq(hi2(r2)));
        const u64 f0 = mul2(m, mul2(y, mul2(y, y)));
        return pack2(t0 ? lo2(f0) : 0.0f, t1 ? hi2(f0) : 0.0f);
    }
    struct Pair {
        u64 dx, dy, dz, f;
    };
    __device__ __forceinline__ void load(const float *rec, int e, Pair &p)
    {
        const ulonglong2 *r = (const ulonglong2 *)(rec + (e >> 1) * RND_REC);
        const ulonglong2 q0 = r[0], q1 = r[1], q2 = r[2], q3 = r[3];
        const uint2 t = *(const uint2 *)(r + 4); // masks
        p.dx = add2(add2(q0.x, nhx), add2(q2.x, nlx));
        p.dy = add2(add2(q0.y, nhy), add2(q2.y, nly));
        p.dz = add2(add2(q1.x, nhz), add2(q3.x, nlz));
        p.f = factor(fma2(p.dx, p.dx, fma2(p.dy, p.dy, fma2(p.dz, p.dz, eps2))), q1.y, t.x & bit,
                     t.y & bit);
    }
    __device__ __forceinline__ void accept(const float *rec, int n)
    {
        int e = 0;
        for (; e + 2 < n; e += 4) {
            Pair p, q;
            load(rec, e, p);
            load(rec, e + 2, q);
            bx = add2(bx, fma2(q.f, q.dx, mul2(p.f, p.dx)));
            by = add2(by, fma2(q.f, q.dy, mul2(p.f, p.dy)));
            bz = add2(bz, fma2(q.f, q.dz, mul2(p.f, p.dz)));
        }
        if (e < n) {
            Pair p;
            load(rec, e, p);
            bx = fma2(p.f, p.dx, bx);
            by = fma2(p.f, p.dy, by);
            bz = fma2(p.f, p.dz, bz);
        }
        fold();
    }
    __device__ __forceinline__ void terms(u64 dx, u64 dy, u64 dz, u64 d2, u64 m, bool t0, bool t1)
    {
        const u64 f = factor(add2(d2, eps2), m, t0, t1);
        bx = fma2(f, dx, bx);
        by = fma2(f, dy, by);
        bz = fma2(f, dz, bz);
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

// One cell, taken or opened lane by lane; returns the lanes that open it.
// count: this warp's takes count (one of a split task's units counts them).
template <bool STATS, class Sink>
__device__ __forceinline__ unsigned walk_cell(const WalkArgs &a, const LaneBody &L, int cell,
                                              unsigned lanes, Sink &sink, WalkStats &st, bool count)
{
    const bool mine = lanes >> (threadIdx.x & 31) & 1u;
    int next;
    bool take, open;
    if (STATS) {
        st.steps++;
        st.active += mine;
    }
    lane_test(a, L, cell, mine, next, take, open, sink);
    if (STATS)
        st.hits += count && take;
    return __ballot_sync(0xffffffffu, open);
}

// A system's cells above its segments: the root, and down to tr.split the cells
// on the way with their other children's subtrees (`mine`: this warp's to walk;
// else only the way is tested). Returns the lanes that open tr.split.
template <bool STATS, class Sink>
__device__ __forceinline__ unsigned walk_top(const WalkArgs &a, RoundShared &sh, const LaneBody &L,
                                             const TaskRange &tr, Sink &sink, WalkStats &st,
                                             bool mine)
{
    int cell = tr.root;
    unsigned open =
        walk_cell<STATS>(a, L, cell, __ballot_sync(0xffffffffu, L.valid), sink, st, mine);
    while (cell != tr.split && open) {
        int down = -1; // the child that holds tr.split (cells are in preorder)
        for (int o = 0; o < 8; o++) {
            const int c = __ldg(&a.child[8 * (size_t)cell + o]);
            if (c > cell && c <= tr.split)
                down = max(down, c);
        }
        if (down < 0) { // not a cell of this tree
            dev_fail(a.sc, CSG_ERR_WALK_LIMIT);
            return 0u;
        }
        for (int o = 0; o < 8 && mine; o++) {
            const int c = __ldg(&a.child[8 * (size_t)cell + o]);
            if (c > cell && c != down)
                walk_subtree<STATS>(a, sh, L, c, open, sink, st);
        }
        open = walk_cell<STATS>(a, L, down, open, sink, st, mine);
        cell = down; // strictly increases: the loop ends
    }
    return open;
}

// The whole task by one warp: a large system's tree from the root; a small
// system's top, then each child subtree of its split cell as a segment, every one closed
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
    int q = -1; // whole: one subtree, the root's; else the split cell's children
    if (tr.small) {
        go = walk_top<STATS>(a, sh.r, L, tr, sum, st, true);
        sum.close(x, y, z);
        q = 0;
    }
    g[0] = x;
    g[CSG_WARP] = y;
    g[2 * CSG_WARP] = z;
    const int qend = tr.small ? (go ? 8 : 0) : 0;
    for (; q < qend; q++) {
        const int c = q < 0 ? tr.root : __ldg(&a.child[8 * (size_t)tr.split + q]);
        if (q >= 0 && c <= tr.split)
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
    const unsigned open = walk_top<false>(a, sh.r, L, tr, sum, st, k == 0);
    double rx, ry, rz, x = 0.0, y = 0.0, z = 0.0;
    sum.close(rx, ry, rz);
    double *g = sh.g + (threadIdx.x & 31);
    g[0] = rx;
    g[CSG_WARP] = ry;
    g[2 * CSG_WARP] = rz;
    const int c = nth_child(a, tr.split, k);
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
    const TaskRange tr{w.pos0, w.count, r.root, r.end, r.split, small_system(a, w.gal)};
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

// Pair terms of the lane's body with queued cells: differences and sums in FP64, m/r^3
// by integers (pair_m_r3). Every system takes them, whatever its extent, masses and
// softening.
struct EvalF64 {
    struct Rec {
        double2 xy, zm;
    };
    const NodeW64 *cells;
    const PairEps eps;
    double px, py, pz;
    double s[3]; // without G

    __device__ __forceinline__ EvalF64(const WalkArgs &a, int me)
        : cells(a.w64), eps(a.eps), px(me >= 0 ? a.x[me] : 0.0), py(me >= 0 ? a.y[me] : 0.0),
          pz(me >= 0 ? a.z[me] : 0.0)
    {
        s[0] = s[1] = s[2] = 0.0;
    }
    __device__ __forceinline__ Rec load(int c) const
    {
        const double2 *w = (const double2 *)&cells[c];
        return Rec{__ldg(w), __ldg(w + 1)};
    }
    __device__ __forceinline__ void term(const Rec &r)
    {
        const double dx = r.xy.x - px, dy = r.xy.y - py, dz = r.zm.x - pz;
        const double f = pair_m_r3(eps, dx, dy, dz, r.zm.y);
        s[0] = fma(f, dx, s[0]);
        s[1] = fma(f, dy, s[1]);
        s[2] = fma(f, dz, s[2]);
    }
    static __device__ __forceinline__ void drop(Rec &r) { r.zm.y = 0.0; }
    // the other consumer's sums of the same body (3 doubles a lane)
    __device__ __forceinline__ void save(double *o) const
    {
#pragma unroll
        for (int d = 0; d < 3; d++)
            o[d * CSG_WARP] = s[d];
    }
    __device__ __forceinline__ void join(const double *o)
    {
#pragma unroll
        for (int d = 0; d < 3; d++)
            s[d] += o[d * CSG_WARP];
    }
};

// A unit's segment partials: part[(3 * k + d) * pstride + body].
__device__ __forceinline__ void put_partial(const WalkArgs &a, int k, int me, double sx, double sy,
                                            double sz)
{
    a.part[(3 * k + 0) * a.pstride + me] = sx;
    a.part[(3 * k + 1) * a.pstride + me] = sy;
    a.part[(3 * k + 2) * a.pstride + me] = sz;
}

// FP64 walk, producer/consumer form. A task's producer warp walks the tree (in
// rounds, the FP32 decisions) and queues every round's cells as a block in
// shared memory, 32 cell ids and, per lane, the word of the cells that lane
// takes; its consumer warps evaluate every lane's cells, each lane reading on
// in the blocks at its own pace. The warps hand over through head and tail
// block counters in shared memory; every wait polls with a sleep and gives up
// after a.wait_polls polls (recording CSG_ERR_DEVICE_WAIT, then all warps leave
// the task). A unit of the split form is one segment of a task: the subtree of
// the split cell's child k0 (segment 0: also the cells above the segments).
//
// Bound: the FP64 pipe, 6 operations a pair (79% busy in the 100k merger, issue 55%).
// Measured, walk inside the substep: r^2 in FP64 too (9 operations), a ring of ids
// per lane and one consumer -> now: 1M 39.0 -> 25.7 ms, 100k merger 2.23 -> 1.41
// ms, 20k disk 0.496 -> 0.34 ms. With blocks and two consumers but 9 operations 42, 2.0
// and 0.49 ms. With positions and sums in fixed point, no FP64 operation at all, 24.9,
// 1.36 and 0.36 ms; a grid of 2^-61 of a system's extent and 96-bit sums lost the
// bits of close pairs near the origin (up to 6e-11 of the acceleration at 1e-4 softenings)
// and of a heavy body among light ones.
//
// Blocks rather than a ring of ids per lane: an id costs 4 bytes a block, not
// 4 bytes a lane that takes it, so the same memory holds several times the
// lead, and lanes that take fewer of the current cells run dry less often. The
// takes of a round reach the lanes by one bit transpose instead of a store per
// cell and lane.
constexpr int WS_BLOCKS = 32; // queue length (power of two; 16: 6% slower at 1M)
constexpr int WS_RES = 21;    // resident warps per SM that the registers are sized for (18 and
                              // 24: 2-6% slower)
constexpr int WS_CONS = 2;    // consumer warps
constexpr int WS_LOW = 2;     // blocks the slowest reader wants ahead before a step

struct WsShared {
    int ids[WS_BLOCKS * CSG_WARP];
    unsigned take[WS_BLOCKS * CSG_WARP];
    int tail;            // blocks published by the producer
    int head[2];         // each consumer's first block that some lane still reads
    int done;            // producer finished (tail final)
    int half;            // the second consumer's sums are in `other`
    int broken;          // a wait gave up: all warps leave
    double other[3 * CSG_WARP];
};

__device__ __forceinline__ int ws_load(const volatile int *p) { return *p; }

// The producer's sink.
struct BlockQueue : LanePos {
    static constexpr bool BLOCKS = true;
    WsShared &sh;
    DevScalars *sc;
    int wait_polls;
    int tail, head_seen;
    bool mute, broken;

    __device__ __forceinline__ BlockQueue(const WalkArgs &a, const LaneBody &L, WsShared &s)
        : LanePos(L), sh(s), sc(a.sc), wait_polls(a.wait_polls), tail(0), head_seen(0),
          mute(false), broken(false)
    {
    }
    // waits until a block is free
    __device__ __forceinline__ void room()
    {
        if (tail - head_seen < WS_BLOCKS || broken)
            return;
        for (int i = 0; i < wait_polls; i++) {
            head_seen = min(ws_load(&sh.head[0]), ws_load(&sh.head[1]));
            if (tail - head_seen < WS_BLOCKS || ws_load(&sh.broken))
                break;
            __nanosleep(64);
        }
        head_seen = __shfl_sync(0xffffffffu, head_seen, 0);
        __threadfence_block(); // the head read before its blocks are overwritten
        if (tail - head_seen >= WS_BLOCKS) { // gave up (or the consumer did)
            if ((threadIdx.x & 31) == 0) {
                dev_fail(sc, CSG_ERR_DEVICE_WAIT);
                ((volatile int *)&sh.broken)[0] = 1;
            }
            broken = true;
        }
    }
    __device__ __forceinline__ void block(int cell, unsigned take)
    {
        if (mute || !__any_sync(0xffffffffu, take != 0u))
            return;
        room();
        if (broken)
            return;
        const int lane = threadIdx.x & 31, b = tail & (WS_BLOCKS - 1);
        sh.ids[b * CSG_WARP + lane] = cell;
        sh.take[b * CSG_WARP + lane] = take;
        tail++;
        __threadfence_block(); // the block before the tail
        __syncwarp();
        if (lane == 0)
            ((volatile int *)&sh.tail)[0] = tail;
    }
};

template <bool STATS, bool UNITS>
__device__ __forceinline__ void ws_produce(const WalkArgs &a, RoundShared &rs, WsShared &sh,
                                           const TaskRange &tr, int k0, WalkStats &st)
{
    const LaneBody L = lane_body(a, rs, tr);
    BlockQueue q(a, L, sh);
    q.mute = UNITS && k0 != 0; // the terms above the segments are segment 0's
    const unsigned open = walk_top<STATS>(a, rs, L, tr, q, st, !q.mute);
    q.mute = false;
    int k = 0; // child (segment) number
    for (int o = 0; o < 8 && open; o++) {
        const int c = __ldg(&a.child[8 * (size_t)tr.split + o]);
        if (c <= tr.split)
            continue;
        if (!UNITS || k == k0)
            walk_subtree<STATS>(a, rs, L, c, open, q, st);
        k++;
    }
    __threadfence_block();
    __syncwarp();
    if ((threadIdx.x & 31) == 0)
        ((volatile int *)&sh.done)[0] = 1; // after the final tail
}

// A lane's place in the queue: the cells left of its current block, and the
// next block.
struct WsReader {
    unsigned left;
    int cur, next;
};

// The lane's next cell, or -1 (none published, or the next block has none for
// it).
__device__ __forceinline__ int ws_next(const WsShared &sh, WsReader &r, int tail, int lane)
{
    if (r.left == 0u && r.next < tail) {
        r.cur = r.next & (WS_BLOCKS - 1);
        r.left = sh.take[r.cur * CSG_WARP + lane];
        r.next += WS_CONS;
    }
    if (r.left == 0u)
        return -1;
    const int j = __ffs((int)r.left) - 1;
    r.left &= r.left - 1u;
    return sh.ids[r.cur * CSG_WARP + j];
}

// Cells a lane evaluates between two looks at the counters: whole tasks (16: 1-3%
// faster than 8 from 100k bodies on), a split task's units (8: 7% faster at 20k).
constexpr int WS_STEP_TASK = 16, WS_STEP_UNIT = 8;

// Consumer `which`: the blocks which, which + 2, ...
template <bool UNITS>
__device__ __forceinline__ void ws_consume(const WalkArgs &a, WsShared &sh, const TaskRange &tr,
                                           int k0, int which)
{
    const int lane = threadIdx.x & 31;
    const bool valid = lane < tr.count;
    const int me = valid ? a.perm[tr.pos0 + lane] : -1;
    EvalF64 ev(a, me);
    WsReader rd{0u, 0, which};
    int polls = 0, head = which;
    // two cells are always on their way: their loads run during the terms of
    // the two before them (massless ones at first; no cell to read: the root)
    EvalF64::Rec ra = ev.load(tr.root), rb = ra;
    ev.drop(ra);
    ev.drop(rb);
    while (true) {
        // read before the tail: it is final then
        const bool done = __shfl_sync(0xffffffffu, ws_load(&sh.done), 0) != 0;
        __threadfence_block();
        const int tail = __shfl_sync(0xffffffffu, ws_load(&sh.tail), 0);
        __threadfence_block(); // the tail before the blocks it covers
        __syncwarp();
        // blocks that the furthest lane still has ahead
        const int ahead =
            tail - (int)__reduce_max_sync(0xffffffffu, (unsigned)(valid ? rd.next : 0));
        if (ahead >= WS_LOW || tail - head >= WS_BLOCKS || (done && head < tail)) {
            auto fetch = [&](EvalF64::Rec &r) {
                const int c = ws_next(sh, rd, tail, lane);
                r = ev.load(c < 0 ? tr.root : c);
                if (c < 0)
                    ev.drop(r);
            };
#pragma unroll 1
            for (int s = 0; s < (UNITS ? WS_STEP_UNIT : WS_STEP_TASK); s += 2) {
                EvalF64::Rec rc, rq;
                fetch(rc);
                fetch(rq);
                ev.term(ra);
                ev.term(rb);
                ra = rc;
                rb = rq;
            }
            // blocks that every lane is through with
            const int h = (int)__reduce_min_sync(
                0xffffffffu, (unsigned)(!valid ? tail + WS_CONS : rd.left ? rd.next - WS_CONS : rd.next));
            __threadfence_block(); // blocks read before the head is published
            __syncwarp();
            if (h != head && lane == 0)
                ((volatile int *)sh.head)[which] = h;
            head = h;
            polls = 0;
            continue;
        }
        if (done) { // head == tail: every block read
            ev.term(ra);
            ev.term(rb);
            break;
        }
        if (__any_sync(0xffffffffu, ws_load(&sh.broken)))
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
    // the second consumer's sums joined to the first's
    if (which == 1) {
        ev.save(sh.other + lane);
        __threadfence_block();
        __syncwarp();
        if (lane == 0)
            ((volatile int *)&sh.half)[0] = 1;
        return;
    }
    for (int i = 0; !__any_sync(0xffffffffu, ws_load(&sh.half)); i++) {
        if (i >= a.wait_polls || __any_sync(0xffffffffu, ws_load(&sh.broken))) {
            if (lane == 0) {
                dev_fail(a.sc, CSG_ERR_DEVICE_WAIT);
                ((volatile int *)&sh.broken)[0] = 1;
            }
            return;
        }
        __nanosleep(64);
    }
    __threadfence_block();
    __syncwarp();
    ev.join(sh.other + lane);
    if (!valid)
        return;
    if (UNITS) { // the segment's partial (zero for one that the walk did not reach)
        put_partial(a, k0, me, ev.s[0], ev.s[1], ev.s[2]);
    } else {
        a.ax[me] = a.G * ev.s[0];
        a.ay[me] = a.G * ev.s[1];
        a.az[me] = a.G * ev.s[2];
    }
}

// One task per block, or (UNITS) one segment of a task, u = 8 task + segment
// (partials into a.part): the producer warp, then the consumers. The producer needs about a
// fifth of a consumer's time. Units of several segments of a task, for fewer root steps,
// needed the segments' ends in the queue and so had one consumer: 30,000 bodies 0.79 ms
// against 0.51, 64 systems of 2,000 to 50,000 18.0 against 12.9.
template <bool STATS, bool UNITS>
__device__ __forceinline__ void walk64ws_body(const WalkArgs &a)
{
    __shared__ WsShared sh;
    __shared__ RoundShared rs;
    const int warp = threadIdx.x >> 5;
    const int nn = a.sc->n_nodes;
    if (nn > a.node_cap || nn < 1)
        return;
    const int u = blockIdx.x;
    const int t = UNITS ? u / WSEGS : u, k0 = UNITS ? u % WSEGS : 0;
    if (t >= a.sc->n_tasks)
        return;
    const WalkTask w = a.tasks[t];
    const DevRoot &r = a.roots[w.gal];
    const TaskRange tr{w.pos0, w.count, r.root, r.end, r.split, small_system(a, w.gal)};
    if (UNITS ? !tr.small : (tr.small && a.skip_small))
        return; // the other form walks this system
    if (tr.root < 0 || tr.end > nn || tr.root >= tr.end) {
        if (threadIdx.x == 0)
            dev_fail(a.sc, CSG_ERR_WALK_LIMIT);
        return;
    }
    if (threadIdx.x == 0) {
        sh.tail = 0;
        sh.head[0] = 0;
        sh.head[1] = 1;
        sh.done = 0;
        sh.half = 0;
        sh.broken = 0;
    }
    __syncthreads(); // counters set before any warp starts (the returns above are the block's)
    if (warp == 0) {
        WalkStats st;
        ws_produce<STATS, UNITS>(a, rs, sh, tr, k0, st);
        if (STATS)
            add_hits(a, st);
    } else {
        ws_consume<UNITS>(a, sh, tr, k0, warp - 1);
    }
}

template <bool STATS>
__global__ void __launch_bounds__((1 + WS_CONS) * CSG_WARP, WS_RES / (1 + WS_CONS))
    k_walk64ws(WalkArgs a)
{
    walk64ws_body<STATS, false>(a);
}

// The FP64 walk split by the split cell's children (few tasks for the GPU): partials
// into a.part, summed by k_walk_sum.
template <bool STATS>
__global__ void __launch_bounds__((1 + WS_CONS) * CSG_WARP, WS_RES / (1 + WS_CONS))
    k_walk64ws_units(WalkArgs a)
{
    walk64ws_body<STATS, true>(a);
}

// Before a walk: dead bodies get a = 0 (src/octree.c:226-230; alive ones are
// overwritten by the walk), and the task counter of the persistent walks is
// rewound.
__global__ void k_walk_prep(const double *__restrict__ m, double *ax, double *ay, double *az, int n,
                            DevScalars *sc)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i == 0)
        sc->task_next = 0;
    if (i < n && m[i] <= 0.0) {
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
    static constexpr bool BLOCKS = true;
    int *ids;
    int k, lim;
    bool mute;

    __device__ __forceinline__ ListSink(const LaneBody &L)
        : LanePos(L), ids(nullptr), k(0), lim(0), mute(false)
    {
    }
    __device__ __forceinline__ void block(int cell, unsigned take)
    {
        if (mute)
            return;
        if (!FILL) {
            k += __popc(take);
            return;
        }
        while (__any_sync(0xffffffffu, take != 0u)) { // each lane its own cells, one a step
            const int c = __shfl_sync(0xffffffffu, cell, __ffs((int)take) - 1);
            if (take != 0u && k < lim)
                ids[k] = c;
            k += take != 0u;
            take &= take - 1u;
        }
    }
};

//
// With segs = WSEGS a warp takes one segment of a task (the root's and then
// the split cell's child subtrees, as the sums of a small system), and a body's
// list is its segments' lists in turn: entry segs i + k of counts and offs is
// body i's segment k. 10,000 bodies are 313 tasks, two warps an SM; split eight
// ways counting takes 64 and filling 90 us instead of 88 and 154.
template <bool FILL, int WARPS>
__global__ void __launch_bounds__(WARPS * CSG_WARP) k_walk_lists(WalkArgs a, int segs, int *counts,
                                                             const int *offs, int *ids, int cap)
{
    __shared__ RoundShared rs_all[WARPS];
    RoundShared &rs = rs_all[threadIdx.x >> 5];
    const int nn = a.sc->n_nodes;
    if (nn > a.node_cap || nn < 1)
        return;
    const int u = blockIdx.x * WARPS + (threadIdx.x >> 5), t = u / segs, k = u % segs;
    if (t >= a.sc->n_tasks)
        return;
    const WalkTask w = a.tasks[t];
    const DevRoot &r = a.roots[w.gal];
    const TaskRange tr{w.pos0, w.count, r.root, r.end, r.split, false};
    if (tr.root < 0 || tr.end > nn || tr.root >= tr.end) {
        dev_fail(a.sc, CSG_ERR_WALK_LIMIT);
        return;
    }
    const LaneBody L = lane_body(a, rs, tr);
    ListSink<FILL> q(L);
    const size_t slot = (size_t)segs * (size_t)max(L.me, 0) + k;
    if (FILL && L.valid) {
        const int base = offs[slot];
        q.ids = ids + base;
        q.lim = min(counts[slot], cap - base);
    }
    WalkStats st;
    if (segs == 1) {
        walk_subtree<false>(a, rs, L, tr.root, __ballot_sync(0xffffffffu, L.valid), q, st);
    } else {
        q.mute = k != 0; // the cells above the segments are segment 0's
        const unsigned open = walk_top<false>(a, rs, L, tr, q, st, k == 0);
        q.mute = false;
        const int c = nth_child(a, tr.split, k);
        if (open && c >= 0)
            walk_subtree<false>(a, rs, L, c, open, q, st);
    }
    if (!FILL && L.valid)
        counts[slot] = q.k;
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
    a.eps = pair_eps(p->softening);
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
    a.split_max = (int)csgd_split_max_bodies(d, p->precision, p->theta);
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
void launch_walk(csgd_t *d, const WalkArgs &a, int precision, double theta, int exact)
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
    } else if (precision == CSG_PREC_FP32_MIXED && !stats && csgd_walk_split(d, theta) &&
               d->wpart && d->wpart_cap >= d->n) {
        // small systems, few tasks: eight warps per task, one per child subtree,
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
    } else { // FP64: producer and consumer warps (the task group applies to FP32 only)
        // small systems (split_max bodies or fewer): a block per (task,
        // segment), partials added by k_walk_sum; the rest a block per task
        const bool units = d->wpart && d->wpart_cap >= d->n &&
                           csgd_sys_min_n(d) <= b.split_max;
        b.skip_small = units;
        if (units) {
            const int gw = (int)(((long long)d->n / CSG_WARP + d->n_gal + 1) * WSEGS);
            b.part = d->wpart;
            b.pstride = d->wpart_cap;
            if (stats)
                k_walk64ws_units<true><<<gw, (1 + WS_CONS) * CSG_WARP, 0, s>>>(b);
            else
                k_walk64ws_units<false><<<gw, (1 + WS_CONS) * CSG_WARP, 0, s>>>(b);
            k_walk_sum<<<csgd_grid(d->n, 256), 256, 0, s>>>(d->wpart, (long long)d->wpart_cap,
                                                              d->m, d->n, b.G, d->ax, d->ay, d->az,
                                                              d->gid, b.sys_n, b.split_max);
            d->launches += 2;
            if (csgd_sys_max_n(d) <= b.split_max)
                return; // every system is small
        }
        const long long tasks = (long long)d->n / CSG_WARP + d->n_gal + 1; // >= n_tasks
        if (stats)
            k_walk64ws<true><<<(int)tasks, (1 + WS_CONS) * CSG_WARP, 0, s>>>(b);
        else
            k_walk64ws<false><<<(int)tasks, (1 + WS_CONS) * CSG_WARP, 0, s>>>(b);
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
    k_walk_prep<<<csgd_grid(n, 256), 256, 0, s>>>(d->m, d->ax, d->ay, d->az, n, d->sc);
    d->launches++;
    if (exact) {
        const int saved = d->walk_warps;
        d->walk_warps = 8;
        launch_walk(d, a, p->precision, p->theta, 1);
        d->walk_warps = saved;
    } else {
        launch_walk(d, a, p->precision, p->theta, 0);
    }
    return csgd_check(d, cudaGetLastError());
}

extern "C" int csgd_gravity(csgd_t *d, const csgd_force_params *p)
{
    return csgd_gravity_ex(d, p, 0);
}

extern "C" int csgd_list_segments(const csgd_t *d, int n)
{
    const long long tasks = (long long)n / CSG_WARP + d->n_gal + 1;
    return tasks < 8LL * d->num_sms ? WSEGS : 1; // a task a warp: fewer than 8 warps an SM
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
    const int segs = csgd_list_segments(d, n);
    const long long tasks = (long long)n / CSG_WARP + d->n_gal + 1;
    const int grid = (int)((tasks * segs + 3) / 4);
    if (fill)
        { k_walk_lists<true, 4><<<grid, 4 * CSG_WARP, 0, d->stream>>>(a, segs, counts, offs, ids, cap); d->launches++; }
    else
        { k_walk_lists<false, 4><<<grid, 4 * CSG_WARP, 0, d->stream>>>(a, segs, counts, offs, ids, cap); d->launches++; }
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
    // persistent candidates: 8, 16 or as many resident warps per SM as their
    // registers are sized for (in whole blocks: 16 with eight warps a block), task
    // groups of 1, 2 or 4
    static const int groups[] = {1, 2, 4};
    static const int resident[] = {8, 16, WALK32_RES};
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
