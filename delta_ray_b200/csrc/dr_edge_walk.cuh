// The edge-tree walks of the shading points, a warp walking the trees of one
// batch of points with its pending nodes in shared memory.  Included by
// dr_edge_kernels.cu.
//
// What bounds it: instruction fetch and latency.  A node decision is 300 to 450
// instructions per child, most of them the BSDF bound's; at the 160x120
// heightfield below issue slots are 55 % busy with 37 % of the warps resident
// (shared memory holds them to 7 blocks per SM), 22.3 of 32 lanes active, and
// warps wait for instructions first (4.4 cycles per issue, then 2.3 for fixed
// latencies).  Two lanes share a node, one per child, so that a lane evaluates
// one bound, reads its child with two 16-byte loads next to its partner's, and
// exchanges importances and tests with one shuffle each: 16 nodes a step.  The
// nodes come off stacks by class, so that the lanes of a step run one path: the
// nodes that split the all walk (three in four of a glossy heightfield's) need no
// draw, no cone tests and only a bound's sides of 0 and 1.  The points' contexts,
// the stacks, the reached leaves and the sampled edges stay in shared memory: a
// node costs no global traffic but its own record, and the items leave in runs of
// consecutive slots, each point's together (the line and ray kernels then read
// one point's data and neighbouring edges from a warp's lanes).
//
// Measured against the walk it replaced (one level of every point's nodes
// per launch, nodes queued in global memory between levels, the point's
// 176-byte context read per node), level and leaf kernels against this one:
// the 130,054-triangle heightfield at 640x480, 1 spp (1.16 G nodes): 254 ->
// 65 ms, at 160x120 (72 M): 22.6 -> 4.6; a 64x64-vertex heightfield at
// 128x96, 8 spp (53 M): 7.9 -> 5.4; a room of smooth spheres (28 M nodes, 90
// per point): 6.0 -> 5.3.  22.3 of 32 lanes are active (10 before).  Without
// the rounds the first took 184 ms and the second 20.7 (its few longest walks
// ran alone); with one step for every node that splits or draws 83 and 5.9.
#pragma once

#include "dr_walk_rules.cuh"

#define DR_WALK_POINTS 4  // points of a batch, at most
#define DR_WALK_ITEMS 128
#ifndef DR_WALK_BLOCKS
#define DR_WALK_BLOCKS 7
#endif
// Steps a warp walks a batch before it hands its pending nodes on, and the
// fewest pending nodes worth handing on.
#ifndef DR_WALK_STEPS
#define DR_WALK_STEPS 64
#endif
#define DR_WALK_HAND 32

// Pending nodes handed on to the next round (k_edge_walk): up to 32 nodes of
// up to DR_WALK_POINTS points (code, apmf, cpmf, lpmf; the code's slot indexes
// `point`).
struct __align__(16) WalkPacket {
    int count, np;
    int point[DR_WALK_POINTS];
    int pad[2];
    uint4 e[32];
};
static_assert(sizeof(WalkPacket) == DR_WALK_PACKET_BYTES, "packet size as the workspace allocates it");

// Words of a point's walk context (k_walk_ctx; BackwardWorkspace::walk_ctx):
// 0 p, 3 n, 6 dl, 7 sl, 8 the frame around wi, 17 the normal in it, 20 the
// lobe's exponent, 21 flags, 22 the light cone's cosine, 23 its axis, 26 the
// picked tree's probability, 27 sample id, 30 seed; 32 the shading frame (the
// proposal's direction bins).  Flags: 1 the point walks a tree, 2 the normal
// tree, 4 its root splits the all walk, 8 the learned descent, model << 4,
// 128 the root is a leaf, bounce << 8.
struct WalkCtx {
    const float *w;
    __device__ __forceinline__ float3 v(int i) const { return f3(w[i], w[i + 1], w[i + 2]); }
    __device__ __forceinline__ float3 p() const { return v(0); }
    __device__ __forceinline__ int flags() const { return __float_as_int(w[21]); }
    __device__ __forceinline__ int tree() const { return (flags() >> 1) & 1; }
    __device__ __forceinline__ BoundCtx bound() const {
        BoundCtx b;
        b.p = v(0);
        b.n = v(3);
        b.dl = w[6];
        b.sl = w[7];
        b.hf.t = v(8);
        b.hf.b = v(11);
        b.hf.n = v(14);
        b.ln = v(17);
        b.rough = 0.f;
        b.expo = w[20];
        b.model = (flags() >> 4) & 7;
        return b;
    }
    __device__ __forceinline__ ConeSpec cone() const {
        ConeSpec c;
        c.o = v(0);
        c.d = v(23);
        c.cos_angle = w[22];
        return c;
    }
    __device__ __forceinline__ NodeRng rng() const {
        NodeRng r;
        r.seed = (uint64_t)__float_as_uint(w[30]) | ((uint64_t)__float_as_uint(w[31]) << 32);
        r.sid = (uint64_t)__float_as_uint(w[27]) | ((uint64_t)__float_as_uint(w[28]) << 32);
        r.bounce = (uint32_t)flags() >> 8;
        return r;
    }
    __device__ __forceinline__ Frame frame() const {
        Frame f;
        f.t = v(32);
        f.b = v(35);
        f.n = v(38);
        return f;
    }
};

// The exact bound of a box, out of line: the walk's loop must stay within the
// instruction cache (with this and the silhouette test's exact part inlined
// where they are needed the fast step ran no faster than the general one,
// waiting on instruction fetches for half of its cycles).
static __device__ __noinline__ float walk_bound(float3 lo, float3 hi, const float *ctx) {
    return bsdf_bound_box(lo, hi, WalkCtx{ctx}.bound(), nullptr);
}

// One warp's shared memory.  A pending node's code: node id, the point's slot
// in the batch << 27, mode << 30, all-split << 31.
template <bool PROP> struct WalkWarp {
    static constexpr int kCtx = PROP ? 44 : 32;  // words of a context
    float4 ctx[DR_WALK_POINTS][kCtx / 4 + 1];    // one float4 of padding: slots start in different banks
    uint2 st[DR_WALK_N0 + DR_WALK_N1 + DR_WALK_N2];  // pending nodes, class after class: code, apmf
    float c[DR_WALK_N0 + DR_WALK_N2];                // cpmf of classes 0 and 2 (class 1's is 0)
    float l[PROP ? DR_WALK_N0 + DR_WALK_N1 + DR_WALK_N2 : 1];  // lpmf
    uint2 leaf[64];        // edge or node | slot << 27 | mode << 30 | many << 31, weight
    uint2 item[DR_WALK_ITEMS];  // edge | slot << 27 | mode << 30, weight
    uint8_t item_code[PROP ? DR_WALK_ITEMS : 1];
    int cnt[DR_WALK_POINTS], point[DR_WALK_POINTS];  // edges sampled per point; the batch's points
};

// Round 0 (in == null) takes batches of points; a later round takes the
// packets round - 1 handed on.  Points' walks are heavy-tailed (a glossy point
// whose bounds stay above 1 splits at every node: hundreds of thousands of
// nodes, a hundred times the mean), so a warp that has walked a batch for
// DR_WALK_STEPS steps hands what is pending to the next round (`out`), whose
// warps spread it; the last round (out == null) walks to the end.

template <bool PROP>
__global__ void __launch_bounds__(128, DR_WALK_BLOCKS) k_edge_walk(const __grid_constant__ DevScene s, BackwardWorkspace ws, int round,
                                                                 const WalkPacket *in, WalkPacket *out) {
    __shared__ WalkWarp<PROP> block_sh[4];
    WalkWarp<PROP> &sh = block_sh[threadIdx.x >> 5];
    const unsigned full = 0xffffffffu;
    const int lane = threadIdx.x & 31;
    const unsigned below = (1u << lane) - 1u;
    const long long m =
        in ? (long long)min(ws.counters->walk_n[round - 1], (unsigned long long)ws.cap_packets) : strided_points(ws);
    // points per batch: one where points are few for the warps there are (a
    // point's walk is the unit that keeps them all busy to the end), up to 4
    // where they are many (their walks fill each other's underfull steps)
    const long long per = m / (4ll * gridDim.x * (blockDim.x >> 5));
    const int batch = in || per < 1 ? 1 : (per < DR_WALK_POINTS ? (int)per : DR_WALK_POINTS);
    unsigned long long visits = 0, walked = 0;  // warp-uniform
    while (true) {
        long long k0 = 0;
        if (lane == 0) k0 = (long long)atomicAdd(&ws.counters->walk_next[round], (unsigned long long)batch);
        k0 = __shfl_sync(full, k0, 0);
        if (k0 >= m) break;
        const WalkPacket *pk = in ? in + k0 : nullptr;
        const int nb = in ? pk->np : (int)min((long long)batch, m - k0);
        if (lane < nb) sh.point[lane] = in ? pk->point[lane] : (int)(ws.pt_begin + (k0 + lane) * ws.pt_stride);
        __syncwarp();
        const auto point_of = [&](int slot) { return sh.point[slot]; };
        for (int b = 0; b < nb; b++) {
            const float *g = reinterpret_cast<const float *>(ws.walk_ctx + (size_t)point_of(b) * DR_CTX_F4);
            float *d = reinterpret_cast<float *>(sh.ctx[b]);
            d[lane] = g[lane];
            if (PROP && lane < 12) d[32 + lane] = g[32 + lane];
        }
        if (lane < DR_WALK_POINTS) sh.cnt[lane] = 0;
        __syncwarp();
        const auto ctx_of = [&](int slot) { return WalkCtx{reinterpret_cast<const float *>(sh.ctx[slot])}; };
        int n0 = 0, n1 = 0, n2 = 0, nl = 0, ni = 0;  // pending nodes by class, leaves, items
        bool two = out != nullptr;                   // nodes may go to class 2
        // a node to its class's stack, every lane's at once
        const int b1 = DR_WALK_N0, b2 = DR_WALK_N0 + DR_WALK_N1;  // where classes 1 and 2 begin
        const auto push_nodes = [&](bool node, unsigned code, float cp, float ap, float lp) {
            const int cls = walk_class(code, cp, two);
            const bool to0 = node && cls == 0, to1 = node && cls == 1, to2 = node && cls == 2;
            const unsigned m0 = __ballot_sync(full, to0), m1 = __ballot_sync(full, to1), m2 = __ballot_sync(full, to2);
            if (node) {
                const int at = to0 ? n0 + __popc(m0 & below)
                                   : (to2 ? b2 + n2 + __popc(m2 & below) : b1 + n1 + __popc(m1 & below));
                sh.st[at] = make_uint2(code, __float_as_uint(ap));
                if (to0) sh.c[at] = cp;
                else if (to2) sh.c[at - DR_WALK_N1] = cp;
                if constexpr (PROP) sh.l[at] = lp;
            }
            n0 += __popc(m0);
            n1 += __popc(m1);
            n2 += __popc(m2);
        };
        // the cone-walk share of the pending node at `at`
        const auto share_at = [&](int at) { return at < b1 ? sh.c[at] : (at >= b2 ? sh.c[at - DR_WALK_N1] : 0.f); };
        if (in) {  // the handed-on nodes
            const bool have = lane < pk->count;
            uint4 e = make_uint4(0, 0, 0, 0);
            if (have) e = pk->e[lane];
            push_nodes(have, e.x, __uint_as_float(e.z), __uint_as_float(e.y), __uint_as_float(e.w));
            __syncwarp();
        } else {  // both walks of every point start at the root of its tree
            bool valid = false, leaf = false;
            unsigned code = 0;
            float pmf = 0.f;
            if (lane < nb) {
                const WalkCtx c = ctx_of(lane);
                valid = c.flags() & 1;
                leaf = valid && (c.flags() & 128);
                code = ((unsigned)lane << 27) | ((c.flags() & 4) ? 1u << 31 : 0u);
                pmf = c.w[26];
            }
            const unsigned mask = __ballot_sync(full, valid && !leaf), ml = __ballot_sync(full, leaf);
            if (valid && !leaf) {
                const int at = 2 * __popc(mask & below);
                sh.st[at] = make_uint2(code, __float_as_uint(pmf));
                sh.st[at + 1] = make_uint2(code | (1u << 30), __float_as_uint(pmf));
                sh.c[at] = sh.c[at + 1] = pmf;
                if constexpr (PROP) sh.l[at] = sh.l[at + 1] = pmf;
            } else if (leaf) {  // a tree of one node: both walks reach it
                float a = pmf;
                if constexpr (PROP) a = ws.proposal_alpha * pmf + (1.f - ws.proposal_alpha) * pmf;
                const float denom = pmf * pmf + a * a;
                const int at = 2 * __popc(ml & below);
                const unsigned many = ((unsigned)lane << 27) | (1u << 31);  // node 0
                sh.leaf[at] = make_uint2(many, __float_as_uint(pmf / denom));
                sh.leaf[at + 1] = make_uint2(many | (1u << 30), __float_as_uint(a / denom));
            }
            n0 = 2 * __popc(mask);
            nl = 2 * __popc(ml);
            walked += n0 + nl;
            visits += nl;
            __syncwarp();
        }
        // the buffered items to the queue: one reservation, consecutive slots
        const auto flush = [&]() {
            __syncwarp();
            unsigned long long first = 0;
            if (lane == 0) first = atomicAdd(&ws.counters->items, (unsigned long long)ni);
            first = __shfl_sync(full, first, 0);
            const unsigned long long cap = (unsigned long long)ws.cap_items;
            if (lane == 0 && first + (unsigned long long)ni > cap)
                set_status(&ws.counters->status, DR_STATUS_ITEM_OVERFLOW);
            for (int i = lane; i < ni; i += 32) {
                const unsigned long long at = first + (unsigned long long)i;
                if (at >= cap) break;
                const uint2 e = sh.item[i];
                const int slot = (e.x >> 27) & 7, ei = (int)(e.x & DR_NODE_MASK), mode = (e.x >> 30) & 1;
                ws.items[at] = make_int4(point_of(slot), (ctx_of(slot).tree() << 30) | ei, (mode << 27) | ei,
                                         PROP ? sh.item_code[i] : 0);
                ws.item_w[at] = __uint_as_float(e.y);
            }
            __syncwarp();
            ni = 0;
        };
        // the top `count` leaves: their silhouette edges become items, one
        // edge of every lane's leaf at a time
        const auto leaves = [&](int count) {
            int off = 0, np = 0, slot = 0;
            unsigned tag = 0, w = 0;
            const EdgeRec *recs = nullptr;
            float3 p = f3(0.f);
            if (lane < count) {
                const uint2 l = sh.leaf[nl - count + lane];
                slot = (l.x >> 27) & 7;
                tag = l.x & (15u << 27);
                w = l.y;
                const WalkCtx c = ctx_of(slot);
                p = c.p();
                recs = c.tree() ? s.nrm_rec : s.sil_rec;
                off = (int)(l.x & DR_NODE_MASK);
                np = 1;
                if (l.x >> 31) {  // several edges: the range is the node's
                    const DevEdgeNode &node = (c.tree() ? s.nrm_nodes : s.sil_nodes)[off];
                    off = node.offset;
                    np = node.nprims;
                }
            }
            nl -= count;
            const int most = (int)__reduce_max_sync(full, (unsigned)np);
            for (int k = 0; k < most; k++) {
                const int ei = off + k;
                const bool e = k < np && is_silhouette_rec(recs + ei, p);
                const unsigned mask = __ballot_sync(full, e);
                if (e) {
                    const int at = ni + __popc(mask & below);
                    sh.item[at] = make_uint2(tag | (unsigned)ei, w);
                    if constexpr (PROP) {
                        int code = 0;
                        if (ws.train_targets) {
                            const WalkCtx c = ctx_of(slot);
                            const DevEdge &edge = (c.tree() ? s.nrm_edges : s.sil_edges)[ei];
                            code = dir_bin(c.frame(), 0.5f * (edge_v0(s, edge) + edge_v1(s, edge)) - p);
                        }
                        sh.item_code[at] = (uint8_t)code;
                    }
                    if (nb > 1) atomicAdd(&sh.cnt[slot], 1);
                }
                if (nb == 1 && lane == 0) sh.cnt[0] += __popc(mask);
                ni += __popc(mask);
                if (ni > DR_WALK_ITEMS - 32) flush();
            }
        };
        for (int steps = 0; n0 + n1 + n2 > 0; steps++) {
            if (two && (!walk_room(n0, n1, n2) || (steps >= DR_WALK_STEPS && n0 + n1 + n2 >= DR_WALK_HAND))) {
                // the pending nodes to the next round: packet q of np takes
                // every np-th, so that large and small subtrees spread
                const int n = n0 + n1 + n2, np = (n + 31) >> 5;
                unsigned long long first = 0;
                if (lane == 0) first = atomicAdd(&ws.counters->walk_n[round], (unsigned long long)np);
                first = __shfl_sync(full, first, 0);
                const bool fits = first + (unsigned long long)np <= (unsigned long long)ws.cap_packets;
                for (int q = 0; q < np; q++) {
                    if (first + (unsigned long long)q >= (unsigned long long)ws.cap_packets) break;
                    WalkPacket *o = out + first + q;
                    const int i = q + lane * np;
                    if (fits && i < n) {
                        const int at = i < n0 ? i : (i < n0 + n1 ? b1 + i - n0 : b2 + i - n0 - n1);
                        const uint2 e = sh.st[at];
                        float l = 0.f;
                        if constexpr (PROP) l = sh.l[at];
                        o->e[lane] = make_uint4(e.x, e.y, __float_as_uint(share_at(at)), __float_as_uint(l));
                    }
                    // no room for all: the packets there is room for are left
                    // empty and the warp walks on itself
                    if (lane == 0) {
                        o->count = fits ? (n - q + np - 1) / np : 0;
                        o->np = fits ? nb : 0;
                    }
                    if (fits && lane < nb) o->point[lane] = sh.point[lane];
                }
                if (fits) break;
                two = false;
            }
            const WalkTake take = walk_take(n0, n1, n2, two);
            const int k0 = take.k0, k1 = take.k1, k2 = take.k2;
            const bool fast = take.fast;
            const int k = k0 + k1 + k2;
            const int j = lane >> 1;
            const bool right = lane & 1, act = j < k;
            unsigned code = 0;
            float cpmf = 0.f, apmf = 0.f, lpmf = 0.f;
            if (act) {
                const int at = j < k2 ? b2 + n2 - 1 - j : (j < k2 + k1 ? b1 + n1 - 1 - (j - k2) : n0 - 1 - (j - k2 - k1));
                const uint2 e = sh.st[at];
                code = e.x;
                apmf = __uint_as_float(e.y);
                cpmf = share_at(at);
                if constexpr (PROP) lpmf = sh.l[at];
            }
            n0 -= k0;
            n1 -= k1;
            n2 -= k2;
            visits += k;
            __syncwarp();
            const int nid = (int)(code & DR_NODE_MASK), slot = (code >> 27) & 7;
            const bool cone_mode = !((code >> 30) & 1), all_split = code >> 31;
            const WalkCtx cx = ctx_of(slot);
            const float3 p = cx.p();
            const int tree = cx.tree();
            // the lane's child
            float3 lo = f3(0.f), hi = f3(0.f);
            float len = 0.f;
            int child = 0;
            bool cs = false;
            if (act) {
                const size_t at = 4 * (size_t)nid + (right ? 2 : 0);
                const float4 *b = (tree ? s.nrm_box : s.sil_box) + at;
                const float4 b0 = __ldg(b), b1 = __ldg(b + 1);
                lo = f3(b0.x, b0.y, b0.z);
                hi = f3(b1.x, b1.y, b1.z);
                len = b0.w;
                child = __float_as_int(b1.w);
                cs = true;
                if (tree) {
                    const float4 d0 = __ldg(s.nrm_dir + at), d1 = __ldg(s.nrm_dir + at + 1);
                    cs = cone_reaches_silhouette(sphere_center(lo, hi), d1.x, f3(d0.x, d0.y, d0.z), d0.w, d1.y, d1.z, p);
                }
            }
            // what becomes of the child: walked, its share of the walks
            bool push = false;
            float bb = 0.f, ccpmf = cpmf, capmf = apmf, clpmf = lpmf;
            if (fast) {
                // a node that splits: a child is walked if it can hold a
                // silhouette and its bound is above 0, as long as the two
                // importances are above the cutoff; its shares of both walks
                // are the node's
                float fm = 0.f, imp = 0.f;
                if (cs) {
                    if (!bsdf_bound_side(lo, hi, cx.bound(), bb, fm)) bb = walk_bound(lo, hi, cx.w);
                    imp = filt_div(bb * len, length_sq(p - 0.5f * (lo + hi)));
                }
                float sum = imp + __shfl_xor_sync(full, imp, 1);
                fm = fmaxf(fm, __shfl_xor_sync(full, fm, 1));
                const bool open = !(sum > 1e-10f * (1.0001f + 2.f * fm) || sum < 1e-10f * (0.9999f - 2.f * fm));
                if (__any_sync(full, act && open)) {
                    if (open && cs) {
                        bb = walk_bound(lo, hi, cx.w);
                        imp = box_importance(lo, hi, len, bb, p);
                    }
                    const float exact = imp + __shfl_xor_sync(full, imp, 1);
                    if (open) sum = exact;
                }
                push = cs && !(sum <= 1e-10f) && !(bb <= 0.f);
            } else {
            // its bound and importance (node_children's rules)
            float imp = 0.f;
            if (cs) {
                bb = walk_bound(lo, hi, cx.w);
                imp = box_importance(lo, hi, len, bb, p);
            }
            const float oimp = __shfl_xor_sync(full, imp, 1);
            const bool ocs = __shfl_xor_sync(full, (int)cs, 1);
            const float il = right ? oimp : imp, ir = right ? imp : oimp;
            bool walk = act && !(il + ir <= 1e-10f);
            bool hc = false;
            // (a node that splits the all walk gives each child its whole share
            // whatever the cone tests say)
            const bool cone_tests =
                walk && (cone_mode || (!all_split && (cpmf != 0.f || !dr_isfinite(il) || !dr_isfinite(ir))));
            if (__any_sync(full, cone_tests)) {
                if (cone_tests) hc = box_cone_box(lo, hi, cx.cone());
            }
            const bool ohc = __shfl_xor_sync(full, (int)hc, 1);
            const bool lhc = right ? ohc : hc, rhc = right ? hc : ohc;
            if (cone_mode && (lhc ? il : 0.f) + (rhc ? ir : 0.f) <= 1e-10f) walk = false;
            const ChildShares sh2 = child_shares(il, ir, lhc, rhc, right ? ocs : cs, right ? cs : ocs, all_split,
                                                 cx.w[22]);
            float pl = right ? sh2.pra : sh2.pla, plleft = sh2.pla;
            if constexpr (PROP) {
                // the proposal's choice: importance times the learned weight
                // of the direction towards each child
                float g = 0.f;
                const bool lrn = walk && !all_split && il > 0.f && ir > 0.f;
                if (lrn) g = imp * box_dir_weight(ws.proposal_q + 32 * (size_t)point_of(slot), cx.frame(), p, lo, hi);
                const float og = __shfl_xor_sync(full, g, 1);
                const float gl = right ? og : g, gr = right ? g : og;
                if (lrn && gl + gr > 0.f) {
                    plleft = gl / (gl + gr);
                    pl = right ? 1.f - plleft : plleft;
                }
            }
            if (walk) {
                if (cone_mode ? sh2.cone_split : all_split) {
                    push = cs && !(bb <= 0.f);
                } else {
                    const float u = cx.rng().draw(cone_mode ? 0 : 1, nid);
                    const float pick = cone_mode ? sh2.plc : ((PROP && (cx.flags() & 8)) ? plleft : sh2.pla);
                    push = ((u < pick) != right) && !(bb <= 0.f);
                }
            }
            ccpmf = (right ? sh2.prc : sh2.plc) * cpmf;
            capmf = (right ? sh2.pra : sh2.pla) * apmf;
            walk_undefined(!cone_mode, ccpmf, capmf);
            clpmf = pl * lpmf;
            }
            const bool leaf = push && (child & DR_CHILD_LEAF);
            float w = 0.f;
            if (leaf) {  // EdgeWalk::leaf's weight; no item of weight 0 is kept
                float a = capmf;
                if constexpr (PROP) a = ws.proposal_alpha * clpmf + (1.f - ws.proposal_alpha) * capmf;
                const float denom = ccpmf * ccpmf + a * a;
                w = cone_mode ? ccpmf / denom : a / denom;
            }
            // an edge that is a silhouette from everywhere is an item at once;
            // the others wait for their test
            const bool sure = leaf && w != 0.f && (child & DR_CHILD_SURE) && !(PROP && ws.train_targets);
            const bool keep = leaf && w != 0.f && !sure, node = push && !leaf;
            const unsigned ml = __ballot_sync(full, keep), ms = __ballot_sync(full, sure);
            visits += __popc(__ballot_sync(full, leaf));
            const unsigned tag = code & (15u << 27);  // slot and mode
            push_nodes(node, tag | (unsigned)child | ((bb > 1.f || box_inside(lo, hi, p)) ? 1u << 31 : 0u), ccpmf, capmf,
                       clpmf);
            if (keep) {
                sh.leaf[nl + __popc(ml & below)] =
                    make_uint2(tag | (unsigned)(child & DR_NODE_MASK) | ((child & DR_CHILD_MANY) ? 1u << 31 : 0u),
                               __float_as_uint(w));
            } else if (sure) {
                const int at = ni + __popc(ms & below);
                sh.item[at] = make_uint2(tag | (unsigned)(child & DR_NODE_MASK), __float_as_uint(w));
                if constexpr (PROP) sh.item_code[at] = 0;
                if (nb > 1) atomicAdd(&sh.cnt[slot], 1);
            }
            if (nb == 1 && lane == 0) sh.cnt[0] += __popc(ms);
            ni += __popc(ms);
            nl += __popc(ml);
            __syncwarp();
            if (ni > DR_WALK_ITEMS - 32) flush();
            if (nl >= 32) leaves(32);
        }
        if (nl > 0) leaves(nl);
        if (ni > 0) flush();
        __syncwarp();
        if (ws.pt_items && lane < nb) {
            if (!in) ws.pt_items[point_of(lane)] = sh.cnt[lane];
            else if (sh.cnt[lane] > 0) atomicAdd(ws.pt_items + point_of(lane), sh.cnt[lane]);
        }
        __syncwarp();
    }
    if (lane == 0) {
        atomicAdd(&ws.counters->visits_tasks, visits);
        atomicAdd(&ws.counters->tasks, walked);
    }
}
