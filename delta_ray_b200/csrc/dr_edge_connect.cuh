// The ray stage of an LBVH scene, first half.  Included by dr_edge_kernels.cu.
#pragma once

// The ray stage of an LBVH scene in two kernels.  k_edge_connect decides
// each line sample's connectivity (the edge's faces and one or two bounded
// occlusion walks; most samples end here) and queues the few that go on;
// k_edge_pairs traces the other side's closest hit of those and runs the
// remaining tests.
//
// A state machine per lane, stepped by the whole warp: when at least half the
// warp has no walk (or none has), those lanes take one line sample each;
// otherwise the walking lanes take a step, nodes and leaves in turn.  (Lanes
// that ran their walks to the end before taking the next sample, and lanes that
// took one as soon as they were idle, left the warp split into groups issuing
// on their own: 5.1 and 3.8 of 32 lanes active.)
//
// What bounds it: L1 throughput (77 % of its peak: each walking lane reads its
// own 128-byte node) and issue (73 % of the slots).  So a lane first tests the
// last triangle it found in the way: samples follow each other by edge, and at
// the 130,054-triangle heightfield a blocker of the sample before blocks about
// half of the occluded right rays, the right ray's four in five of the left rays
// beside it, and a walk saved is about 45 nodes.  Any triangle that the walk
// would test and that blocks gives its answer (leaf_entered).  The boxes are
// tested with fused multiply-adds, which enter a few more than the walk's own
// test would.  The walk's stack lies in shared memory, a column per lane (in
// local memory it took as much of the L1's throughput as the nodes).  Measured
// there: 99 -> 69.5 ms at 640x480, 1 spp (120 M samples), 6.3 -> 4.5 at 160x120,
// 17.1 of 32 lanes active (14.7 before).  Dropped: lanes taking runs of 2, 4 or 8
// samples (7.1 ms with 8: neighbouring samples no longer share their nodes' cache
// lines across the warp), 6 and 7 blocks per SM.
#define DR_CONNECT_STACK 20  // deeper entries (up to DR_WIDE_STACK) go to local memory
__global__ void __launch_bounds__(128, DR_CONNECT_BLOCKS) k_edge_connect(const __grid_constant__ DevScene s, BackwardWorkspace ws) {
    __shared__ int stack[DR_CONNECT_STACK][128];
    int deep[DR_WIDE_STACK - DR_CONNECT_STACK];
    const long long n = (long long)min(ws.counters->survivors, (unsigned long long)ws.cap_items);
    const float tnear = 1e-3f;
    long long k = 0;  // the lane's sample
    int phase = 0;  // 0 no walk, 1 walking the right ray, 2 walking the left ray
    bool more = true, cr = false;
    float3 p = f3(0.f), d = f3(0.f), ldir = f3(0.f);
    FastRay ray = fast_ray(f3(0.f), f3(1.f));
    int r_tri = -1, l_tri = -1, node = 0, sp = 0, leaf = -1, blocker = -1;
    float l_t = 0.f, ta = 0.f;
    int ida = -1;
    const auto push = [&](int c) {
        if (sp < DR_CONNECT_STACK) stack[sp][threadIdx.x] = c;
        else if (sp < DR_WIDE_STACK) deep[sp - DR_CONNECT_STACK] = c;
        sp++;
    };
    const auto pop = [&]() {
        sp--;
        return sp < DR_CONNECT_STACK ? stack[sp][threadIdx.x] : deep[sp - DR_CONNECT_STACK];
    };
    // whether leaf's triangle hits ahead of (t_face, face) along dir
    const auto blocks = [&](int leaf, float3 dir, float t_face, int face) {
        const float4 a = __ldg(s.bvh_tris + 3 * leaf), b = __ldg(s.bvh_tris + 3 * leaf + 1),
                     c = __ldg(s.bvh_tris + 3 * leaf + 2);
        float t;
        return hit_triangle(a, b, c, p, dir, t) && t > tnear &&
               (t < t_face || (t == t_face && __float_as_int(a.w) < face)) &&
               leaf_entered(a, b, c, p, f3(safe_inv(dir.x), safe_inv(dir.y), safe_inv(dir.z)), t_face);
    };
    const auto begin = [&](int ph, float3 dir, float t_face, int face) {
        d = dir;
        ray = fast_ray(p, f3(safe_inv(d.x), safe_inv(d.y), safe_inv(d.z)));
        ta = t_face;
        ida = face;
        sp = 0;
        node = s.bvh_root;
        leaf = -1;
        phase = ph;
    };
    const auto candidate = [&](int side, int face) {
        const long long j = next_task(&ws.counters->cands);
        ws.hits[j] = make_int4((int)k, face, side, 0);
    };
    // the right ray is decided (cr): the left one decides the sample, unless
    // it hits no face; both connected, or neither, ends it
    const auto after_right = [&]() {
        phase = 0;
        if (l_tri < 0) {
            if (cr) candidate(0, r_tri);
        } else if (blocker >= 0 && blocks(blocker, ldir, l_t, l_tri)) {
            if (cr) candidate(0, r_tri);
        } else {
            begin(2, ldir, l_t, l_tri);
        }
    };
    while (true) {
        const unsigned walking = __ballot_sync(0xffffffffu, phase != 0);
        const unsigned idle = __ballot_sync(0xffffffffu, phase == 0 && more);
        if (walking == 0 && idle == 0) break;  // every lane's queue has ended
        const bool fetch = idle != 0 && (__popc(idle) >= 16 || walking == 0);
        if (fetch && phase == 0 && more) {  // one sample each
            k = next_task(&ws.counters->ray_next);
            more = k < n;
        }
        if (fetch && phase == 0 && more) {
            const float4 a = ws.survivors[2 * k];
            const int4 it = ws.items[__float_as_int(a.x)];
            const float *pw = ws.pt + (size_t)it.x * DR_PT_WORDS;  // the point's position: words 0-2
            const EdgeRec *rec = ((it.y >> 30) ? s.nrm_rec : s.sil_rec) + (it.y & ((1 << 30) - 1));
            p = f3(pw[0], pw[1], pw[2]);
            EdgeLine el;
            el.sample_p = f3(a.y, a.z, a.w);
            float3 sdir, rdir;
            edge_side_dirs(el, rec_v0(rec), rec_v1(rec), p, sdir, rdir, ldir);
            // the connectivity test of edge_connect_bvh, its walks stepped below
            Hit fr, fl;
            hit_faces_pair(rec, p, rdir, ldir, tnear, fr, fl);
            r_tri = fr.tri;
            l_tri = fl.tri;
            l_t = fl.t;
            cr = false;
            if (r_tri >= 0 && !(blocker >= 0 && blocks(blocker, rdir, fr.t, fr.tri))) begin(1, rdir, fr.t, fr.tri);
            else after_right();
        }
        if (fetch) continue;
        // A step of the walks: an inner node of every lane that has one, as long
        // as at least half of the walking lanes do; otherwise the leaves the
        // lanes have found.  A lane keeps one leaf aside and walks on past it
        // (Aila and Laine 2009, "Understanding the efficiency of ray traversal
        // on GPUs": speculative traversal), so that both kinds of step run
        // with most lanes.
        const unsigned inner = __ballot_sync(0xffffffffu, phase != 0 && node >= 0 && node != DR_WIDE_EMPTY);
        int res = 0;  // 1 a triangle ahead, 2 none, 0 not known yet
        if (2 * __popc(inner) >= __popc(walking)) {
            if (phase != 0 && node >= 0 && node != DR_WIDE_EMPTY) {
                const FastKids kids = fast_kids(s.bvh_wide + (size_t)DR_WIDE_F4 * node, ray, ta);
                if (!kids.any) {
                    node = sp > 0 ? pop() : DR_WIDE_EMPTY;
                } else {
                    if (sp <= DR_CONNECT_STACK - 3) {
                        for (int i = 3; i > 0; i--)
                            if (kids.hit[i]) stack[sp++][threadIdx.x] = kids.c[i];
                    } else {
                        for (int i = 3; i > 0; i--)
                            if (kids.hit[i]) push(kids.c[i]);
                    }
                    node = kids.c[0];
                }
                if (node < 0 && leaf < 0) {
                    leaf = ~node;
                    node = sp > 0 ? pop() : DR_WIDE_EMPTY;
                }
                if (node == DR_WIDE_EMPTY && leaf < 0) res = 2;
            }
        } else if (phase != 0 && leaf >= 0) {
            if (blocks(leaf, d, ta, ida)) {
                res = 1;
                blocker = leaf;
                leaf = -1;
            } else {
                leaf = -1;
                if (node < 0) {
                    leaf = ~node;
                    node = sp > 0 ? pop() : DR_WIDE_EMPTY;
                }
                if (node == DR_WIDE_EMPTY && leaf < 0) res = 2;
            }
        }
        if (res == 0) continue;
        if (phase == 1) {
            cr = res == 2;  // no triangle ahead of the right face hit
            after_right();
        } else {
            const bool cl = res == 2;
            phase = 0;
            if (cr != cl) candidate(cr ? 0 : 1, cr ? r_tri : l_tri);
        }
    }
}
