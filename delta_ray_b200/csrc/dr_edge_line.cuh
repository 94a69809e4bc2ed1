// The line samples of the sampled edges: the point on each edge and the hits
// of its two side rays on the edge's own faces.  Included by
// dr_edge_kernels.cu.
#pragma once

// Each point's line-sample setup (line_setup: the point's edge draw, lobe
// pick and LTC transforms), the same for all of its thousands of edges: the
// line kernel reads it instead of setting it up per edge.  Layout, float4:
// 0-2 minv and 3-5 m with the lobe's pick probability, the draw's u, ok and
// the point's position in the last words of the two matrices' rows; MIS (the
// lobe mixture weight): 6-8 the other lobe's transform and its pick
// probability.
template <bool MIS>
__global__ void __launch_bounds__(128, 8) k_line_ctx(const __grid_constant__ DevScene s, uint64_t seed, BackwardWorkspace ws) {
    const long long n = min(min((long long)ws.counters->points, ws.cap_points), ws.pt_end);
    for (long long p = ws.pt_begin + (long long)blockIdx.x * blockDim.x + threadIdx.x; p < n;
         p += (long long)gridDim.x * blockDim.x) {
        PointRecord pt;
        pt.load(ws.pt + (size_t)p * DR_PT_WORDS);
        Rng prng;
        prng.init(point_seed(ws, pt.view, seed), kStreamEdgePoint, pt.sid, (uint32_t)pt.bounce);
        const EdgeSample es = draw_edge(prng);
        const SurfacePoint sp = pt.surface();
        const LineSetup ls = line_setup(s, es, pt.wi, pt.tri, sp);
        const float *a = ls.minv.m, *b = ls.m.m;
        float4 *o = ws.line_ctx + (size_t)p * DR_LCTX_F4;
        o[0] = make_float4(a[0], a[1], a[2], a[3]);
        o[1] = make_float4(a[4], a[5], a[6], a[7]);
        o[2] = make_float4(a[8], b[0], b[1], b[2]);
        o[3] = make_float4(b[3], b[4], b[5], b[6]);
        o[4] = make_float4(b[7], b[8], ls.mpmf, es.u);
        o[5] = make_float4(ls.ok ? 1.f : 0.f, pt.p.x, pt.p.y, pt.p.z);
        if constexpr (MIS) {
            float opmf = 0.f;
            M3 om = ls.minv;
            if (ls.ok) {
                const bool sel_diffuse = es.bsdf_component <= ls.dpmf;
                opmf = sel_diffuse ? ls.spmf : ls.dpmf;
                if (opmf > 0.f) om = other_lobe(s, ls.mi, sp, pt.wi, ls.frame, sel_diffuse);
            }
            o[6] = make_float4(om.m[0], om.m[1], om.m[2], om.m[3]);
            o[7] = make_float4(om.m[4], om.m[5], om.m[6], om.m[7]);
            o[8] = make_float4(om.m[8], opmf, 0.f, 0.f);
        }
    }
}

// A warp's tile of lines, by field: the item and the draw's u, the clipped edge
// (a, b: 6 fields from kVoX) and then its LineState, last the kept samples'
// records (8 fields from kItem).
#define DR_TILE 128
struct LineTile {
    float f[13][DR_TILE];
};
enum { kItem, kU, kVoX, kVoY, kVoZ, kWtX, kWtY, kWtZ, kD, kIl0, kNorm, kL0, kL1 };

// A warp takes a run of items and works in phases over shared memory, so that
// the lanes of each phase mostly have work: clip every edge and drop those
// whose faces the side rays surely miss (faces_out_of_reach), gathering the
// rest into a tile of up to 128; set the tile's lines up; solve for the offsets
// (a lane takes the tile's next line as its own converges: 2 to 19 steps);
// sample the points and test the edges' faces, keeping the samples that hit
// one.
//
// What bounds it: instruction issue (about 2,100 instructions per solved item;
// divisions and square roots are IEEE sequences).  One lane per item from start
// to end issued with 15.7 of 32 lanes active, most steps waiting for the few
// lines of the warp that ran all 20.  At the 130,054-triangle heightfield half
// of the items are dropped before they are solved (two thirds of those whose
// rays miss the faces).  Measured there: 88 -> 40 ms at 640x480, 1 spp (508 M
// items), 5.5 -> 2.6 at 160x120; with the lobe mixture weight on a 64x64-vertex
// heightfield (15.5 M items) 5.4 -> 2.6.  21 of 32 lanes active.
template <bool MIS>
__global__ void __launch_bounds__(128, DR_LINE_BLOCKS) k_edge_line(const __grid_constant__ DevScene s, BackwardWorkspace ws) {
    __shared__ LineTile block_tile[4];
    LineTile &t = block_tile[threadIdx.x >> 5];
    const unsigned full = 0xffffffffu;
    const int lane = threadIdx.x & 31;
    const unsigned below = (1u << lane) - 1u;
    const long long n = (long long)min(ws.counters->items, (unsigned long long)ws.cap_items);
    const long long warps = (long long)gridDim.x * (blockDim.x >> 5);
    // runs of up to 512 items, shorter where items are few for the warps there are
    const long long run = 32 * max(1ll, min(16ll, n / (64 * warps)));
    const auto rec_of = [&](const int4 &it) {
        return ((it.y >> 30) ? s.nrm_rec : s.sil_rec) + (it.y & ((1 << 30) - 1));
    };
    for (long long base = ((long long)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5)) * run; base < n;
         base += warps * run) {
        const long long end = min(base + run, n);
        long long pos = base;
        while (pos < end) {
            // clip and gather
            int cnt = 0;
            for (; cnt <= DR_TILE - 32 && pos < end; pos += 32) {
                const long long i = pos + lane;
                float3 a = f3(0.f), b = f3(0.f);
                float u = 0.f;
                bool ok = false;
                if (i < end) {
                    const int4 it = ws.items[i];
                    const EdgeRec *rec = rec_of(it);
                    const float4 *c = ws.line_ctx + (size_t)it.x * DR_LCTX_F4;
                    const float4 c0 = c[0], c1 = c[1], c2 = c[2], c3 = c[3], c4 = c[4], c5 = c[5];
                    const M3 minv = {{c0.x, c0.y, c0.z, c0.w, c1.x, c1.y, c1.z, c1.w, c2.x}};
                    const M3 m = {{c2.y, c2.z, c2.w, c3.x, c3.y, c3.z, c3.w, c4.x, c4.y}};
                    const float3 v0 = rec_v0(rec), v1 = rec_v1(rec), p = f3(c5.y, c5.z, c5.w);
                    u = c4.w;
                    ok = c5.x != 0.f && line_clip(minv, v0, v1, p, a, b) &&
                         !faces_out_of_reach(rec, v0, v1, p, m, fmaxf(abs_sum(a), abs_sum(b)));
                }
                const unsigned mask = __ballot_sync(full, ok);
                if (ok) {
                    const int j = cnt + __popc(mask & below);
                    t.f[kItem][j] = __int_as_float((int)i), t.f[kU][j] = u;
                    t.f[kVoX][j] = a.x, t.f[kVoY][j] = a.y, t.f[kVoZ][j] = a.z;
                    t.f[kWtX][j] = b.x, t.f[kWtY][j] = b.y, t.f[kWtZ][j] = b.z;
                }
                cnt += __popc(mask);
            }
            __syncwarp();
            // set the lines up
            for (int j = lane; j < cnt; j += 32) {
                LineState ln;
                const bool ok = line_begin(f3(t.f[kVoX][j], t.f[kVoY][j], t.f[kVoZ][j]),
                                           f3(t.f[kWtX][j], t.f[kWtY][j], t.f[kWtZ][j]), ln);
                t.f[kVoX][j] = ln.vo.x, t.f[kVoY][j] = ln.vo.y, t.f[kVoZ][j] = ln.vo.z;
                t.f[kWtX][j] = ln.wt.x, t.f[kWtY][j] = ln.wt.y, t.f[kWtZ][j] = ln.wt.z;
                t.f[kD][j] = ln.d, t.f[kIl0][j] = ln.Il0;
                t.f[kNorm][j] = ok ? ln.norm : -1.f;  // -1: no line (a line's norm is above 1e-10, or NaN)
                t.f[kL0][j] = ln.l0, t.f[kL1][j] = ln.l1;
            }
            __syncwarp();
            // solve: a lane's line stays in registers until it converges; idle
            // lanes take new lines together once a quarter of the warp is idle
            {
                LineState ln;
                ln.vo = ln.wt = f3(0.f);  // the solve needs the z parts only
                ln.d = ln.l0 = ln.l1 = ln.Il0 = ln.norm = 0.f;
                LineSolve sv;
                sv.begin(ln);
                float u = 0.f;
                int idx = -1, next = 0;
                while (true) {
                    const unsigned idle = __ballot_sync(full, idx < 0);
                    if (next < cnt && (__popc(idle) >= 8 || idle == full)) {
                        const int mine = next + __popc(idle & below);
                        if (idx < 0 && mine < cnt && t.f[kNorm][mine] != -1.f) {
                            idx = mine;
                            ln.vo.z = t.f[kVoZ][idx], ln.wt.z = t.f[kWtZ][idx];
                            ln.d = t.f[kD][idx], ln.Il0 = t.f[kIl0][idx], ln.norm = t.f[kNorm][idx];
                            ln.l0 = t.f[kL0][idx], ln.l1 = t.f[kL1][idx], u = t.f[kU][idx];
                            sv.begin(ln);
                        }
                        next += __popc(idle);
                        continue;
                    }
                    if (idle == full) break;
                    if (idx >= 0 && sv.step(ln, u)) {
                        t.f[kL0][idx] = sv.l;
                        idx = -1;
                    }
                }
            }
            __syncwarp();
            // sample and test the faces; the kept samples' records gather at
            // the front of the tile, over lines that have been read
            int kept = 0;
            for (int j0 = 0; j0 < cnt; j0 += 32) {
                const int j = j0 + lane;
                bool ok = j < cnt && t.f[kNorm][j] != -1.f;
                float3 sample_p = f3(0.f), mwt = f3(0.f);
                float q = 0.f;
                int i = 0;
                if (ok) {
                    LineState ln;
                    ln.vo = f3(t.f[kVoX][j], t.f[kVoY][j], t.f[kVoZ][j]);
                    ln.wt = f3(t.f[kWtX][j], t.f[kWtY][j], t.f[kWtZ][j]);
                    ln.d = t.f[kD][j], ln.norm = t.f[kNorm][j];
                    const float l = t.f[kL0][j], pdf = ln.pdf(l);
                    i = __float_as_int(t.f[kItem][j]);
                    ok = !(pdf <= 0.f);
                    if (ok) {
                        const int4 it = ws.items[i];
                        const EdgeRec *rec = rec_of(it);
                        const float4 *c = ws.line_ctx + (size_t)it.x * DR_LCTX_F4;
                        const float4 c2 = c[2], c3 = c[3], c4 = c[4], c5 = c[5];
                        const M3 m = {{c2.y, c2.z, c2.w, c3.x, c3.y, c3.z, c3.w, c4.x, c4.y}};
                        const float3 p = f3(c5.y, c5.z, c5.w), v0 = rec_v0(rec), v1 = rec_v1(rec);
                        EdgeLine el;
                        el.sample_p = sample_p = mul(m, ln.vo + l * ln.wt);
                        mwt = mul(m, ln.wt);
                        q = c4.z * pdf;
                        // the connectivity test's first part: a sample neither of
                        // whose rays hits one of the edge's faces is connected on
                        // no side
                        float3 sdir, rdir, ldir;
                        edge_side_dirs(el, v0, v1, p, sdir, rdir, ldir);
                        Hit fr, fl;
                        hit_faces_pair(rec, p, rdir, ldir, 1e-3f, fr, fl);
                        ok = fr.tri >= 0 || fl.tri >= 0;
                        if constexpr (MIS) {
                            const float4 c6 = c[6], c7 = c[7], c8 = c[8];
                            if (ok && c8.y > 0.f) {
                                const M3 om = {{c6.x, c6.y, c6.z, c6.w, c7.x, c7.y, c7.z, c7.w, c8.x}};
                                q += c8.y * lobe_line_density(om, v0 - p, v1 - p, sample_p, mwt);
                            }
                        }
                    }
                }
                const unsigned mask = __ballot_sync(full, ok);
                __syncwarp();  // every lane has read its line (a vote orders no memory)
                if (ok) {
                    const int k = kept + __popc(mask & below);
                    t.f[0][k] = __int_as_float(i);
                    t.f[1][k] = sample_p.x, t.f[2][k] = sample_p.y, t.f[3][k] = sample_p.z;
                    t.f[4][k] = mwt.x, t.f[5][k] = mwt.y, t.f[6][k] = mwt.z, t.f[7][k] = q;
                }
                kept += __popc(mask);
                __syncwarp();
            }
            unsigned long long first = 0;
            if (lane == 0 && kept > 0) first = atomicAdd(&ws.counters->survivors, (unsigned long long)kept);
            first = __shfl_sync(full, first, 0);
            // two lanes write one 32-byte record
            for (int k = lane; k < 2 * kept; k += 32) {
                const int a = k >> 1, h = 4 * (k & 1);
                ws.survivors[2 * first + k] = make_float4(t.f[h][a], t.f[h + 1][a], t.f[h + 2][a], t.f[h + 3][a]);
            }
            __syncwarp();
        }
    }
}

// The same without the points' setups (the no-alloc backward, whose scratch
// holds none): one lane per item, the setup per edge.  EXT:
// DR_FLAG_EDGE_LOBE_MIS or proposal training in use.
template <bool EXT>
__global__ void __launch_bounds__(128, 4) k_edge_line_point(const __grid_constant__ DevScene s, uint64_t seed, BackwardWorkspace ws) {
    const long long n = (long long)min(ws.counters->items, (unsigned long long)ws.cap_items);
    const long long stride = (long long)gridDim.x * blockDim.x;
    // warp-uniform loop: the survivor append is warp-aggregated
    for (long long base = (long long)blockIdx.x * blockDim.x + (threadIdx.x & ~31); base < n; base += stride) {
        const long long i = base + (threadIdx.x & 31);
        EdgeLine el;
        bool ok = false;
        if (i < n) {
            const int4 it = ws.items[i];
            const int tree = it.y >> 30, ei = it.y & ((1 << 30) - 1);
            PointRecord pt;
            pt.load(ws.pt + (size_t)it.x * DR_PT_WORDS);
            ok = item_line<EXT>(s, pt, tree, ei, point_seed(ws, pt.view, seed), el);
            if (ok) {
                const EdgeRec *rec = (tree ? s.nrm_rec : s.sil_rec) + ei;
                float3 sdir, rdir, ldir;
                edge_side_dirs(el, rec_v0(rec), rec_v1(rec), pt.p, sdir, rdir, ldir);
                Hit fr, fl;
                hit_faces_pair(rec, pt.p, rdir, ldir, 1e-3f, fr, fl);
                ok = fr.tri >= 0 || fl.tri >= 0;
            }
        }
        __syncwarp();
        const unsigned long long slot = warp_reserve(&ws.counters->survivors, ok ? 1 : 0);
        if (ok) {
            ws.survivors[2 * slot] = make_float4(__int_as_float((int)i), el.sample_p.x, el.sample_p.y, el.sample_p.z);
            ws.survivors[2 * slot + 1] = make_float4(el.mwt.x, el.mwt.y, el.mwt.z, el.q);
        }
    }
}
