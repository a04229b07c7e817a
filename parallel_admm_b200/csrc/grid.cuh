// grid.cuh -- uniform-grid (spatial hash) broad phase for the DCD.
//
// The contact pair set of the reference's DCD (lbvh.cu:1693-1813) does not
// depend on the acceleration structure: a pair is reported when the query box
// overlaps the element box under the reference's rule (lbvh.cu:43-49) and the
// region-0 narrow phase accepts it.  A BVH query is a chain of dependent node
// loads (tens of L2 round trips per query for a few thousand queries, far too
// few threads to hide them); a grid query issues the loads of all of its cells
// at once, so a DCD costs a handful of round trips.
//
// Layout: every surface triangle and edge whose box spans at most kGridMaxSpan
// cells per axis is inserted into each cell it overlaps, in a hash table of
// (cell, type) buckets built by count -> place -> scatter; each entry carries
// the element's box and the key of the cell it was entered for, so that other
// cells sharing the bucket are rejected by one 8-byte compare and the box test
// needs no further load.  Larger
// elements (and any that do not fit the entry capacity) go to a per-type "big"
// list that the queries scan directly.
//
// Each pair is reported once: a query visits the cells of its box inflated by
// the gap (plus a margin that covers the rounding of the overlap test), and
// accepts an element only in the cell that is the lower corner of the overlap
// of the two cell ranges -- the cell that, on every axis, is the first of the
// query's range or the first of the element's (entries carry the latter as
// three bits).  Edge-edge pairs (a, b), a < b, with both edges in the
// grid belong to a; a pair of one grid edge and one big edge belongs to the
// grid edge; a pair of two big edges to the smaller index.  Every query sorts
// its output segment by partner index, so the contact list is independent of
// atomic arrival order.
#pragma once
#include "common.cuh"
#include "contact.cuh"
#include "lbvh.cuh"
#include "scene_dev.cuh"

namespace admm {

constexpr int kGridMaxSpan = 16;  // cells per axis an element may span in the grid

ADMM_DEV int grid_cell(float v, float inv_c) {
    float f = floorf(v * inv_c);
    f = fminf(fmaxf(f, -1048575.f), 1048575.f);  // the cell key holds 21 bits per coordinate
    return (int)f;
}

// Bucket of a cell: the low bits of the cell's Morton code, triangles in the
// lower half of the table, edges in the upper half.  Neighbouring cells land in
// neighbouring buckets, so the queries of neighbouring mesh vertices (which run
// in the same warps) read the same cache lines; cells whose codes differ only
// above the table size share a bucket and are told apart by the entry's cell key.
ADMM_DEV unsigned grid_spread10(unsigned v) {
    v &= 0x3ffu;
    v = (v | (v << 16)) & 0x030000ffu;
    v = (v | (v << 8)) & 0x0300f00fu;
    v = (v | (v << 4)) & 0x030c30c3u;
    v = (v | (v << 2)) & 0x09249249u;
    return v;
}

ADMM_DEV int grid_bucket(int ix, int iy, int iz, int type, int hmask) {
    const unsigned m = grid_spread10((unsigned)ix) | (grid_spread10((unsigned)iy) << 1) |
                       (grid_spread10((unsigned)iz) << 2);
    const unsigned half = (unsigned)hmask >> 1;  // hmask + 1 is a power of two >= 2
    return (int)((m & half) + (type ? half + 1u : 0u));
}

// 64-bit key of a cell (21 bits per coordinate, offset to non-negative).
ADMM_DEV unsigned long long grid_cell_key(int ix, int iy, int iz) {
    const unsigned long long o = 1ull << 20, m = (1ull << 21) - 1ull;
    return (((unsigned long long)(ix + (int)o) & m) << 42) | (((unsigned long long)(iy + (int)o) & m) << 21) |
           ((unsigned long long)(iz + (int)o) & m);
}

// Box of surface element u (triangles first, then edges); type 0 = triangle.
ADMM_DEV void grid_elem_box(const DevScene& s, int u, int& type, int& id, float4& lo, float4& up) {
    lo = f4(1e32f, 1e32f, 1e32f);
    up = f4(-1e32f, -1e32f, -1e32f);
    if (u < s.nst) {
        type = 0;
        id = u;
        const int4 t = s.st[u];
        box_add(lo, up, s.x[t.x]);
        box_add(lo, up, s.x[t.y]);
        box_add(lo, up, s.x[t.z]);
    } else {
        type = 1;
        id = u - s.nst;
        const int2 e = s.se[id];
        box_add(lo, up, s.x[e.x]);
        box_add(lo, up, s.x[e.y]);
    }
}

ADMM_DEV void grid_range(const float4& lo, const float4& up, float inv_c, int3& a, int3& b) {
    a = make_int3(grid_cell(lo.x, inv_c), grid_cell(lo.y, inv_c), grid_cell(lo.z, inv_c));
    b = make_int3(grid_cell(up.x, inv_c), grid_cell(up.y, inv_c), grid_cell(up.z, inv_c));
}

// Cell range of a query box inflated by the gap.  The margin keeps every element
// that passes box_overlap inside the range despite the rounding of its
// subtractions (a few ulps of the coordinates).
ADMM_DEV float grid_pad(float v, float gap) { return gap + fmaxf(gap, fabsf(v)) * (1.f / 1048576.f); }

// A query whose cell range is larger than this (a stretched element or far-out
// coordinates) tests every grid element of the type directly instead.
constexpr int kGridMaxQueryCells = 8192;

ADMM_DEV bool grid_range_small(int3 a, int3 b) {
    const long long n = (long long)(b.x - a.x + 1) * (long long)(b.y - a.y + 1) * (long long)(b.z - a.z + 1);
    return n >= 1 && n <= kGridMaxQueryCells;
}

ADMM_DEV void grid_query_range(const float4& lo, const float4& up, float gap, float inv_c, int3& a, int3& b) {
    a = make_int3(grid_cell(lo.x - grid_pad(lo.x, gap), inv_c), grid_cell(lo.y - grid_pad(lo.y, gap), inv_c),
                  grid_cell(lo.z - grid_pad(lo.z, gap), inv_c));
    b = make_int3(grid_cell(up.x + grid_pad(up.x, gap), inv_c), grid_cell(up.y + grid_pad(up.y, gap), inv_c),
                  grid_cell(up.z + grid_pad(up.z, gap), inv_c));
}

// Calls f(cell, bucket) for every cell [a, b] of one element.
template <class F>
ADMM_DEV void grid_for_cells(int3 a, int3 b, int type, int hmask, F f) {
    for (int iz = a.z; iz <= b.z; iz++)
        for (int iy = a.y; iy <= b.y; iy++)
            for (int ix = a.x; ix <= b.x; ix++) f(make_int4(ix, iy, iz, 0), grid_bucket(ix, iy, iz, type, hmask));
}

// Pass 1: bucket counts; elements that are too large (or beyond the entry
// capacity) go to the big lists.  ctr[0] = entries reserved, ctr[1..2] = big
// triangle / edge counts (zero before the launch).  Also clears the last detection's contact
// counts.
__global__ void __launch_bounds__(256) k_grid_count(DevScene s) {
    ADMM_PDL_PROLOGUE();
    const GridDev& g = s.grid;
    const int u = blockIdx.x * blockDim.x + threadIdx.x;
    contact_clear(s, u, gridDim.x * blockDim.x);
    if (u >= s.nst + s.nse) return;
    int type, id;
    float4 lo, up;
    grid_elem_box(s, u, type, id, lo, up);
    int3 a, b;
    grid_range(lo, up, g.inv_c, a, b);
    const int sx = b.x - a.x + 1, sy = b.y - a.y + 1, sz = b.z - a.z + 1;
    bool in_grid = sx >= 1 && sy >= 1 && sz >= 1 && sx <= kGridMaxSpan && sy <= kGridMaxSpan && sz <= kGridMaxSpan;
    if (in_grid) {
        const int nc = sx * sy * sz;
        const int r = atomicAdd(&g.ctr[0], nc);
        in_grid = r + nc <= g.cap;
    }
    g.mode[u] = in_grid ? 1 : 0;
    if (in_grid) {
        grid_for_cells(a, b, type, g.hmask, [&](int4, int bk) { atomicAdd(&g.cnt[bk], 1); });
    } else {
        const int k = atomicAdd(&g.ctr[1 + type], 1);
        (type == 0 ? g.big_tri : g.big_edge)[k] = id;
    }
}

// The buckets' places among the entries: consecutive within a block's 2048 buckets, the blocks in
// the order of their atomics (nothing depends on the entries' order: every query sorts its
// partners).  A bucket's place and size are one load for the queries, and no launch waits for
// a scan over all buckets.
__global__ void __launch_bounds__(kScanThreads) k_grid_alloc(DevScene s, int buckets) {
    ADMM_PDL_PROLOGUE();
    __shared__ int sh[32];
    __shared__ int first;
    const GridDev& g = s.grid;
    const int base = blockIdx.x * kScanTile + threadIdx.x * kScanItems;
    int v[kScanItems], t = 0;
#pragma unroll
    for (int k = 0; k < kScanItems; k++) {
        v[k] = base + k < buckets ? g.cnt[base + k] : 0;
        t += v[k];
    }
    int run = block_exclusive_scan(t, sh);
    if (threadIdx.x == kScanThreads - 1) first = run + t ? atomicAdd(&g.ctr[3], run + t) : 0;
    __syncthreads();
    run += first;
#pragma unroll
    for (int k = 0; k < kScanItems; k++) {
        if (base + k < buckets) g.bkt[base + k] = make_int2(run, v[k]);
        run += v[k];
    }
}

// Pass 2: entries, one per element
// and cell; the counts are consumed back to zero for the next DCD.
__global__ void __launch_bounds__(256) k_grid_scatter(DevScene s) {
    ADMM_PDL_PROLOGUE();
    const GridDev& g = s.grid;
    const int u = blockIdx.x * blockDim.x + threadIdx.x;
    if (u >= s.nst + s.nse || !g.mode[u]) return;
    int type, id;
    float4 lo, up;
    grid_elem_box(s, u, type, id, lo, up);
    int3 a, b;
    grid_range(lo, up, g.inv_c, a, b);
    lo.w = __int_as_float(id);
    grid_for_cells(a, b, type, g.hmask, [&](int4 c, int bk) {
        const int pos = g.bkt[bk].x + atomicSub(&g.cnt[bk], 1) - 1;
        // w of up: for each axis, whether this cell is the element's first
        const int first = (c.x == a.x ? 1 : 0) | (c.y == a.y ? 2 : 0) | (c.z == a.z ? 4 : 0);
        g.ent_lo[pos] = lo;
        g.ent_up[pos] = make_float4(up.x, up.y, up.z, __int_as_float(first));
        g.ent_key[pos] = grid_cell_key(c.x, c.y, c.z);
    });
}

// Insertion sort of the contact slots [b, e) by partner index.
ADMM_DEV void grid_sort_segment(const DevScene& s, int b, int e) {
    int* key = s.grid.qkey;
    for (int k = b + 1; k < e; k++) {
        const int kk = key[k];
        const int4 pr = s.pairs[k];
        const float4 pt = s.point[k], ba = s.bary[k], nr = s.nrm[k];
        int j = k - 1;
        while (j >= b && key[j] > kk) {
            key[j + 1] = key[j];
            s.pairs[j + 1] = s.pairs[j];
            s.point[j + 1] = s.point[j];
            s.bary[j + 1] = s.bary[j];
            s.nrm[j + 1] = s.nrm[j];
            j--;
        }
        key[j + 1] = kk;
        s.pairs[j + 1] = pr;
        s.point[j + 1] = pt;
        s.bary[j + 1] = ba;
        s.nrm[j + 1] = nr;
    }
}

// ---------------------------------------------------------------------------
// Queries: k_grid_count_pairs (L lanes per query) counts and records each query's partners,
// k_grid_write_pairs writes the contacts.  grid_walk is the walk of one query by a whole warp, for
// the few queries whose range or partners outgrow those kernels.
// ---------------------------------------------------------------------------
constexpr int kQueryThreads = 128;  // block size of the query kernels
constexpr int kQueryHitsMax = 32;   // partners the count pass records per query

ADMM_DEV int3 grid_cell_at(int3 a, int3 b, int ci) {
    const int dx = b.x - a.x + 1, dy = b.y - a.y + 1;
    return make_int3(a.x + ci % dx, a.y + (ci / dx) % dy, a.z + ci / (dx * dy));
}

ADMM_DEV int grid_cells(int3 a, int3 b) { return (b.x - a.x + 1) * (b.y - a.y + 1) * (b.z - a.z + 1); }

ADMM_DEV float4 tri_box_lo(const DevScene& s, int f, float4& up) {
    const int4 t = s.st[f];
    float4 lo = f4(1e32f, 1e32f, 1e32f);
    up = f4(-1e32f, -1e32f, -1e32f);
    box_add(lo, up, s.x[t.x]);
    box_add(lo, up, s.x[t.y]);
    box_add(lo, up, s.x[t.z]);
    return lo;
}

ADMM_DEV float4 edge_box_lo(const DevScene& s, int o, float4& up) {
    const int2 e = s.se[o];
    float4 lo = f4(1e32f, 1e32f, 1e32f);
    up = f4(-1e32f, -1e32f, -1e32f);
    box_add(lo, up, s.x[e.x]);
    box_add(lo, up, s.x[e.y]);
    return lo;
}

// Candidate partners waiting for the narrow phase (64 slots in shared memory; the fill n is the
// same in every lane).
struct GridQueue {
    int* buf;
    int n;
};

// Queues the partner of every lane with ok set (called by the whole warp);
// once 32 or more wait, hands the first 32 to narrow(partner, true).
template <class F>
ADMM_DEV void grid_queue_push(GridQueue& q, bool ok, int partner, F& narrow) {
    const int lane = threadIdx.x & 31;
    const unsigned m = __ballot_sync(~0u, ok);
    if (ok) q.buf[q.n + __popc(m & ((1u << lane) - 1u))] = partner;
    q.n += __popc(m);
    if (q.n >= 32) {
        __syncwarp();
        const int p = q.buf[lane];
        if (lane < q.n - 32) q.buf[lane] = q.buf[32 + lane];
        __syncwarp();
        q.n -= 32;
        narrow(p, true);
    }
}

template <class F>
ADMM_DEV void grid_queue_drain(GridQueue& q, F& narrow) {
    if (q.n == 0) return;
    __syncwarp();
    const int lane = threadIdx.x & 31;
    const bool valid = lane < q.n;
    const int p = valid ? q.buf[lane] : 0;
    __syncwarp();
    q.n = 0;
    narrow(p, valid);
}

// A warp's walk of one query.  Vertex query (vf): position P = lo = up
// against the triangles.  Edge query: edge e with box [lo, up] against grid
// edges with a larger index (grid edge e), every big edge (grid edge e) or big
// edges with a larger index (big edge e).  Grid part: the cells of the query's
// range, or every grid element of the type when the range is too large.
template <bool CPU, class F>
ADMM_DEV void grid_walk(const DevScene& s, bool vf, int e, float4 lo, float4 up, GridQueue& q, F& narrow) {
    const GridDev& g = s.grid;
    const float gap = s.thickness;
    constexpr int G = 32;
    const int sub = threadIdx.x & 31;
    const unsigned gm = ~0u;
    const int type = vf ? 0 : 1;
    const bool small = vf || g.mode[s.nst + e] != 0;
    if (small) {
        int3 a, b;
        grid_query_range(lo, up, gap, g.inv_c, a, b);
        if (grid_range_small(a, b)) {
            const int nc = grid_cells(a, b);
            for (int c0 = 0; c0 < nc; c0 += G) {
                int cnt = 0, d = 0, qfirst = 0;
                unsigned long long key = 0ull;
                if (c0 + sub < nc) {
                    const int3 c = grid_cell_at(a, b, c0 + sub);
                    const int bk = grid_bucket(c.x, c.y, c.z, type, g.hmask);
                    const int2 e = g.bkt[bk];
                    d = e.x;
                    cnt = e.y;
                    key = grid_cell_key(c.x, c.y, c.z);
                    qfirst = (c.x == a.x ? 1 : 0) | (c.y == a.y ? 2 : 0) | (c.z == a.z ? 4 : 0);
                }
                int incl = cnt;
#pragma unroll
                for (int o = 1; o < G; o <<= 1) {
                    const int y = __shfl_up_sync(gm, incl, o, G);
                    if (sub >= o) incl += y;
                }
                d -= incl - cnt;  // entry number k of the round lies at d of its cell + k
                const int tot = __shfl_sync(gm, incl, G - 1, G);
                for (int k0 = 0; k0 < tot; k0 += G) {
                    const int k = k0 + sub;
                    // the cell of entry k: the first lane of the group whose inclusive count exceeds k
                    int j = 0;
#pragma unroll
                    for (int st = G / 2; st >= 1; st >>= 1) {
                        if (__shfl_sync(gm, incl, j + st - 1, G) <= k) j += st;
                    }
                    const int dj = __shfl_sync(gm, d, j, G);
                    const int fj = __shfl_sync(gm, qfirst, j, G);
                    const unsigned long long kj = __shfl_sync(gm, key, j, G);
                    bool ok = false;
                    int partner = 0;
                    if (k < tot) {
                        const int ent = dj + k;
                        const unsigned long long ek = g.ent_key[ent];
                        const float4 eup = g.ent_up[ent];
                        const float4 elo = g.ent_lo[ent];
                        partner = __float_as_int(elo.w);
                        // same cell (not another of the bucket); larger edge index; once per pair:
                        // this cell is the first of the query's or of the element's range on every axis
                        ok = ek == kj && (vf || partner > e) && ((fj | __float_as_int(eup.w)) & 7) == 7 &&
                             (CPU || box_overlap(lo, up, elo, eup, gap));
                    }
                    grid_queue_push(q, ok, partner, narrow);
                }
            }
        } else {
            const int n = vf ? s.nst : s.nse;
            for (int t0 = vf ? 0 : e + 1; t0 < n; t0 += G) {
                const int t = t0 + sub;
                bool ok = false;
                if (t < n && g.mode[vf ? t : s.nst + t]) {
                    float4 eup;
                    const float4 elo = vf ? tri_box_lo(s, t, eup) : edge_box_lo(s, t, eup);
                    ok = CPU || box_overlap(lo, up, elo, eup, gap);
                }
                grid_queue_push(q, ok, t, narrow);
            }
        }
    }
    const int nb = g.ctr[1 + type];
    for (int j0 = 0; j0 < nb; j0 += G) {
        const int j = j0 + sub;
        bool ok = false;
        int o = 0;
        if (j < nb) {
            o = vf ? g.big_tri[j] : g.big_edge[j];
            if (vf || (o != e && (small || o > e))) {
                float4 oup;
                const float4 olo = vf ? tri_box_lo(s, o, oup) : edge_box_lo(s, o, oup);
                ok = CPU || box_overlap(lo, up, olo, oup, gap);  // the overlap rule is symmetric
            }
        }
        grid_queue_push(q, ok, o, narrow);
    }
    grid_queue_drain(q, narrow);
}

// ---------------------------------------------------------------------------
// Cheap distance filters in front of the exact narrow phase of the CPU backend's predicates (its
// closest points over all regions are long; the GPU backend's predicate rejects by region within
// fewer operations than the filter takes).  Closest points by
// the Voronoi-region construction (point-triangle) and the clamped-parameter
// construction (segment-segment), in ordinary FP32 arithmetic.  A pair is
// dropped only when this distance exceeds 1.1 x thickness plus 1e-5 of the
// largest coordinate -- orders of magnitude above the rounding of either
// computation -- so the exact predicate (d < thickness) could not have accepted
// it; non-finite intermediate values never drop a pair.  On flat cloth most
// box-overlapping non-adjacent pairs are neighbours a cell apart, and this
// keeps them out of the heavy non-contracting narrow phase.
// ---------------------------------------------------------------------------
ADMM_DEV float d3(float4 a, float4 b) { return a.x * b.x + a.y * b.y + a.z * b.z; }

ADMM_DEV float fast_pt_dist2(float4 p, float4 a, float4 b, float4 c) {
    const float4 ab = sub3(b, a), ac = sub3(c, a), ap = sub3(p, a);
    const float q1 = d3(ab, ap), q2 = d3(ac, ap);
    float4 x;
    if (q1 <= 0.f && q2 <= 0.f) {
        x = a;
    } else {
        const float4 bp = sub3(p, b);
        const float q3 = d3(ab, bp), q4 = d3(ac, bp);
        const float4 cp = sub3(p, c);
        const float q5 = d3(ab, cp), q6 = d3(ac, cp);
        const float vc = q1 * q4 - q3 * q2, vb = q5 * q2 - q1 * q6, va = q3 * q6 - q5 * q4;
        if (q3 >= 0.f && q4 <= q3) {
            x = b;
        } else if (vc <= 0.f && q1 >= 0.f && q3 <= 0.f) {
            x = add3(a, scale3(ab, q1 / (q1 - q3)));
        } else if (q6 >= 0.f && q5 <= q6) {
            x = c;
        } else if (vb <= 0.f && q2 >= 0.f && q6 <= 0.f) {
            x = add3(a, scale3(ac, q2 / (q2 - q6)));
        } else if (va <= 0.f && (q4 - q3) >= 0.f && (q5 - q6) >= 0.f) {
            x = add3(b, scale3(sub3(c, b), (q4 - q3) / ((q4 - q3) + (q5 - q6))));
        } else {
            const float den = 1.f / (va + vb + vc);
            x = add3(a, add3(scale3(ab, vb * den), scale3(ac, vc * den)));
        }
    }
    const float4 d = sub3(p, x);
    return d3(d, d);
}

ADMM_DEV float fast_ee_dist2(float4 p1, float4 q1, float4 p2, float4 q2) {
    const float4 u = sub3(q1, p1), v = sub3(q2, p2), w = sub3(p1, p2);
    const float a = d3(u, u), e = d3(v, v), f = d3(v, w);
    float sp, tp;
    const float tiny = 1e-30f;
    if (a <= tiny && e <= tiny) {
        sp = tp = 0.f;
    } else if (a <= tiny) {
        sp = 0.f;
        tp = fminf(fmaxf(f / e, 0.f), 1.f);
    } else {
        const float c = d3(u, w);
        if (e <= tiny) {
            tp = 0.f;
            sp = fminf(fmaxf(-c / a, 0.f), 1.f);
        } else {
            const float b = d3(u, v), den = a * e - b * b;
            sp = den > 0.f ? fminf(fmaxf((b * f - c * e) / den, 0.f), 1.f) : 0.f;
            tp = (b * sp + f) / e;
            if (tp < 0.f) {
                tp = 0.f;
                sp = fminf(fmaxf(-c / a, 0.f), 1.f);
            } else if (tp > 1.f) {
                tp = 1.f;
                sp = fminf(fmaxf((b - c) / a, 0.f), 1.f);
            }
        }
    }
    const float4 d = sub3(add3(p1, scale3(u, sp)), add3(p2, scale3(v, tp)));
    return d3(d, d);
}

ADMM_DEV bool surely_apart(float d2, float thickness, float4 a, float4 b, float4 c, float4 d) {
    const float r = fmaxf(fmaxf(fmaxf(fabsf(a.x), fabsf(a.y)), fmaxf(fabsf(a.z), fabsf(b.x))),
                          fmaxf(fmaxf(fabsf(b.y), fabsf(b.z)), fmaxf(fmaxf(fabsf(c.x), fabsf(c.y)),
                                                                      fmaxf(fabsf(c.z), fmaxf(fmaxf(fabsf(d.x), fabsf(d.y)), fabsf(d.z))))));
    const float lim = 1.1f * thickness + 1e-5f * r;
    return d2 > lim * lim;  // false for NaN
}

// Narrow phase of vertex v against triangle f: the GPU backend's (region 0,
// 0 <= d < thickness) or, with cpu_contact, the CPU backend's (no pair of two
// static elements, any closest point, d <= thickness).
template <bool CPU>
ADMM_DEV bool grid_hit_vf(const DevScene& s, int v, float4 P, int f, int4& ids, NpResult& r) {
    const int4 tri = s.st[f];
    if (v == tri.x || v == tri.y || v == tri.z) return false;
    if (CPU && v >= s.nd && tri.x >= s.nd) return false;
    ids = make_int4(v, tri.x, tri.y, tri.z);
    const float4 a = s.x[tri.x], b = s.x[tri.y], c = s.x[tri.z];
    if (CPU) {
        if (surely_apart(fast_pt_dist2(P, a, b, c), s.thickness, P, a, b, c)) return false;
        closest_pt_all(P, a, b, c, r);
        return r.dist <= s.thickness;
    }
    return narrow_pt(P, a, b, c, r) && r.dist < s.thickness && r.dist >= 0.f;
}

// Narrow phase of edges e and o (no shared vertex), lower index first: the GPU
// backend's (region 0) or, with cpu_contact, the CPU backend's (no pair of two
// static edges, d < thickness unless both closest points are end points).
template <bool CPU>
ADMM_DEV bool grid_hit_ee(const DevScene& s, int e, int o, int4& ids, NpResult& r) {
    const int2 ed = s.se[e], od = s.se[o];
    if (ed.x == od.x || ed.x == od.y || ed.y == od.x || ed.y == od.y) return false;
    const int2 lo = o > e ? ed : od, hi = o > e ? od : ed;
    if (CPU && lo.x >= s.nd && hi.x >= s.nd) return false;
    ids = make_int4(lo.x, lo.y, hi.x, hi.y);
    const float4 p0 = s.x[lo.x], p1 = s.x[lo.y], q0 = s.x[hi.x], q1 = s.x[hi.y];
    if (CPU) {
        if (surely_apart(fast_ee_dist2(p0, p1, q0, q1), s.thickness, p0, p1, q0, q1)) return false;
        closest_ee_all(p0, p1, q0, q1, r);
        const bool corner = (r.bary[0] == 0.f || r.bary[0] == 1.f) && (r.bary[1] == 0.f || r.bary[1] == 1.f);
        return r.dist < s.thickness && !corner;
    }
    return narrow_ee(p0, p1, q0, q1, r) && r.dist < s.thickness && r.dist >= 0.f;
}

// Is (query q, partner) a pair?  Surface vertices first, then edges.
template <bool CPU>
ADMM_DEV bool grid_pair(const DevScene& s, int q, int partner, int4& ids, NpResult& r) {
    if (q < s.nsv) {
        const int v = s.sv[q];
        return grid_hit_vf<CPU>(s, v, s.x[v], partner, ids, r);
    }
    return grid_hit_ee<CPU>(s, q - s.nsv, partner, ids, r);
}

// Box of query q.
ADMM_DEV void grid_query_box(const DevScene& s, int q, float4& lo, float4& up) {
    if (q < s.nsv) lo = up = s.x[s.sv[q]];
    else lo = edge_box_lo(s, q - s.nsv, up);
}

// Count pass: the pair count of every query (qcount) and up to kQueryHitsMax of its partners
// (qhits, in no order).
//
// L lanes serve a query, 32 / L queries a warp, and the warp stays together.  The non-empty cells
// of every query's range are listed in shared memory (kQueryCells at a time); each lane then takes
// every L-th entry of its query's cells, one per turn of the loop, and goes on to the next cell by
// itself, so a turn costs the loads of an entry's box and a few compares: no scan over the cells
// and no search for an entry's cell.  The cell key is read only for entries that pass the box test.
// Candidates of all the warp's queries go to one queue, from which the narrow phase takes 32 at a
// time.  A query whose range has more than kQueryWarpCells cells is walked by the whole warp.
// Bound by instruction issue and the entries' load latency: a typical edge query looks at 50 to 110
// entries, of which ten pass the box test.  64 registers (8 blocks per SM): with 88 the detections
// of a substep of the 147 k queries of 24 bodies took 1.51 ms, with 64 1.25, with 48 1.37; before
// (a scan over the cells, a search for each entry's cell, a queue per query and the distance filter in
// front of both predicates) 1.78.  140 k queries of the two 128 x 128 sheets: 1.33 -> 1.09 ms.
constexpr int kQueryCells = 32;
constexpr int kQueryWarpCells = 256;

template <int L, bool CPU>
__global__ void __launch_bounds__(kQueryThreads, 8) k_grid_count_pairs(DevScene s) {
    ADMM_PDL_PROLOGUE();
    constexpr int NQ = 32 / L, W = kQueryThreads / 32;
    constexpr unsigned all = ~0u;
    __shared__ int4 cell_list[W][NQ][kQueryCells];
    __shared__ int2 queue_buf[W][64];
    __shared__ int hit_count[W][NQ];
    const GridDev& g = s.grid;
    const int nq = s.nsv + s.nse;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, qi = lane / L, sub = lane % L;
    const int q0 = (blockIdx.x * W + warp) * NQ;
    if (q0 >= nq) return;
    int4* cells = cell_list[warp][qi];
    int2* queue = queue_buf[warp];
    int* hits = hit_count[warp];
    const int q = q0 + qi;
    const bool live = q < nq;
    const bool vf = q < s.nsv;
    const int type = vf ? 0 : 1;
    const int e = vf ? -1 : q - s.nsv;  // edge queries take partners of a larger index
    const bool small = live && (vf || g.mode[s.nst + e] != 0);
    const float gap = s.thickness;
    float4 lo = f4(0.f, 0.f, 0.f), up = lo;
    int3 a = make_int3(0, 0, 0), b = a;
    int nc = 0, nb = live ? g.ctr[1 + type] : 0;
    bool wide = false;
    if (live) grid_query_box(s, q, lo, up);
    if (small) {
        grid_query_range(lo, up, gap, g.inv_c, a, b);
        wide = !grid_range_small(a, b) || grid_cells(a, b) > kQueryWarpCells;
        nc = wide ? 0 : grid_cells(a, b);
    }
    if (wide) nb = 0;
    if (lane < NQ) hits[lane] = 0;
    const int dx = b.x - a.x + 1, dy = b.y - a.y + 1;
    const int mx = 65535 / dx + 1, my = 65535 / dy + 1;  // n / d = n * m >> 16 for n < 256
    int c0 = 0;          // cells of the range listed so far
    int li = 0, ln = 0;  // the lane's place in the list, the list's length
    int ent = 0, rem = 0, first = 0;  // the lane's next entry, entries from there to the cell's end
    float4 elo = lo, eup = lo;        // that entry's box, loaded a turn ahead
    auto fetch = [&]() {
        while (rem <= 0 && li < ln) {
            const int2 c = *reinterpret_cast<const int2*>(cells + li++);
            ent = c.x + sub;
            rem = (c.y & 0x1fffffff) - sub;
            first = (int)((unsigned)c.y >> 29);
        }
        if (rem > 0) {
            elo = g.ent_lo[ent];
            eup = g.ent_up[ent];
        }
    };
    int j = sub;  // place in the big list
    int n = 0;    // queued candidates (the same in every lane)
    auto push = [&](bool ok, int from, int what) {
        const unsigned m = __ballot_sync(all, ok);
        if (ok) queue[n + __popc(m & ((1u << lane) - 1u))] = make_int2(from, what);
        n += __popc(m);
    };
    bool big = false;
    for (;;) {
        bool more;
        if (!big) {
            while ((more = __any_sync(all, rem > 0)) && n < 32) {
                // larger edge index; once per pair: this cell is the first of the query's or of the
                // element's range on every axis
                const bool ok = rem > 0 && __float_as_int(elo.w) > e && ((first | __float_as_int(eup.w)) & 7) == 7 &&
                                (CPU || box_overlap(lo, up, elo, eup, gap));
                const int from = qi | (li << 8), what = ent;
                ent += L;
                rem -= L;
                fetch();
                push(ok, from, what);
            }
        } else {
            while ((more = __any_sync(all, j < nb)) && n < 32) {
                bool ok = false;
                int partner = 0;
                if (j < nb) {
                    partner = vf ? g.big_tri[j] : g.big_edge[j];
                    if (vf || (partner != e && (small || partner > e))) {
                        float4 oup;
                        const float4 olo = vf ? tri_box_lo(s, partner, oup) : edge_box_lo(s, partner, oup);
                        ok = CPU || box_overlap(lo, up, olo, oup, gap);  // the rule is symmetric
                    }
                    j += L;
                }
                push(ok, qi, partner);
            }
        }
        if (n >= 32 || (!more && n > 0)) {
            __syncwarp();
            bool valid = lane < n;
            const int2 it = valid ? queue[lane] : make_int2(0, 0);
            const int2 nx = lane + 32 < n ? queue[lane + 32] : make_int2(0, 0);
            __syncwarp();
            if (lane + 32 < n) queue[lane] = nx;
            n = max(n - 32, 0);
            const int iq = it.x & 255, pos = it.x >> 8;
            int partner = it.y;
            if (pos > 0) {  // an entry: of the cell itself, not of another in its bucket?
                const int4 c = cell_list[warp][iq][pos - 1];
                partner = __float_as_int(g.ent_lo[it.y].w);
                valid = valid && g.ent_key[it.y] == ((unsigned long long)(unsigned)c.z | ((unsigned long long)(unsigned)c.w << 32));
            }
            int4 ids;
            NpResult r;
            if (valid && grid_pair<CPU>(s, q0 + iq, partner, ids, r)) {
                const int h = atomicAdd(&hits[iq], 1);
                if (h < kQueryHitsMax) g.qhits[(size_t)(q0 + iq) * kQueryHitsMax + h] = partner;
            }
            __syncwarp();
        } else if (!more) {
            if (big) break;
            if (__any_sync(all, c0 < nc)) {
                int len = 0;
                for (int t = 0; t < kQueryCells && __any_sync(all, c0 + t < nc); t += L) {
                    const int ci = c0 + t + sub;
                    int4 c = make_int4(0, 0, 0, 0);
                    if (ci < nc) {
                        const int row = ci * mx >> 16, layer = row * my >> 16;
                        const int3 p = make_int3(a.x + ci - row * dx, a.y + row - layer * dy, a.z + layer);
                        const int2 r = g.bkt[grid_bucket(p.x, p.y, p.z, type, g.hmask)];
                        const unsigned long long kk = grid_cell_key(p.x, p.y, p.z);
                        const unsigned f = (p.x == a.x ? 1 : 0) | (p.y == a.y ? 2 : 0) | (p.z == a.z ? 4 : 0);
                        c = make_int4(r.x, r.y, (int)(unsigned)kk, (int)(unsigned)(kk >> 32));
                        if (r.y > 0) c.y |= (int)(f << 29);
                    }
                    const unsigned mm = (__ballot_sync(all, c.y != 0) >> (lane - sub)) & (L == 32 ? all : (1u << L) - 1u);
                    if (c.y != 0) cells[len + __popc(mm & ((1u << sub) - 1u))] = c;
                    len += __popc(mm);
                }
                __syncwarp();
                c0 += kQueryCells;
                li = 0;
                ln = len;
                fetch();
            } else {
                big = true;
            }
        }
    }
    for (unsigned wm = __ballot_sync(all, wide && sub == 0); wm; wm &= wm - 1) {
        const int wq = q0 + (__ffs(wm) - 1) / L;
        float4 wlo, wup;
        grid_query_box(s, wq, wlo, wup);
        GridQueue gq{reinterpret_cast<int*>(queue), 0};
        int nhit = 0;
        auto narrow = [&](int partner, bool valid) {
            int4 ids;
            NpResult r;
            const bool hit = valid && grid_pair<CPU>(s, wq, partner, ids, r);
            const unsigned m = __ballot_sync(all, hit);
            const int h = nhit + __popc(m & ((1u << lane) - 1u));
            if (hit && h < kQueryHitsMax) g.qhits[(size_t)wq * kQueryHitsMax + h] = partner;
            nhit += __popc(m);
        };
        grid_walk<CPU>(s, wq < s.nsv, wq - s.nsv, wlo, wup, gq, narrow);
        if (lane == 0) hits[wq - q0] = nhit;
    }
    __syncwarp();
    if (lane < NQ && q0 + lane < nq) s.qcount[q0 + lane] = hits[lane];
}

// Write pass: places each recorded partner at the query's offset + its rank among the query's
// partners, so the segment comes out sorted by partner, and counts the contacts' vertices.  A lane
// holds a query, and the pairs of the warp's 32 queries are dealt out over its lanes.  A query
// with more partners than were recorded walks the grid again with the whole warp, writes in walk
// order and sorts its segment.
template <bool CPU>
__global__ void __launch_bounds__(kQueryThreads) k_grid_write_pairs(DevScene s) {
    ADMM_PDL_PROLOGUE();
    constexpr unsigned all = ~0u;
    __shared__ int qbuf[kQueryThreads / 32][64];
    const int nq = s.nsv + s.nse;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int q0 = blockIdx.x * kQueryThreads + warp * 32;
    if (q0 >= nq) return;
    const int total = q0 + lane < nq ? s.qcount[q0 + lane] : 0;
    if (!__any_sync(all, total > 0)) return;
    const int base = total > 0 ? query_offset(s, q0 + lane) : 0;
    int incl = total <= kQueryHitsMax ? total : 0;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int y = __shfl_up_sync(all, incl, o);
        if (lane >= o) incl += y;
    }
    const int sum = __shfl_sync(all, incl, 31);
    for (int i0 = 0; i0 < sum; i0 += 32) {
        const int i = i0 + lane;
        int j = 0;  // the query of pair i: the first lane whose inclusive count exceeds i
#pragma unroll
        for (int st = 16; st >= 1; st >>= 1)
            if (__shfl_sync(all, incl, j + st - 1) <= i) j += st;
        const int tj = __shfl_sync(all, total, j), bj = __shfl_sync(all, base, j), ij = __shfl_sync(all, incl, j);
        if (i < sum) {
            const int q = q0 + j;
            const int* qh = s.grid.qhits + (size_t)q * kQueryHitsMax;
            const int partner = qh[i - (ij - tj)];
            int rank = 0;
            for (int k = 0; k < tj; k++) rank += qh[k] < partner ? 1 : 0;
            int4 ids;
            NpResult r;
            const int slot = bj + rank;
            if (grid_pair<CPU>(s, q, partner, ids, r) && slot < s.cap) {
                write_contact(s, slot, ids, r, q >= s.nsv);
                contact_touch(s, slot, ids);
            }
        }
    }
    for (unsigned wm = __ballot_sync(all, total > kQueryHitsMax); wm; wm &= wm - 1) {
        const int l = __ffs(wm) - 1, q = q0 + l;
        const int wbase = __shfl_sync(all, base, l), end = min(wbase + __shfl_sync(all, total, l), s.cap);
        float4 lo, up;
        grid_query_box(s, q, lo, up);
        GridQueue gq{qbuf[warp], 0};
        int nhit = 0;
        auto emit = [&](int partner, bool valid) {
            int4 ids;
            NpResult r;
            const bool hit = valid && grid_pair<CPU>(s, q, partner, ids, r);
            const unsigned m = __ballot_sync(all, hit);
            const int slot = wbase + nhit + __popc(m & ((1u << lane) - 1u));
            if (hit && slot < s.cap) {
                write_contact(s, slot, ids, r, q >= s.nsv);
                s.grid.qkey[slot] = partner;
            }
            nhit += __popc(m);
        };
        grid_walk<CPU>(s, q < s.nsv, q - s.nsv, lo, up, gq, emit);
        __syncwarp();
        if (lane == 0 && end - wbase > 1) grid_sort_segment(s, wbase, end);
        __syncwarp();
        for (int c = wbase + lane; c < end; c += 32) contact_touch(s, c, s.pairs[c]);
    }
}

}  // namespace admm
