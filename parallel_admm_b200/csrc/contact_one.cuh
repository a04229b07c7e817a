// contact_one.cuh -- the friction-cone projections of one ADMM iteration (project_impl,
// contact_solver.cu:316-431, after the warm start of k_contact_p) in one launch of one block, for
// detections of up to kOneContacts contacts.
#pragma once
#include "contact.cuh"

namespace admm {

constexpr int kOneVerts = 4 * kOneContacts;
constexpr int kOneShort = 4;                   // lists of up to so many entries: a thread per vertex

struct ContactOneSmem {
    float4 p[kOneVerts];          // of the vertices with contacts, in the order of tvr (w: vertex)
    float4 du[kOneContacts];
    float2 ent[4 * kOneContacts]; // ginc
    unsigned list[kOneVerts];     // list begin | entries << 16; static vertices: 0 entries
    unsigned short shorts[kOneVerts], longs[kOneVerts];  // dynamic vertices by length of their lists
    int nshort, nlong;
};

// What lanes b + sub, b + sub + 8, ... of a group add up in gather_group (v: du).
template <class Entry, class Du>
ADMM_DEV float4 contact_lane_sum(int b, int e, int sub, unsigned gmask, Entry entry, Du du) {
    float ax = 0.f, ay = 0.f, az = 0.f;
    for (int k = b + sub; k < e; k += kGatherLanes) {
        const float2 gi = entry(k);
        const float4 d = du(__float_as_int(gi.x));
        ax = fmaf(d.x, gi.y, ax);
        ay = fmaf(d.y, gi.y, ay);
        az = fmaf(d.z, gi.y, az);
    }
#pragma unroll
    for (int o = kGatherLanes / 2; o > 0; o >>= 1) {
        ax += __shfl_xor_sync(gmask, ax, o, kGatherLanes);
        ay += __shfl_xor_sync(gmask, ay, o, kGatherLanes);
        az += __shfl_xor_sync(gmask, az, o, kGatherLanes);
    }
    return f4(ax, ay, az);
}

// The same for a list of 1 to kOneShort entries by one thread: the partial sums of lanes 0..3,
// combined as by the xor shuffles.
template <class Entry, class Du>
ADMM_DEV float4 contact_short_sum(int b, int len, Entry entry, Du du) {
    float4 a[kOneShort];
#pragma unroll
    for (int l = 0; l < kOneShort; l++) {
        const float2 gi = entry(l < len ? b + l : b);
        const float4 d = du(__float_as_int(gi.x));
        a[l] = l < len ? f4(fmaf(d.x, gi.y, 0.f), fmaf(d.y, gi.y, 0.f), fmaf(d.z, gi.y, 0.f)) : f4(0.f, 0.f, 0.f);
    }
    return add3(add3(a[0], a[2]), add3(a[1], a[3]));
}

// More contacts than fit (the host switches to a launch per pass where that pays, see
// pick_contact_passes):
// the same passes in global memory.
ADMM_DEV void contact_one_global(const DevScene& s, int nc, int passes) {
    const int lane = threadIdx.x & 31, sub = lane % kGatherLanes, grp = lane / kGatherLanes, ntv = *s.ntv;
    const unsigned gmask = 0xffu << (lane & ~(kGatherLanes - 1));
    auto entry = [&](int k) { return s.ginc[k]; };
    auto du = [&](int c) { return s.du[c]; };
    for (int pass = 1; pass <= passes; pass++) {
        for (int c = threadIdx.x; c < nc; c += blockDim.x) {
            const ContactRec R = contact_rec(s, c);
            const float4 r = s.rc[c];
            float ux, uy, uz;
            contact_u_bk(R.b, R.kc, s.p[R.q.x], s.p[R.q.y], s.p[R.q.z], s.p[R.q.w], ux, uy, uz);
            const float4 d = cone_du(R.n, R.mu, ux, uy, uz, r);
            s.du[c] = d;
            s.rc[c] = f4(r.x + d.x, r.y + d.y, r.z + d.z);
        }
        __syncthreads();
        if (ntv <= 4 * kOneContacts / kGatherLanes) {  // few turns: a group per vertex
            for (int t = threadIdx.x / kGatherLanes; t < ntv; t += kOneContacts / kGatherLanes) {
                const int4 v = s.tvr[t];
                if (v.x >= s.nd) continue;  // the same in the whole group
                const float4 a = contact_lane_sum(v.y, v.z, sub, gmask, entry, du);
                if (sub == 0) s.p[v.x] = add3(s.p[v.x], a);
            }
            __syncthreads();
            continue;
        }
        // a thread per vertex with a short list, the long lists of a warp's vertices four at a time
        for (int t0 = 0; t0 < ntv; t0 += kOneContacts) {
            // one turn: dealt out over the warps; more: consecutive vertices, read together
            const int t = ntv <= kOneContacts ? lane * (kOneContacts / 32) + (threadIdx.x >> 5) : t0 + threadIdx.x;
            const int4 v = t < ntv ? s.tvr[t] : make_int4(0, 0, 0, 0);
            const int len = v.x < s.nd ? v.z - v.y : 0;
            if (len > 0 && len <= kOneShort) s.p[v.x] = add3(s.p[v.x], contact_short_sum(v.y, len, entry, du));
            for (unsigned m = __ballot_sync(~0u, len > kOneShort); m;) {
                unsigned r = m;
                for (int k = 0; k < grp; k++) r &= r - 1;  // this group's vertex: bit number grp
                const int from = r ? __ffs(r) - 1 : 0;
                const int x = __shfl_sync(~0u, v.x, from), b = __shfl_sync(~0u, v.y, from), n = __shfl_sync(~0u, len, from);
                if (r) {
                    const float4 a = contact_lane_sum(b, b + n, sub, gmask, entry, du);
                    if (sub == 0) s.p[x] = add3(s.p[x], a);
                }
                for (int k = 0; k < 32 / kGatherLanes; k++) m &= m - 1;
            }
        }
        __syncthreads();
    }
}

// One block holds the whole contact problem: p of the touched vertices, du and the incidence
// entries in shared memory, a contact's record and r_c in its thread's registers.  A pass is the
// projection of every contact (k_contact_du), a block barrier, p of every touched vertex
// (k_contact_gather, the same sums in the same order) and another: no launch, which cost 2.5 us
// whatever its size.  The kernel before it (k_contact_p) waits before it triggers, so the
// detection's data is loaded before the wait (see contact.cuh).
__global__ void __launch_bounds__(kOneContacts, 1) k_contact_one(DevScene s, int passes) {
    extern __shared__ __align__(128) unsigned char csm[];
    ContactOneSmem& m = *(ContactOneSmem*)csm;
    const int nc = __ldcg(s.nc);
    if (nc == 0 || nc > kOneContacts) {
        ADMM_PDL_WAIT_THEN_TRIGGER();
        if (nc > 0) contact_one_global(s, nc, passes);
        return;
    }
    const int tid = threadIdx.x, ntv = __ldcg(s.ntv);  // at most 4 nc
    if (tid == 0) m.nshort = m.nlong = 0;
    ContactRec R = {};
    int t01 = 0, t23 = 0;  // places of the contact's vertices among the touched ones
    if (tid < nc) {
        R = contact_rec(s, tid);
        t01 = __ldcg(&s.cinc[4 * tid]).w | __ldcg(&s.cinc[4 * tid + 1]).w << 16;
        t23 = __ldcg(&s.cinc[4 * tid + 2]).w | __ldcg(&s.cinc[4 * tid + 3]).w << 16;
    }
    for (int k = tid; k < 4 * nc; k += kOneContacts) m.ent[k] = __ldcg(&s.ginc[k]);
    __syncthreads();
    for (int t = tid; t < ntv; t += kOneContacts) {
        const int4 v = __ldcg(&s.tvr[t]);
        const int len = v.x < s.nd ? v.z - v.y : 0;
        m.list[t] = (unsigned)v.y | (unsigned)len << 16;
        m.p[t].w = __int_as_float(v.x);
        if (len > kOneShort) m.longs[atomicAdd(&m.nlong, 1)] = (unsigned short)t;
        else if (len > 0) m.shorts[atomicAdd(&m.nshort, 1)] = (unsigned short)t;
    }
    ADMM_PDL_WAIT_THEN_TRIGGER();
    for (int t = tid; t < ntv; t += kOneContacts) {
        const float w = m.p[t].w;
        const float4 p = s.p[__float_as_int(w)];
        m.p[t] = make_float4(p.x, p.y, p.z, w);
    }
    float4 rc = tid < nc ? s.rc[tid] : f4(0.f, 0.f, 0.f);
    __syncthreads();
    const int nshort = m.nshort, nlong = m.nlong, sub = tid % kGatherLanes;
    const unsigned gmask = 0xffu << (tid & 31 & ~(kGatherLanes - 1));
    for (int pass = 1; pass <= passes; pass++) {
        if (tid < nc) {
            float ux, uy, uz;
            contact_u_bk(R.b, R.kc, m.p[t01 & 0xffff], m.p[t01 >> 16], m.p[t23 & 0xffff], m.p[t23 >> 16], ux, uy, uz);
            const float4 d = cone_du(R.n, R.mu, ux, uy, uz, rc);
            rc = f4(rc.x + d.x, rc.y + d.y, rc.z + d.z);
            m.du[tid] = d;
        }
        __syncthreads();
        const bool last = pass == passes;
        auto finish = [&](int t, float4 a) {
            float4 p = m.p[t];
            p = make_float4(p.x + a.x, p.y + a.y, p.z + a.z, p.w);
            if (last) s.p[__float_as_int(p.w)] = f4(p.x, p.y, p.z);
            else m.p[t] = p;
        };
        for (int k = tid; k < nshort; k += kOneContacts) {
            const int t = m.shorts[k], b = m.list[t] & 0xffffu, len = m.list[t] >> 16;
            finish(t, contact_short_sum(b, len, [&](int e) { return m.ent[e]; }, [&](int c) { return m.du[c]; }));
        }
        for (int k = tid / kGatherLanes; k < nlong; k += kOneContacts / kGatherLanes) {
            const int t = m.longs[k], b = m.list[t] & 0xffffu;
            const float4 a = contact_lane_sum(b, b + (int)(m.list[t] >> 16), sub, gmask, [&](int e) { return m.ent[e]; },
                                              [&](int c) { return m.du[c]; });
            if (sub == 0) finish(t, a);
        }
        if (!last) __syncthreads();
    }
    if (tid < nc) s.rc[tid] = rc;
}

}  // namespace admm
