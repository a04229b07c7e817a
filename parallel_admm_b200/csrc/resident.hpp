// resident.hpp -- host plan of the cluster-resident global step (resident.cuh).
//
// The rows of the off-diagonal matrix are split into groups that share no entry (whole
// connected components), one thread-block cluster per group; within a group the rows are cut
// into one spatially compact range per CTA.  A CTA keeps its rows' matrix entries and the
// iterate (its own rows and the halo rows their entries reach) in shared memory for all
// sweeps of a global step; after a sweep it writes its new values into the halo slots of the
// CTAs of its cluster that read them.
//
// A row is summed as k_jacobi sums it (kernels.cuh: EllRowPf): entry k of the row goes to
// partial sum k % T in the order of k, and the T partial sums are combined in the order of
// the xor shuffles with distances 1, 2, 4 of partial indices, so both give the same bits.  TP
// threads of a warp share a row: thread j holds the partial sums j * Q .. j * Q + Q - 1
// (Q = T / TP).
#pragma once
#include <algorithm>
#include <cstdint>
#include <cstring>
#include <numeric>
#include <utility>
#include <vector>

#include "setup.hpp"

namespace admm {

// One CTA's part of the plan; offsets in bytes from the start of its blob (16-byte aligned).
struct ResidentCta {
    int own, halo;         // rows it computes; rows it only reads (slots own .. own + halo - 1)
    int slices;            // warps' worth of own rows (32 / TP rows each)
    int off_grow;          // int [own + halo]: global row of a slot
    int off_pptr;          // uint16 [own + 1]: push list of an own row
    int off_push;          // uint32 [pushes]: target CTA rank << 16 | its slot
    int off_sptr;          // int [slices + 1]: first pair step of a slice
    int off_val, off_col;  // float2 / uint32 (two slots) per pair step and lane; the diagonal is at 0
    int bytes;             // blob size, a multiple of 16
    int pad_;
    long long blob;        // offset of the blob in the plan's buffer
};

struct HostResident {
    bool ok = false;
    int cluster = 0, groups = 0, tp = 0, q = 0, threads = 0;
    int max_own = 0, max_local = 0, max_blob = 0;
    long long max_entries = 0;  // padded entries of the largest CTA
    std::vector<ResidentCta> cta;
    std::vector<unsigned char> blob;
};

constexpr int kResidentThreads = 512;  // most threads of a CTA (128 registers each)

// Connected components of the pattern: comp[i] in [0, count).
inline int row_components(const HostCsr& A, int nd, std::vector<int>& comp) {
    comp.assign(nd, -1);
    std::vector<int> stack;
    int count = 0;
    for (int r = 0; r < nd; r++) {
        if (comp[r] >= 0) continue;
        comp[r] = count;
        stack.push_back(r);
        while (!stack.empty()) {
            const int i = stack.back();
            stack.pop_back();
            for (int k = A.start[i]; k < A.start[i + 1]; k++)
                if (comp[A.col[k]] < 0) {
                    comp[A.col[k]] = count;
                    stack.push_back(A.col[k]);
                }
        }
        count++;
    }
    return count;
}

// Work of a row in the resident sweep: its entries plus what a row costs besides.
inline long long resident_weight(const HostCsr& A, int r) { return A.start[r + 1] - A.start[r] + 4; }

// The rows of every component in the order of a Morton curve through their positions (10 bits
// per axis), components in descending order of work.
struct ResidentOrder {
    std::vector<int> row;             // rows, component after component
    std::vector<int> begin;           // [components + 1] first row of a component
    std::vector<long long> weight;    // [components]
    long long total = 0;
};

inline ResidentOrder resident_order(const HostCsr& A, int nd, const float* pos, int stride) {
    ResidentOrder o;
    std::vector<int> comp;
    const int nc = row_components(A, nd, comp);
    std::vector<long long> w(nc, 0);
    for (int r = 0; r < nd; r++) w[comp[r]] += resident_weight(A, r);
    std::vector<int> by(nc), rank(nc);
    std::iota(by.begin(), by.end(), 0);
    std::stable_sort(by.begin(), by.end(), [&](int a, int b) { return w[a] > w[b]; });
    for (int k = 0; k < nc; k++) rank[by[k]] = k;
    std::vector<float> lo(3 * (size_t)nc, 1e30f), hi(3 * (size_t)nc, -1e30f);
    for (int r = 0; r < nd; r++)
        for (int k = 0; k < 3; k++) {
            const float p = pos[(size_t)stride * r + k];
            lo[3 * (size_t)comp[r] + k] = std::min(lo[3 * (size_t)comp[r] + k], p);
            hi[3 * (size_t)comp[r] + k] = std::max(hi[3 * (size_t)comp[r] + k], p);
        }
    std::vector<std::pair<uint64_t, int>> key(nd);
    for (int r = 0; r < nd; r++) {
        const int c = comp[r];
        float ext = 0.f;
        for (int k = 0; k < 3; k++) ext = std::max(ext, hi[3 * (size_t)c + k] - lo[3 * (size_t)c + k]);
        uint32_t q[3];
        for (int k = 0; k < 3; k++) {
            const float u = ext > 0.f ? (pos[(size_t)stride * r + k] - lo[3 * (size_t)c + k]) / ext : 0.f;
            q[k] = u > 0.f ? (uint32_t)std::min(1023.f, u * 1023.f) : 0u;  // non-finite positions: 0
        }
        key[r] = {(uint64_t)rank[c] << 32 | (spread10_host(q[0]) | spread10_host(q[1]) << 1 | spread10_host(q[2]) << 2),
                  r};
    }
    std::sort(key.begin(), key.end());
    o.row.resize(nd);
    for (int k = 0; k < nd; k++) o.row[k] = key[k].second;
    o.begin.assign(nc + 1, 0);
    for (int r = 0; r < nd; r++) o.begin[rank[comp[r]] + 1]++;
    for (int k = 0; k < nc; k++) o.begin[k + 1] += o.begin[k];
    o.weight.resize(nc);
    for (int k = 0; k < nc; k++) {
        o.weight[k] = w[by[k]];
        o.total += o.weight[k];
    }
    return o;
}

// Components to groups, largest first to the lightest group; the heaviest group's work.
inline long long resident_groups(const ResidentOrder& o, int groups, std::vector<int>* of = nullptr) {
    std::vector<std::pair<long long, int>> heap;
    for (int g = 0; g < groups; g++) heap.push_back({0, g});
    auto cmp = [](const std::pair<long long, int>& a, const std::pair<long long, int>& b) { return a > b; };
    if (of) of->assign(o.weight.size(), 0);
    long long most = 0;
    for (size_t c = 0; c < o.weight.size(); c++) {
        std::pop_heap(heap.begin(), heap.end(), cmp);
        heap.back().first += o.weight[c];
        if (of) (*of)[c] = heap.back().second;
        most = std::max(most, heap.back().first);
        std::push_heap(heap.begin(), heap.end(), cmp);
    }
    return most;
}

// Shared memory of a CTA: two iterates, `own_bytes` per own row, the blob.
inline long long resident_smem(const HostResident& p, int own_bytes) {
    return 2ll * 16 * p.max_local + (long long)own_bytes * ((p.max_own + 3) / 4 * 4) + p.max_blob;
}

// The plan for `groups` clusters of `cluster` CTAs and T partial sums per row.
inline HostResident build_resident(const HostCsr& A, const std::vector<float>& diag, int nd, int T,
                                   const ResidentOrder& o, int cluster, int groups) {
    HostResident p;
    std::vector<int> group_of;
    resident_groups(o, groups, &group_of);
    std::vector<std::vector<int>> rows(groups);
    std::vector<long long> work(groups, 0);
    for (size_t c = 0; c < o.weight.size(); c++) {
        auto& g = rows[group_of[c]];
        g.insert(g.end(), o.row.begin() + o.begin[c], o.row.begin() + o.begin[c + 1]);
        work[group_of[c]] += o.weight[c];
    }
    std::vector<std::vector<int>> own;  // per CTA
    std::vector<int> cta_of(nd), slot_of(nd);
    for (int g = 0; g < groups; g++) {
        long long acc = 0;
        const int base = (int)own.size();
        own.resize(base + cluster);
        for (int r : rows[g]) {
            const long long w = resident_weight(A, r);
            const int k = (int)std::min<long long>(cluster - 1, (2 * acc + w) * cluster / (2 * work[g]));
            own[base + k].push_back(r);
            cta_of[r] = base + k;
            acc += w;
        }
    }
    auto len = [&](int r) { return A.start[r + 1] - A.start[r]; };
    for (auto& v : own) {
        // by length, so that the rows of a slice are about equally long, then by row
        std::sort(v.begin(), v.end(), [&](int a, int b) { return len(a) != len(b) ? len(a) > len(b) : a < b; });
        for (size_t k = 0; k < v.size(); k++) slot_of[v[k]] = (int)k;
        p.max_own = std::max(p.max_own, (int)v.size());
    }
    p.cluster = cluster;
    p.groups = groups;
    p.tp = 1;
    while (p.tp * 2 <= T && p.max_own * p.tp * 2 <= kResidentThreads) p.tp *= 2;
    p.q = T / p.tp;
    {
        // whole slices per warp: the fewest rounds, then the fewest warps that still need no more
        const int slices = std::max(1, (p.max_own * p.tp + 31) / 32), most = kResidentThreads / 32;
        const int rounds = (slices + most - 1) / most;
        p.threads = std::max(64, (slices + rounds - 1) / rounds * 32);
    }
    const int S = 32 / p.tp;  // rows per slice
    // halo rows of every CTA (by source CTA, then row) and the pushes that fill them
    std::vector<std::vector<int>> halo(own.size());
    std::vector<std::vector<std::pair<int, uint32_t>>> push(own.size());  // (own slot, target)
    std::vector<std::vector<std::pair<int, int>>> halo_slot(own.size());  // (row, slot), by row
    std::vector<int> mark(nd, -1);
    for (size_t c = 0; c < own.size(); c++) {
        auto& h = halo[c];
        for (int r : own[c])
            for (int k = A.start[r]; k < A.start[r + 1]; k++) {
                const int j = A.col[k];
                if (cta_of[j] != (int)c && mark[j] != (int)c) {
                    mark[j] = (int)c;
                    h.push_back(j);
                }
            }
        std::sort(h.begin(), h.end(), [&](int a, int b) {
            return cta_of[a] != cta_of[b] ? cta_of[a] < cta_of[b] : slot_of[a] < slot_of[b];
        });
        for (size_t k = 0; k < h.size(); k++) {
            const int slot = (int)(own[c].size() + k);
            halo_slot[c].push_back({h[k], slot});
            push[cta_of[h[k]]].push_back({slot_of[h[k]], (uint32_t)(c % cluster) << 16 | (uint32_t)slot});
        }
        std::sort(halo_slot[c].begin(), halo_slot[c].end());
        p.max_local = std::max(p.max_local, (int)(own[c].size() + h.size()));
    }
    if (p.max_local > 65535) return p;
    auto slot_in = [&](int c, int j) {
        if (cta_of[j] == c) return slot_of[j];
        return std::lower_bound(halo_slot[c].begin(), halo_slot[c].end(), std::make_pair(j, -1))->second;
    };
    auto align16 = [](size_t v) { return (v + 15) / 16 * 16; };
    for (size_t c = 0; c < own.size(); c++) {
        const int no = (int)own[c].size(), nh = (int)halo[c].size(), ns = (no + S - 1) / S;
        ResidentCta d = {};
        d.own = no;
        d.halo = nh;
        d.slices = ns;
        std::vector<int> sptr(ns + 1, 0);
        for (int s = 0; s < ns; s++) {
            int steps = 0;  // entries per thread: whole rounds of the T partial sums
            for (int k = s * S; k < std::min(no, (s + 1) * S); k++) steps = std::max(steps, (len(own[c][k]) + T - 1) / T * p.q);
            sptr[s + 1] = sptr[s] + (steps + 1) / 2;
        }
        auto& pl = push[c];
        std::stable_sort(pl.begin(), pl.end(), [](const std::pair<int, uint32_t>& a, const std::pair<int, uint32_t>& b) { return a.first < b.first; });
        if (pl.size() > 65535) return p;
        size_t off = align16(sizeof(float) * (size_t)no);
        d.off_grow = (int)off;
        off = align16(off + sizeof(int) * (size_t)(no + nh));
        d.off_pptr = (int)off;
        off = align16(off + sizeof(uint16_t) * (size_t)(no + 1));
        d.off_push = (int)off;
        off = align16(off + sizeof(uint32_t) * pl.size());
        d.off_sptr = (int)off;
        off = align16(off + sizeof(int) * (size_t)(ns + 1));
        d.off_val = (int)off;
        off = align16(off + 8ull * 32 * (size_t)sptr[ns]);
        d.off_col = (int)off;
        off = align16(off + 4ull * 32 * (size_t)sptr[ns]);
        d.bytes = (int)off;
        d.blob = (long long)p.blob.size();
        if (off > (size_t)1 << 20) return p;
        p.blob.resize(p.blob.size() + off, 0);
        unsigned char* b = p.blob.data() + d.blob;
        for (int k = 0; k < no; k++) ((float*)b)[k] = diag[own[c][k]];
        int* grow = (int*)(b + d.off_grow);
        for (int k = 0; k < no; k++) grow[k] = own[c][k];
        for (int k = 0; k < nh; k++) grow[no + k] = halo[c][k];
        uint16_t* pptr = (uint16_t*)(b + d.off_pptr);
        uint32_t* pu = (uint32_t*)(b + d.off_push);
        for (size_t k = 0; k < pl.size(); k++) {
            pptr[pl[k].first + 1]++;
            pu[k] = pl[k].second;
        }
        for (int k = 0; k < no; k++) pptr[k + 1] = (uint16_t)(pptr[k + 1] + pptr[k]);
        std::memcpy(b + d.off_sptr, sptr.data(), sizeof(int) * sptr.size());
        float* val = (float*)(b + d.off_val);
        uint16_t* col = (uint16_t*)(b + d.off_col);
        for (int s = 0; s < ns; s++)
            for (int lane = 0; lane < 32; lane++) {
                const int k = s * S + lane / p.tp, j = lane % p.tp;
                const int r = k < no ? own[c][k] : -1;
                for (int t = 0; t < 2 * (sptr[s + 1] - sptr[s]); t++) {
                    const size_t at = 2 * (32 * (size_t)(sptr[s] + t / 2) + lane) + t % 2;
                    const int e = t / p.q * T + j * p.q + t % p.q;  // entry of the row
                    if (r >= 0 && e < len(r)) {
                        val[at] = (float)A.val[A.start[r] + e];
                        col[at] = (uint16_t)slot_in((int)c, A.col[A.start[r] + e]);
                    } else {
                        col[at] = (uint16_t)(k < no ? k : 0);
                    }
                }
            }
        p.max_blob = std::max(p.max_blob, d.bytes);
        p.max_entries = std::max(p.max_entries, 64ll * sptr[ns]);
        p.cta.push_back(d);
    }
    p.ok = true;
    return p;
}

}  // namespace admm
