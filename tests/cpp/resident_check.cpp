// Checks of the resident global step's plan (parallel_admm_b200/csrc/resident.hpp), by doing in
// C++ what the kernels of resident.cuh do on the GPU, every index checked against its section:
//
//  1. every row is computed by exactly one CTA, every group holds whole components, and every
//     halo slot is filled by exactly one push per sweep;
//  2. sweeps over the plan give the same bits as sweeps over the sliced ELL in the lane order of
//     k_jacobi, for every T and for one to several groups and CTAs per cluster.
// Exit code 0 on success; a message on stderr and exit code 1 otherwise.
#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <random>

#include "resident.hpp"

using namespace admm;

#define CHECK(cond, ...)                  \
    do {                                  \
        if (!(cond)) {                    \
            std::fprintf(stderr, __VA_ARGS__); \
            std::fprintf(stderr, " (line %d)\n", __LINE__); \
            std::exit(1);                 \
        }                                 \
    } while (0)

struct V3 {
    float x, y, z;
};

static V3 add(V3 a, V3 b) { return {a.x + b.x, a.y + b.y, a.z + b.z}; }
static V3 fma3(float a, V3 q, V3 s) { return {std::fmaf(a, q.x, s.x), std::fmaf(a, q.y, s.y), std::fmaf(a, q.z, s.z)}; }

// Lattice blocks (each a component) with 27-point couplings, randomly thinned, plus lone rows.
static HostCsr blocks_csr(const std::vector<int>& edge, int lone, std::mt19937& rng, std::vector<float>& pos, std::vector<float>& diag) {
    std::vector<std::vector<std::pair<int, double>>> rows;
    std::uniform_real_distribution<double> u(-1.0, 1.0);
    float shift = 0.f;
    for (int n : edge) {
        const int base = (int)rows.size();
        auto at = [&](int i, int j, int k) { return base + (i * n + j) * n + k; };
        rows.resize(base + n * n * n);
        for (int i = 0; i < n; i++)
            for (int j = 0; j < n; j++)
                for (int k = 0; k < n; k++) {
                    for (float c : {shift + i, (float)j, (float)k}) pos.push_back(c);
                    for (int a = -1; a <= 1; a++)
                        for (int b = -1; b <= 1; b++)
                            for (int c = -1; c <= 1; c++) {
                                const int x = i + a, y = j + b, z = k + c;
                                if (x < 0 || y < 0 || z < 0 || x >= n || y >= n || z >= n) continue;
                                const int p = at(i, j, k), q = at(x, y, z);
                                // keep the axis neighbours (connected), thin the others
                                if (p < q && (std::abs(a) + std::abs(b) + std::abs(c) == 1 || rng() % 3 == 0)) {
                                    const double v = u(rng);
                                    rows[p].push_back({q, v});
                                    rows[q].push_back({p, v});
                                }
                            }
                }
        shift += n + 2;
    }
    for (int k = 0; k < lone; k++) {
        rows.emplace_back();
        for (float c : {shift + k, 0.f, 0.f}) pos.push_back(c);
    }
    HostCsr c;
    c.start.push_back(0);
    for (auto& r : rows) {
        std::sort(r.begin(), r.end());
        for (auto& e : r) {
            c.col.push_back(e.first);
            c.val.push_back(e.second);
        }
        c.start.push_back((int)c.col.size());
    }
    diag.resize(rows.size());
    for (auto& d : diag) d = 20.f + (float)u(rng);
    return c;
}

static std::vector<V3> sweep_ell(const HostEll& e, const std::vector<float>& diag, const std::vector<V3>& b, const std::vector<V3>& x) {
    const int T = e.lanes, S = 32 / T;
    std::vector<V3> out(x.size());
    for (int w = 0; w < e.nslices; w++)
        for (int lr = 0; lr < S; lr++) {
            const int r = e.rowid[w * S + lr];
            if (r >= e.rows) continue;
            std::vector<V3> p(T, V3{0.f, 0.f, 0.f});
            for (int j = 0; j < T; j++)
                for (int k = e.ptr[w] + j * S + lr; k < e.ptr[w + 1]; k += 32) p[j] = fma3(e.val[k], x[e.col[k]], p[j]);
            for (int o = 1; o < T; o <<= 1)
                for (int j = 0; j < T; j += 2 * o) p[j] = add(p[j], p[j + o]);
            out[r] = {(b[r].x - p[0].x) / diag[r], (b[r].y - p[0].y) / diag[r], (b[r].z - p[0].z) / diag[r]};
        }
    return out;
}

static std::vector<V3> sweeps_plan(const HostResident& p, int nd, const std::vector<V3>& b, const std::vector<V3>& x0, int sweeps) {
    const int nc = (int)p.cta.size(), S = 32 / p.tp;
    const float nan = std::nanf("");
    std::vector<std::vector<V3>> cur(nc), nxt(nc);
    std::vector<V3> out(nd, V3{nan, nan, nan});
    std::vector<int> seen(nd, 0);
    for (int c = 0; c < nc; c++) {
        const ResidentCta& d = p.cta[c];
        CHECK(d.bytes <= p.max_blob && d.bytes % 16 == 0 && d.blob % 16 == 0 && d.blob + d.bytes <= (long long)p.blob.size(), "blob of CTA %d", c);
        CHECK(d.own <= p.max_own && d.own + d.halo <= p.max_local && (d.own + S - 1) / S == d.slices, "rows of CTA %d", c);
        CHECK((size_t)d.off_grow >= sizeof(float) * d.own && (size_t)d.off_pptr >= d.off_grow + 4u * (d.own + d.halo) &&
                  (size_t)d.off_push >= d.off_pptr + 2u * (d.own + 1) && d.off_col % 16 == 0 && d.off_val % 16 == 0, "sections of CTA %d", c);
        const int* grow = (const int*)(p.blob.data() + d.blob + d.off_grow);
        for (int k = 0; k < d.own + d.halo; k++) CHECK(grow[k] >= 0 && grow[k] < nd, "row of slot %d", k);
        for (int k = 0; k < d.own; k++) CHECK(seen[grow[k]]++ == 0, "row %d twice", grow[k]);
        for (int k = 0; k < d.own + d.halo; k++) cur[c].push_back(x0[grow[k]]);
    }
    for (int r = 0; r < nd; r++) CHECK(seen[r] == 1, "row %d in no CTA", r);
    for (int it = 0; it < sweeps; it++) {
        for (int c = 0; c < nc; c++) nxt[c].assign(cur[c].size(), V3{nan, nan, nan});
        std::vector<std::vector<int>> filled(nc);
        for (int c = 0; c < nc; c++) filled[c].assign(cur[c].size(), 0);
        for (int c = 0; c < nc; c++) {
            const ResidentCta& d = p.cta[c];
            const unsigned char* bl = p.blob.data() + d.blob;
            const float* diag = (const float*)bl;
            const int *grow = (const int*)(bl + d.off_grow), *sptr = (const int*)(bl + d.off_sptr);
            const uint16_t *pptr = (const uint16_t*)(bl + d.off_pptr), *col = (const uint16_t*)(bl + d.off_col);
            const uint32_t* push = (const uint32_t*)(bl + d.off_push);
            const float* val = (const float*)(bl + d.off_val);
            CHECK(d.off_push + 4ll * pptr[d.own] <= d.off_sptr, "pushes of CTA %d", c);
            CHECK(d.off_val + 256ll * sptr[d.slices] <= d.off_col && d.off_col + 128ll * sptr[d.slices] <= d.bytes, "entries of CTA %d", c);
            for (int s = 0; s < d.slices; s++)
                for (int rl = 0; rl < S; rl++) {
                    const int r = s * S + rl;
                    std::vector<V3> part(p.tp * p.q, V3{0.f, 0.f, 0.f});
                    for (int j = 0; j < p.tp; j++)
                        for (int t = 0; t < 2 * (sptr[s + 1] - sptr[s]); t++) {
                            const size_t at = 2 * (32 * (size_t)(sptr[s] + t / 2) + rl * p.tp + j) + t % 2;
                            CHECK(col[at] < cur[c].size() || d.own == 0, "slot %d of CTA %d", col[at], c);
                            V3& q = part[j * p.q + t % p.q];
                            q = fma3(val[at], cur[c][col[at]], q);
                        }
                    if (r >= d.own) continue;
                    const int T = p.tp * p.q;
                    for (int o = 1; o < T; o <<= 1)
                        for (int j = 0; j < T; j += 2 * o) part[j] = add(part[j], part[j + o]);
                    const int g = grow[r];
                    const V3 v = {(b[g].x - part[0].x) / diag[r], (b[g].y - part[0].y) / diag[r], (b[g].z - part[0].z) / diag[r]};
                    nxt[c][r] = v;
                    filled[c][r]++;
                    out[g] = v;
                    for (int k = pptr[r]; k < pptr[r + 1]; k++) {
                        const int to = c / p.cluster * p.cluster + (int)(push[k] >> 16), slot = (int)(push[k] & 0xffffu);
                        CHECK((int)(push[k] >> 16) < p.cluster && slot >= p.cta[to].own && slot < p.cta[to].own + p.cta[to].halo, "push of CTA %d", c);
                        CHECK(((const int*)(p.blob.data() + p.cta[to].blob + p.cta[to].off_grow))[slot] == g, "push to another row's slot");
                        nxt[to][slot] = v;
                        filled[to][slot]++;
                    }
                }
        }
        for (int c = 0; c < nc; c++)
            for (size_t k = 0; k < filled[c].size(); k++) CHECK(filled[c][k] == 1, "slot %zu of CTA %d filled %d times", k, c, filled[c][k]);
        cur.swap(nxt);
    }
    return out;
}

int main() {
    std::mt19937 rng(3);
    std::uniform_real_distribution<float> u(-1.f, 1.f);
    const std::vector<std::vector<int>> scenes = {{1}, {2}, {9}, {3, 5, 2, 4, 7}, {12}, {2, 2, 2, 2, 2, 2}};
    int checked = 0;
    for (const auto& sc : scenes)
        for (int T : {1, 2, 4, 8})
            for (int cluster : {1, 2, 8, 16})
                for (int groups : {1, 3}) {
                    std::vector<float> pos, diag;
                    const HostCsr A = blocks_csr(sc, checked % 3, rng, pos, diag);
                    const int nd = (int)diag.size();
                    const ResidentOrder o = resident_order(A, nd, pos.data(), 3);
                    const int g = std::min(groups, (int)o.weight.size());
                    const HostResident p = build_resident(A, diag, nd, T, o, cluster, g);
                    CHECK(p.ok && p.tp * p.q == T && p.threads % 32 == 0 && p.threads <= kResidentThreads, "plan");
                    CHECK((int)p.cta.size() == g * cluster, "CTAs");
                    std::vector<V3> b(nd), x(nd);
                    for (auto& v : b) v = {u(rng), u(rng), u(rng)};
                    for (auto& v : x) v = {u(rng), u(rng), u(rng)};
                    const HostEll e = csr_to_sliced_ell(A, nd, T, true);
                    std::vector<V3> want = x;
                    for (int k = 0; k < 3; k++) want = sweep_ell(e, diag, b, want);
                    const std::vector<V3> got = sweeps_plan(p, nd, b, x, 3);
                    CHECK(std::memcmp(want.data(), got.data(), sizeof(V3) * nd) == 0, "bits (T %d, cluster %d, groups %d)", T, cluster, g);
                    checked++;
                }
    std::printf("%d plans ok\n", checked);
    return 0;
}
