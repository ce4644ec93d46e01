// Host-side validation, colouring and partition plan (see plan.h).
#include "plan.h"

#include <algorithm>
#include <atomic>
#include <cmath>
#include <cstring>
#include <new>
#include <numeric>
#include <thread>

namespace pg {

// Every value finite: the exponent bits of a NaN or infinity are all ones (no
// early exit, so the loop vectorises).
bool finite_f(const float* a, size_t n) {
    uint32_t bad = 0;
    for (size_t i = 0; i < n; i++) {
        uint32_t u;
        std::memcpy(&u, a + i, sizeof u);
        bad |= (u & 0x7f800000u) == 0x7f800000u;
    }
    return bad == 0;
}

std::string validate_header(const pg_problem& p, bool need_rhs) {
    if (p.nodes_per_element != 3 && p.nodes_per_element != 4)
        return "nodes_per_element must be 3 (DKT) or 4 (Q4)";
    if (p.node_count > (1u << 26) || p.element_count > (1u << 26))
        return "problem too large (node_count and element_count must be < 2^26)";
    if (p.node_count > 0 && !p.nodes) return "nodes is NULL";
    if (p.element_count > 0 && !p.elements) return "elements is NULL";
    if (p.node_count > 0 && !p.constrained) return "constrained is NULL";
    if (need_rhs && p.node_count > 0 && !p.F) return "F is NULL";
    if (!std::isfinite(p.E) || !std::isfinite(p.nu) || !std::isfinite(p.t))
        return "material E, nu, t must be finite";
    if (p.color_count > 0 && (!p.color_offsets || !p.elements_by_color)) return "colouring arrays are NULL";
    if (p.color_count > 0 && (p.color_offsets[0] != 0 || p.color_offsets[p.color_count] != p.element_count))
        return "color_offsets must start at 0 and end at element_count";
    return "";
}

std::string validate_problem(const pg_problem& p, bool need_rhs) {
    std::string e = validate_header(p, need_rhs);
    if (!e.empty()) return e;
    if (p.node_count && !finite_f(p.nodes, 2 * (size_t)p.node_count))
        return "node coordinates must be finite";
    if (p.elem_t && p.element_count && !finite_f(p.elem_t, p.element_count))
        return "elem_t must be finite";
    const size_t ne = (size_t)p.element_count * p.nodes_per_element;
    uint32_t top = 0;
    for (size_t i = 0; i < ne; i++) top = std::max(top, p.elements[i]);
    if (ne && top >= p.node_count) return "element node index out of range";
    if (p.color_count > 0) {
        for (uint32_t c = 0; c < p.color_count; c++)
            if (p.color_offsets[c + 1] < p.color_offsets[c]) return "color_offsets must not decrease";
        std::vector<uint8_t> seen(p.element_count, 0);
        for (uint32_t i = 0; i < p.element_count; i++) {
            uint32_t e = p.elements_by_color[i];
            if (e >= p.element_count || seen[e]) return "elements_by_color must list every element once";
            seen[e] = 1;
        }
    }
    return "";
}

std::string build_structure(const pg_problem& p, HostPlan& plan) {
    const int Nn = (int)p.node_count, Ne = (int)p.element_count, npe = (int)p.nodes_per_element;
    plan.Nn = Nn;
    plan.Ne = Ne;
    plan.npe = npe;
    // node -> incident (element, position), element ids ascending
    plan.inc_ptr.assign(Nn + 1, 0);
    for (int e = 0; e < Ne; e++)
        for (int k = 0; k < npe; k++) plan.inc_ptr[p.elements[(size_t)e * npe + k] + 1]++;
    for (int n = 0; n < Nn; n++) plan.inc_ptr[n + 1] += plan.inc_ptr[n];
    plan.inc_idx.assign(plan.inc_ptr[Nn], 0);
    {
        std::vector<int> fill(plan.inc_ptr.begin(), plan.inc_ptr.end() - 1);
        for (int e = 0; e < Ne; e++)
            for (int k = 0; k < npe; k++)
                plan.inc_idx[fill[p.elements[(size_t)e * npe + k]]++] = e * 4 + k;
    }
    // colour of every element from the caller's lists
    std::vector<int> color(Ne, -1);
    bool valid = p.color_count > 0;
    if (valid) {
        for (uint32_t c = 0; c < p.color_count; c++)
            for (uint32_t q = p.color_offsets[c]; q < p.color_offsets[c + 1]; q++)
                color[p.elements_by_color[q]] = (int)c;
        // conflict check (verifyColoring, coloring.ts:188-225)
        std::vector<int> stamp(std::max<int>(p.color_count, 1), -1);
        for (int n = 0; n < Nn && valid; n++) {
            for (int q = plan.inc_ptr[n]; q < plan.inc_ptr[n + 1]; q++) {
                int c = color[plan.inc_idx[q] / 4];
                if (stamp[c] == n) { valid = false; break; }
                stamp[c] = n;
            }
        }
    }
    if (!valid && Ne > 0) {
        // greedy first-fit colouring in element order (coloring.ts:92-177)
        plan.recolored = p.color_count > 0;
        std::fill(color.begin(), color.end(), -1);
        std::vector<int> used(64, -1);
        for (int e = 0; e < Ne; e++) {
            for (int k = 0; k < npe; k++) {
                int n = (int)p.elements[(size_t)e * npe + k];
                for (int q = plan.inc_ptr[n]; q < plan.inc_ptr[n + 1]; q++) {
                    int nb = plan.inc_idx[q] / 4;
                    if (nb != e && color[nb] >= 0) {
                        if (color[nb] >= (int)used.size()) used.resize(color[nb] * 2 + 2, -1);
                        used[color[nb]] = e;
                    }
                }
            }
            int c = 0;
            while (c < (int)used.size() && used[c] == e) c++;
            color[e] = c;
        }
    }
    int C = 1;
    for (int e = 0; e < Ne; e++) C = std::max(C, color[e] + 1);
    plan.colors = C;
    plan.color_offsets.assign(C + 1, 0);
    for (int e = 0; e < Ne; e++) plan.color_offsets[color[e] + 1]++;
    for (int c = 0; c < C; c++) plan.color_offsets[c + 1] += plan.color_offsets[c];
    plan.elements_by_color.assign(Ne, 0);
    {
        std::vector<uint32_t> fill(plan.color_offsets.begin(), plan.color_offsets.end() - 1);
        if (valid) {
            for (uint32_t c = 0; c < p.color_count; c++)
                for (uint32_t q = p.color_offsets[c]; q < p.color_offsets[c + 1]; q++)
                    plan.elements_by_color[fill[c]++] = p.elements_by_color[q];
        } else {
            for (int e = 0; e < Ne; e++) plan.elements_by_color[fill[color[e]]++] = (uint32_t)e;
        }
    }
    return "";
}

namespace {

// Order-preserving map of a finite float to an unsigned key (-0 as +0, so
// keys compare as the values do).
inline uint32_t float_key(float v) {
    if (v == 0.0f) v = 0.0f;
    uint32_t u;
    std::memcpy(&u, &v, sizeof u);
    return (u & 0x80000000u) ? ~u : (u | 0x80000000u);
}

struct SortKey {
    uint64_t k;  // primary coordinate key << 32 | secondary coordinate key
    int id;
};

// Stable sort of v[b, e) by k: equal keys keep their incoming order.  Merges
// the ascending runs it finds, so meshes numbered row by row, whose nodes
// arrive sorted by (y, x) and whose strips are then a few sorted rows, cost one
// pass and a few merges (60k-DOF plate: 0.9 -> 0.25 ms for all strips); a
// shuffled mesh costs what std::stable_sort does.
void sort_keys(std::vector<SortKey>& v, size_t b, size_t e) {
    auto less = [](const SortKey& u, const SortKey& w) { return u.k < w.k; };
    std::vector<size_t> run{b};
    for (size_t i = b + 1; i < e; i++)
        if (v[i].k < v[i - 1].k) run.push_back(i);
    if (run.size() == 1) return;
    if (run.size() > (e - b) / 8 + 1) {  // short runs: nothing to gain
        std::stable_sort(v.begin() + b, v.begin() + e, less);
        return;
    }
    run.push_back(e);
    std::vector<SortKey> tmp(e - b);
    SortKey* src = v.data() + b;
    SortKey* dst = tmp.data();
    while (run.size() > 2) {
        std::vector<size_t> next{b};
        for (size_t r = 0; r + 1 < run.size(); r += 2) {
            const size_t lo = run[r] - b, mid = run[r + 1] - b, hi = (r + 2 < run.size() ? run[r + 2] : run[r + 1]) - b;
            std::merge(src + lo, src + mid, src + mid, src + hi, dst + lo, less);
            next.push_back(hi + b);
        }
        run.swap(next);
        std::swap(src, dst);
    }
    if (src != v.data() + b) std::copy(src, src + (e - b), v.begin() + b);
}

}  // namespace

// Near-square partition of a node cloud into G parts (see plan.h).
void strip_partition(const float* xy, int Nn, int G, std::vector<int>& part_of) {
    part_of.assign(Nn, 0);
    if (G <= 1 || Nn == 0) return;
    float lo[2] = {INFINITY, INFINITY}, hi[2] = {-INFINITY, -INFINITY};
    for (int n = 0; n < Nn; n++)
        for (int d = 0; d < 2; d++) {
            lo[d] = std::min(lo[d], xy[2 * n + d]);
            hi[d] = std::max(hi[d], xy[2 * n + d]);
        }
    const double W = std::max(1e-30, (double)hi[0] - lo[0]), H = std::max(1e-30, (double)hi[1] - lo[1]);
    int R = (int)std::lround(std::sqrt((double)G * H / W));
    R = std::max(1, std::min(R, G));
    // first by (y, x, id), then each strip by (x, y, id): stable sorts of the
    // packed coordinate keys, the ids entering in increasing order (and a
    // strip's equal (x, y) pairs keep the id order of the first sort)
    std::vector<SortKey> keys(Nn);
    std::vector<uint32_t> kx(Nn), ky(Nn);
    for (int n = 0; n < Nn; n++) {
        kx[n] = float_key(xy[2 * n]);
        ky[n] = float_key(xy[2 * n + 1]);
        keys[n] = SortKey{(uint64_t)ky[n] << 32 | kx[n], n};
    }
    sort_keys(keys, 0, (size_t)Nn);
    int part = 0;
    long long done_blocks = 0;
    int start = 0;
    for (int s = 0; s < R; s++) {
        const int blocks = G / R + (s < G % R ? 1 : 0);
        done_blocks += blocks;
        const int end = (int)((long long)Nn * done_blocks / G);
        for (int i = start; i < end; i++) {
            const int n = keys[i].id;
            keys[i].k = (uint64_t)kx[n] << 32 | ky[n];
        }
        sort_keys(keys, (size_t)start, (size_t)end);
        const int len = end - start;
        for (int b = 0; b < blocks; b++) {
            const int b0 = start + (int)((long long)len * b / blocks);
            const int b1 = start + (int)((long long)len * (b + 1) / blocks);
            for (int i = b0; i < b1; i++) part_of[keys[i].id] = part;
            part++;
        }
        start = end;
    }
}

std::string build_partition(const pg_problem& p, int G, int rings, HostPlan& plan, bool with_tasks) {
    const int Nn = plan.Nn, npe = plan.npe;
    if (G < 1) G = 1;
    if (G > std::max(Nn, 1)) G = std::max(Nn, 1);
    plan.G = G;
    plan.rings = rings == 2 ? 2 : 1;
    std::vector<int> part_of;
    strip_partition(p.nodes, Nn, G, part_of);

    std::vector<std::vector<int>> owned(G);
    for (int n = 0; n < Nn; n++) owned[part_of[n]].push_back(n);

    plan.node_off.assign(G + 1, 0);
    plan.nown.assign(G, 0);
    plan.task_off.assign(G + 1, 0);
    plan.tp_off.assign(G + 1, 0);
    plan.nodes.clear();
    plan.task_elem.clear();
    plan.task_pos.clear();
    plan.task_nodes.clear();
    plan.tptr.clear();
    plan.n1.assign(G, 0);
    plan.max_nloc = plan.max_nown = plan.max_ntask = plan.max_n1 = 0;

    // Each part's lists are built independently (host threads over parts,
    // each with its own node -> local-index map), then concatenated in part
    // order.
    struct PartOut {
        std::vector<int> nodes, tptr, task_elem;
        std::vector<int> steps;  // q-steps of each group of 10 rows
        std::vector<uint8_t> task_pos;
        std::vector<uint16_t> task_nodes;
        int nown = 0, n1 = 0, nloc = 0, ntask = 0;
        bool too_large = false;
    };
    std::vector<PartOut> out(G);
    const bool two = rings == 2;
    auto build_part = [&](int g, std::vector<int>& local, std::vector<int>& ghosts, std::vector<int>& ring2,
                          std::vector<int>& stamp, int& row_id) {
        // fills `dst` (sorted) with the nodes of elements around `from` not yet numbered
        auto next_ring = [&](const std::vector<int>& from, std::vector<int>& dst) {
            dst.clear();
            for (int n : from)
                for (int q = plan.inc_ptr[n]; q < plan.inc_ptr[n + 1]; q++) {
                    const int e = plan.inc_idx[q] / 4;
                    for (int k = 0; k < npe; k++) {
                        const int m = (int)p.elements[(size_t)e * npe + k];
                        if (local[m] == -1) { local[m] = -2; dst.push_back(m); }
                    }
                }
            std::sort(dst.begin(), dst.end());
        };
        PartOut& o = out[g];
        const std::vector<int>& own = owned[g];
        for (size_t i = 0; i < own.size(); i++) local[own[i]] = (int)i;
        next_ring(own, ghosts);
        for (size_t i = 0; i < ghosts.size(); i++) local[ghosts[i]] = (int)(own.size() + i);
        ring2.clear();
        if (two) {
            next_ring(ghosts, ring2);
            for (size_t i = 0; i < ring2.size(); i++) local[ring2[i]] = (int)(own.size() + ghosts.size() + i);
        }
        o.nloc = (int)(own.size() + ghosts.size() + ring2.size());
        o.nown = (int)own.size();
        o.n1 = two ? (int)(own.size() + ghosts.size()) : (int)own.size();
        o.too_large = o.nloc > 65535;
        if (!o.too_large) {
            o.nodes.reserve(o.nloc);
            o.nodes.insert(o.nodes.end(), own.begin(), own.end());
            o.nodes.insert(o.nodes.end(), ghosts.begin(), ghosts.end());
            o.nodes.insert(o.nodes.end(), ring2.begin(), ring2.end());
            const int ntn = o.n1;
            for (int i = 0; i < ntn; i++) o.ntask += plan.inc_ptr[o.nodes[i] + 1] - plan.inc_ptr[o.nodes[i]];
            if (with_tasks) {
                for (int i = 0; i < ntn; i++) {
                    const int n = o.nodes[i];
                    o.tptr.push_back((int)o.task_elem.size());
                    for (int q = plan.inc_ptr[n]; q < plan.inc_ptr[n + 1]; q++) {
                        const int e = plan.inc_idx[q] / 4, k = plan.inc_idx[q] % 4;
                        o.task_elem.push_back(e);
                        o.task_pos.push_back((uint8_t)k);
                        for (int j = 0; j < npe; j++)
                            o.task_nodes.push_back((uint16_t)local[p.elements[(size_t)e * npe + (k + j) % npe]]);
                    }
                }
                o.tptr.push_back((int)o.task_elem.size());
            }
            // slots of each row: the distinct nodes of its elements
            o.steps.assign((ntn + 9) / 10, 0);
            for (int i = 0; i < ntn; i++, row_id++) {
                const int n = o.nodes[i];
                int slots = 0;
                for (int q = plan.inc_ptr[n]; q < plan.inc_ptr[n + 1]; q++) {
                    const uint32_t* en = p.elements + (size_t)(plan.inc_idx[q] / 4) * npe;
                    for (int k = 0; k < npe; k++)
                        if (stamp[en[k]] != row_id) {
                            stamp[en[k]] = row_id;
                            slots++;
                        }
                }
                o.steps[i / 10] = std::max(o.steps[i / 10], (slots + 2) / 3);
            }
        }
        for (int n : own) local[n] = -1;
        for (int n : ghosts) local[n] = -1;
        for (int n : ring2) local[n] = -1;
    };
    const int nth = std::max(1, std::min({(int)std::thread::hardware_concurrency(), 16, G, 1 + Nn / 4096}));
    std::atomic<int> next{0};
    std::atomic<bool> failed{false};
    auto worker = [&]() {
        // an exception must not leave a worker thread (std::terminate):
        // recorded here, raised again on the calling thread
        try {
            std::vector<int> local(Nn, -1), ghosts, ring2, stamp(Nn, -1);
            int row_id = 0;
            for (int g; !failed && (g = next.fetch_add(1)) < G;) build_part(g, local, ghosts, ring2, stamp, row_id);
        } catch (...) {
            failed = true;
        }
    };
    {
        std::vector<std::thread> th;
        for (int t = 1; t < nth; t++) th.emplace_back(worker);
        worker();
        for (auto& t : th) t.join();
    }
    if (failed) throw std::bad_alloc();
    size_t tot_nodes = 0, tot_tasks = 0, tot_tptr = 0;
    for (int g = 0; g < G; g++) {
        if (out[g].too_large) return "a part has more than 65535 local nodes: use more ctas";
        tot_nodes += out[g].nodes.size();
        tot_tasks += out[g].task_elem.size();
        tot_tptr += out[g].tptr.size();
    }
    plan.nodes.reserve(tot_nodes);
    plan.task_elem.reserve(tot_tasks);
    plan.task_pos.reserve(tot_tasks);
    plan.task_nodes.reserve(tot_tasks * npe);
    plan.tptr.reserve(tot_tptr);
    for (int g = 0; g < G; g++) {
        const PartOut& o = out[g];
        plan.nown[g] = o.nown;
        plan.n1[g] = o.n1;
        plan.nodes.insert(plan.nodes.end(), o.nodes.begin(), o.nodes.end());
        plan.node_off[g + 1] = (int)plan.nodes.size();
        plan.tp_off[g] = (int)plan.tptr.size();
        plan.tptr.insert(plan.tptr.end(), o.tptr.begin(), o.tptr.end());
        plan.task_elem.insert(plan.task_elem.end(), o.task_elem.begin(), o.task_elem.end());
        plan.task_pos.insert(plan.task_pos.end(), o.task_pos.begin(), o.task_pos.end());
        plan.task_nodes.insert(plan.task_nodes.end(), o.task_nodes.begin(), o.task_nodes.end());
        plan.task_off[g + 1] = (int)plan.task_elem.size();
        plan.max_nloc = std::max(plan.max_nloc, o.nloc);
        plan.max_nown = std::max(plan.max_nown, o.nown);
        plan.max_n1 = std::max(plan.max_n1, o.n1);
        plan.max_ntask = std::max(plan.max_ntask, o.ntask);
    }
    plan.tp_off[G] = (int)plan.tptr.size();
    plan.grp_off.assign(1, 0);
    plan.grp_q.assign(1, 0);
    for (int g = 0; g < G; g++) {
        for (int w : out[g].steps) plan.grp_q.push_back(plan.grp_q.back() + w);
        plan.grp_off.push_back((int)plan.grp_q.size() - 1);
    }
    return "";
}

std::string build_coarse_meta(const pg_problem& p, HostPlan& plan) {
    const int G = plan.G, Nn = plan.Nn;
    const int C = 3 * G;
    plan.C = C;
    plan.coarse_owner.assign(Nn, 0);
    plan.coarse_geom.assign(3 * (size_t)G, 0.0);
    std::vector<int>& owner = plan.coarse_owner;
    for (int g = 0; g < G; g++) {
        const int n0 = plan.node_off[g], no = plan.nown[g];
        double sx = 0, sy = 0, lo[2] = {INFINITY, INFINITY}, hi[2] = {-INFINITY, -INFINITY};
        for (int k = 0; k < no; k++) {
            const int n = plan.nodes[n0 + k];
            owner[n] = g;
            const double x = p.nodes[2 * n], y = p.nodes[2 * n + 1];
            sx += x;
            sy += y;
            lo[0] = std::min(lo[0], x); hi[0] = std::max(hi[0], x);
            lo[1] = std::min(lo[1], y); hi[1] = std::max(hi[1], y);
        }
        double cx = 0, cy = 0, ih = 1.0;
        if (no > 0) {
            cx = sx / no;
            cy = sy / no;
            const double h = std::max(hi[0] - lo[0], hi[1] - lo[1]);
            ih = h > 0 ? 1.0 / h : 1.0;
        }
        plan.coarse_geom[3 * g] = cx;
        plan.coarse_geom[3 * g + 1] = cy;
        plan.coarse_geom[3 * g + 2] = ih;
    }
    // per part: aggregates of its local nodes, node slots and basis data
    plan.node_basis.assign(3 * plan.nodes.size(), 0.0);
    plan.node_slot.assign(plan.nodes.size(), 0);
    plan.cagg_off.assign(G + 1, 0);
    plan.cagg.clear();
    plan.ainv_off.assign(G + 1, 0);
    plan.ainv_src.clear();
    plan.max_kagg = 0;
    std::vector<int> slot_of(G, -1);
    for (int g = 0; g < G; g++) {
        // aggregates of the nodes where the part forms u: owned and ring 1
        // (ring-2 nodes, rings = 2, carry only r, s and w: slot 0, unused)
        const int n0 = plan.node_off[g], nl = plan.node_off[g + 1] - n0;
        const int nu = plan.rings == 2 ? plan.n1[g] : nl;
        std::vector<int> list = {g};
        slot_of[g] = 0;
        for (int k = 0; k < nu; k++) {
            const int a = owner[plan.nodes[n0 + k]];
            if (slot_of[a] < 0) { slot_of[a] = (int)list.size(); list.push_back(a); }
        }
        for (int k = 0; k < nl; k++) {
            const int n = plan.nodes[n0 + k], a = owner[n];
            const double* ge = plan.coarse_geom.data() + 3 * a;
            plan.node_slot[n0 + k] = k < nu ? slot_of[a] : 0;
            plan.node_basis[3 * (n0 + k)] = (p.nodes[2 * n] - ge[0]) * ge[2];
            plan.node_basis[3 * (n0 + k) + 1] = (p.nodes[2 * n + 1] - ge[1]) * ge[2];
            plan.node_basis[3 * (n0 + k) + 2] = ge[2];
        }
        plan.ainv_off[g] = (int)plan.ainv_src.size();
        for (int a : list)
            for (int m = 0; m < 3; m++) plan.ainv_src.push_back(3 * a + m);
        plan.cagg.insert(plan.cagg.end(), list.begin(), list.end());
        plan.cagg_off[g + 1] = (int)plan.cagg.size();
        plan.max_kagg = std::max(plan.max_kagg, (int)list.size());
        for (int a : list) slot_of[a] = -1;
    }
    plan.ainv_off[G] = (int)plan.ainv_src.size();
    return "";
}

std::string schedule_batch(const std::vector<int>& nodes, const std::vector<int>& caps, int sms, BatchSchedule& out,
                           int part_nodes) {
    const double target = part_nodes;
    out = BatchSchedule{};
    const int count = (int)nodes.size();
    if (count == 0) return "empty batch";
    if (sms < 1 || (int)caps.size() != count) return "no blocks to schedule";
    int top = 1;  // largest power of two <= sms
    while (top * 2 <= sms) top *= 2;
    std::vector<int> d(count);
    std::vector<double> w(count);
    for (int i = 0; i < count; i++) {
        const double n = std::max(1, nodes[i]);
        const int cap = std::max(1, caps[i]);
        int need = 1;
        while (need < std::ceil(n / cap)) need *= 2;
        if (need > top) {
            if ((double)sms * cap < n) return "a plate of the batch needs more blocks than the device has";
            need = sms;
        }
        const int pref = std::max(1, (int)std::lround(std::exp2(std::round(std::log2(std::max(1.0, n / target))))));
        d[i] = std::max(need, std::min(top, pref));
        w[i] = std::sqrt(n) * (n + 300.0 * d[i]);
    }
    out.plate_phase.assign(count, -1);
    out.plate_team.assign(count, -1);
    out.plate_size = d;
    std::vector<int> order(count);
    std::iota(order.begin(), order.end(), 0);
    std::stable_sort(order.begin(), order.end(), [&](int a, int b) { return w[a] > w[b]; });
    // team sizes, largest first, first-fit into phases (one team of each size
    // fits)
    std::vector<int> cs;
    for (int i = 0; i < count; i++)
        if (std::find(cs.begin(), cs.end(), d[i]) == cs.end()) cs.push_back(d[i]);
    std::sort(cs.rbegin(), cs.rend());
    std::vector<std::vector<int>> phase_sizes;
    std::vector<int> phase_sum;
    for (int c : cs) {
        size_t ph = 0;
        while (ph < phase_sizes.size() && phase_sum[ph] + c > sms) ph++;
        if (ph == phase_sizes.size()) {
            phase_sizes.emplace_back();
            phase_sum.push_back(0);
        }
        phase_sizes[ph].push_back(c);
        phase_sum[ph] += c;
    }
    for (size_t ph = 0; ph < phase_sizes.size(); ph++) {
        const std::vector<int>& pc = phase_sizes[ph];  // descending
        const int nc = (int)pc.size();
        std::vector<double> W(nc, 0.0);
        std::vector<int> teams(nc, 1), nplates(nc, 0);
        for (int i = 0; i < count; i++) {
            const auto it = std::find(pc.begin(), pc.end(), d[i]);
            if (it == pc.end()) continue;
            W[it - pc.begin()] += w[i];
            nplates[it - pc.begin()]++;
        }
        int used = phase_sum[ph];
        for (;;) {  // one more team to the size with the most work per block
            int best = -1;
            double bw = 0.0;
            for (int k = 0; k < nc; k++) {
                if (used + pc[k] > sms || teams[k] >= nplates[k]) continue;
                const double per = W[k] / ((double)teams[k] * pc[k]);
                if (per > bw) { bw = per; best = k; }
            }
            if (best < 0) break;
            teams[best]++;
            used += pc[best];
        }
        BatchPhase P;
        for (int k = 0; k < nc; k++)
            for (int t = 0; t < teams[k]; t++) {
                P.team_base.push_back(P.grid);
                P.team_size.push_back(pc[k]);
                P.grid += pc[k];
            }
        const int T = (int)P.team_size.size();
        P.team_load.assign(T, 0.0);
        std::vector<std::vector<int>> q(T);
        for (int i : order) {
            if (std::find(pc.begin(), pc.end(), d[i]) == pc.end()) continue;
            int bt = -1;
            for (int t = 0; t < T; t++)
                if (P.team_size[t] == d[i] && (bt < 0 || P.team_load[t] < P.team_load[bt])) bt = t;
            out.plate_phase[i] = (int)out.phases.size();
            out.plate_team[i] = bt;
            P.team_load[bt] += w[i];
            q[bt].push_back(i);
        }
        P.queue_off.assign(T + 1, 0);
        for (int t = 0; t < T; t++) {
            P.queue_off[t + 1] = P.queue_off[t] + (int)q[t].size();
            P.queue.insert(P.queue.end(), q[t].begin(), q[t].end());
        }
        // the dynamic queues: one per class (team size), largest work first
        std::vector<std::vector<int>> cq(nc);
        for (int i : order) {
            const auto it = std::find(pc.begin(), pc.end(), d[i]);
            if (it != pc.end()) cq[it - pc.begin()].push_back(i);
        }
        P.class_off.assign(nc + 1, 0);
        for (int k = 0; k < nc; k++) {
            P.class_off[k + 1] = P.class_off[k] + (int)cq[k].size();
            P.class_queue.insert(P.class_queue.end(), cq[k].begin(), cq[k].end());
        }
        P.log_off.assign(T + 1, 0);
        for (int t = 0; t < T; t++) {
            const int k = (int)(std::find(pc.begin(), pc.end(), P.team_size[t]) - pc.begin());
            P.team_class.push_back(k);
            P.log_off[t + 1] = P.log_off[t] + (int)cq[k].size();
        }
        out.phases.push_back(std::move(P));
    }
    return "";
}

}  // namespace pg
