// solver.cu -- multigrid preconditioner and outer Krylov recurrences for the composite pressure.
//
// Preconditioner: the reference's two-stage cycle (src/core/fluid/amr_pressure.cu:1103-1154):
// damped Jacobi (omega 2/3) on the finest composite graph around a Galerkin-style aggregation
// hierarchy built on the level-0 Cartesian lattice (setup :857-1069): every active DOF is summed
// into its level-0 cell, coarse levels aggregate 2x2x2 lattice cells through union-find, and the
// coarsest level (<= 512 cells or 8 levels) takes 96 Jacobi sweeps.  The small levels, the
// coarsest sweeps included, run as one cluster launch (stage_tail.cu); a Jacobi sweep is
// order-independent per row, so the results are those of separate launches.
//
// Outer solvers: FP64 PCG with periodic true-residual replacement (reference :1267-1353) for an
// orthogonal operator and flexible GCRO/LGMRES(24) with 3 recycled vectors (reference :1390-1698)
// when WLS non-orthogonal corrections are present.
#include "pcfd_internal.h"

#include <cuda_fp16.h>

#include <cstring>

#include <algorithm>
#include <array>
#include <cmath>
#include <limits>
#include <type_traits>
#include <unordered_map>

namespace pcfd
{
    namespace
    {
        // One level of an aggregation hierarchy, assembled on the host: a weighted graph
        // Laplacian (the couplings) plus a non-negative sink per cell, the part of the row that no
        // coupling represents (outlet and gauge terms).  Keeping the sink explicit gives every
        // coarser diagonal as a plain sum, with no subtraction of nearly equal numbers.
        struct Coupling { int lo, hi; double weight; };
        struct GraphLevel
        {
            int cells = 0;
            std::vector<double> sink, diagonal;       // diagonal = sink + incident coupling weights
            std::vector<Coupling> couplings;          // lo < hi, sorted, each pair once
            std::vector<int> row_offset, neighbour;   // symmetric CSR of the couplings
            std::vector<double> weight;
            std::vector<int> parent;                  // cell of the next coarser level (empty on the coarsest)
            std::vector<int> member_offset, member;   // members of each next-level cell (restriction)
        };

        // Members of each group of `map` (entries < 0 belong to none) as CSR over [0, groups), each
        // group's members in ascending order.
        void group_members(const std::vector<int>& map, int groups, std::vector<int>& offset, std::vector<int>& member)
        {
            offset.assign(size_t(groups) + 1, 0);
            for (const int g : map)
                if (g >= 0) ++offset[size_t(g) + 1];
            for (int g = 0; g < groups; ++g) offset[size_t(g) + 1] += offset[size_t(g)];
            member.resize(size_t(offset.back()));
            std::vector<int> fill(offset.begin(), offset.end() - 1);
            for (int q = 0; q < int(map.size()); ++q)
                if (map[q] >= 0) member[size_t(fill[size_t(map[q])]++)] = q;
        }

        // Merges the coupling records of `level` by cell pair, then derives the diagonal and the
        // CSR rows.  `records` holds (lo, hi, weight) with lo < hi, in any order and repeated.
        void assemble(GraphLevel& level, std::vector<Coupling>& records)
        {
            std::sort(records.begin(), records.end(),
                      [](const Coupling& x, const Coupling& y) { return x.lo != y.lo ? x.lo < y.lo : x.hi < y.hi; });
            level.couplings.clear();
            for (const Coupling& r : records)
            {
                if (!level.couplings.empty() && level.couplings.back().lo == r.lo && level.couplings.back().hi == r.hi)
                    level.couplings.back().weight += r.weight;
                else
                    level.couplings.push_back(r);
            }
            level.diagonal = level.sink;
            std::vector<int> degree(size_t(level.cells), 0);
            for (const Coupling& c : level.couplings)
            {
                level.diagonal[size_t(c.lo)] += c.weight;
                level.diagonal[size_t(c.hi)] += c.weight;
                ++degree[size_t(c.lo)];
                ++degree[size_t(c.hi)];
            }
            level.row_offset.assign(size_t(level.cells) + 1, 0);
            for (int q = 0; q < level.cells; ++q) level.row_offset[size_t(q) + 1] = level.row_offset[size_t(q)] + degree[size_t(q)];
            level.neighbour.resize(size_t(level.row_offset.back()));
            level.weight.resize(size_t(level.row_offset.back()));
            std::vector<int> fill(level.row_offset.begin(), level.row_offset.end() - 1);
            for (const Coupling& c : level.couplings)
            {
                int slot = fill[size_t(c.lo)]++;
                level.neighbour[size_t(slot)] = c.hi;
                level.weight[size_t(slot)] = c.weight;
                slot = fill[size_t(c.hi)]++;
                level.neighbour[size_t(slot)] = c.lo;
                level.weight[size_t(slot)] = c.weight;
            }
        }

        template <class T> void upload_level(MgLevel<T>& d, const GraphLevel& h)
        {
            d.cells = h.cells;
            d.row_offset.upload(h.row_offset);
            d.neighbour.upload(h.neighbour);
            d.coefficient.upload(std::vector<T>(h.weight.begin(), h.weight.end()));
            d.diagonal.upload(std::vector<T>(h.diagonal.begin(), h.diagonal.end()));
            d.rhs.alloc(h.cells); d.x.alloc(h.cells); d.temporary.alloc(h.cells); d.residual.alloc(h.cells);
            d.aggregate.upload(h.parent);
            d.restrict_offset.upload(h.member_offset);
            d.restrict_dof.upload(h.member);
        }

        // Brick-structured copy of a level numbered as 64 rows per brick (the first composite
        // stage): every CSR coupling to a face neighbour goes to its face slot, the others to the
        // row's rest entries, both in CSR order.  `convert` gives the stored coefficient (TK, the
        // type the kernels read).  Leaves the level in CSR form when a row has more than 31 rest
        // entries.
        template <class T, class TK, class Convert>
        void upload_brick_rows(MgLevel<T>& d, const GraphLevel& h, const std::vector<int>& neighbour, Convert convert,
                               DBuf<TK>& rest_coefficient)
        {
            constexpr int W = (6 * int(sizeof(TK)) + 4 + 15) / 16;
            if (h.cells % 64 != 0 || neighbour.size() != size_t(h.cells / 64) * 6) return;
            std::vector<uint4> rows(size_t(h.cells) * W, make_uint4(0u, 0u, 0u, 0u));
            std::vector<int> rest_column;
            std::vector<TK> rest_value;
            for (int q = 0; q < h.cells; ++q)
            {
                const int cell = q & 63, i = cell & 3, j = (cell >> 2) & 3, k = cell >> 4;
                const int* nb = neighbour.data() + 6 * size_t(q >> 6);
                auto across = [&](int f, int shift) { return nb[f] >= 0 ? nb[f] * 64 + cell + shift : -1; };
                const int n[6] = {k > 0 ? q - 16 : across(4, 48), j > 0 ? q - 4 : across(2, 12), i > 0 ? q - 1 : across(0, 3),
                                  i < 3 ? q + 1 : across(1, -3),  j < 3 ? q + 4 : across(3, -12), k < 3 ? q + 16 : across(5, -48)};
                TK c[6];
                bool set[6] = {false, false, false, false, false, false};
                for (int f = 0; f < 6; ++f) c[f] = convert(0.0);
                const int first = int(rest_column.size());
                for (int e = h.row_offset[size_t(q)]; e < h.row_offset[size_t(q) + 1]; ++e)
                {
                    const int column = h.neighbour[size_t(e)];
                    int f = 0;
                    while (f < 6 && (set[f] || n[f] != column)) ++f;
                    if (f < 6)
                    {
                        c[f] = convert(h.weight[size_t(e)]);
                        set[f] = true;
                    }
                    else
                    {
                        rest_column.push_back(column);
                        rest_value.push_back(convert(h.weight[size_t(e)]));
                    }
                }
                const int count = int(rest_column.size()) - first;
                if (count > 31 || first >= (1 << 27)) return;
                const uint32_t descriptor = (uint32_t(first) << 5) | uint32_t(count);
                unsigned char* row = reinterpret_cast<unsigned char*>(rows.data() + size_t(q) * W);
                std::memcpy(row, c, sizeof(c));
                std::memcpy(row + sizeof(c), &descriptor, sizeof(descriptor));
            }
            d.brick_rows.upload(rows);
            d.brick_neighbour.upload(neighbour);
            d.rest_column.upload(rest_column);
            rest_coefficient.upload(rest_value);
        }

        std::vector<HostRows> host_rows(const std::vector<GraphLevel>& levels)
        {
            std::vector<HostRows> rows;
            for (const GraphLevel& l : levels)
                rows.push_back(HostRows{l.cells, &l.row_offset, &l.neighbour, &l.parent, &l.member_offset, &l.member, &l.weight, &l.diagonal});
            return rows;
        }

        double connection_factor(const pcfd_connections& c, int e)
        {
            const double f = c.orthogonal_gradient_factor[e];
            return f > 0 ? f : (c.normal_distance[e] > 0 ? 1.0 / c.normal_distance[e] : 0.0);
        }

        // The fine orthogonal operator's two-point couplings: same-level faces of every
        // non-covered brick (minus cut faces), then the coarse/fine, embedded and regular
        // correction edges with their two-point weights.
        template <class F> void fine_couplings(const pcfd_topology& t, F&& add)
        {
            const int bs = t.brick_size, c3 = bs * bs * bs;
            for (int l = 0; l < t.level_count; ++l)
            {
                const pcfd_level& lev = t.levels[l];
                for (int brick = 0; brick < lev.brick_count; ++brick)
                {
                    if (lev.flags[brick] & PCFD_BRICK_COVERED) continue;
                    for (int c = 0; c < c3; ++c)
                    {
                        const int a = lev.level_offset + brick * c3 + c;
                        if (!t.active[a]) continue;
                        const int ijk[3] = {c % bs, (c / bs) % bs, c / (bs * bs)};
                        for (int axis = 0; axis < 3; ++axis)
                        {
                            if (t.cut_face_mask[a] & (1u << axis)) continue;
                            int q[3] = {ijk[0], ijk[1], ijk[2]}, b = -1;
                            if (++q[axis] < bs) b = lev.level_offset + brick * c3 + (q[2] * bs + q[1]) * bs + q[0];
                            else
                            {
                                const int nb = lev.neighbors[brick * 6 + 2 * axis + 1];
                                if (nb >= 0 && !(lev.flags[nb] & PCFD_BRICK_COVERED))
                                {
                                    q[axis] = 0;
                                    b = lev.level_offset + nb * c3 + (q[2] * bs + q[1]) * bs + q[0];
                                }
                            }
                            add(a, b, lev.h);
                        }
                    }
                }
            }
            for (int e = 0; e < t.coarse_fine.count; ++e)
                add(t.coarse_fine.coarse_dof[e], t.coarse_fine.fine_dof[e], t.coarse_fine.open_area[e] * connection_factor(t.coarse_fine, e));
            for (int e = 0; e < t.embedded.count; ++e)
                add(t.embedded.coarse_dof[e], t.embedded.fine_dof[e], t.embedded.open_area[e] * connection_factor(t.embedded, e));
            for (int e = 0; e < t.regular.count; ++e)
                add(t.regular.lower_dof[e], t.regular.upper_dof[e], t.regular.open_area[e] * t.regular.two_point_delta[e]);
        }

        // Galerkin product of the fine orthogonal operator with the piecewise-constant map of the
        // active DOFs onto `cells` coarse cells (map[q] < 0: DOF q is not represented).  Couplings
        // inside one coarse cell cancel; the outlet (2h on X-max faces) and gauge terms become sinks.
        GraphLevel galerkin_level(const pcfd_topology& t, const std::vector<int>& map, int cells, bool outlet)
        {
            GraphLevel level;
            level.cells = cells;
            level.sink.assign(size_t(cells), 0.0);
            std::vector<Coupling> records;
            records.reserve(size_t(cells) * 3 + 16);
            fine_couplings(t, [&](int a, int b, double w) {
                if (a < 0 || b < 0 || a == b || !t.active[a] || !t.active[b] || !(w > 0)) return;
                const int ca = map[size_t(a)], cb = map[size_t(b)];
                if (ca < 0 || cb < 0 || ca == cb) return;
                records.push_back({std::min(ca, cb), std::max(ca, cb), w});
            });
            const int bs = t.brick_size, c3 = bs * bs * bs;
            if (outlet)
                for (int l = 0; l < t.level_count; ++l)
                {
                    const pcfd_level& lev = t.levels[l];
                    for (int b = 0; b < lev.brick_count; ++b)
                    {
                        if ((lev.flags[b] & PCFD_BRICK_COVERED) || !(lev.flags[b] & PCFD_BRICK_XMAX)) continue;
                        for (int c = bs - 1; c < c3; c += bs)
                        {
                            const int q = lev.level_offset + b * c3 + c;
                            if (t.active[q] && map[size_t(q)] >= 0) level.sink[size_t(map[size_t(q)])] += 2.0 * lev.h;
                        }
                    }
                }
            for (int g = 0; g < t.gauge_count; ++g)
            {
                const int q = t.gauge_dof[g];
                if (t.active[q] && map[size_t(q)] >= 0) level.sink[size_t(map[size_t(q)])] += t.gauge_coefficient[g];
            }
            assemble(level, records);
            return level;
        }

        // Galerkin coarsening of `fine` through `parent` (cell -> coarse cell, < 0: none).
        GraphLevel coarsen(const GraphLevel& fine, const std::vector<int>& parent, int cells)
        {
            GraphLevel coarse;
            coarse.cells = cells;
            coarse.sink.assign(size_t(cells), 0.0);
            for (int q = 0; q < fine.cells; ++q)
                if (parent[size_t(q)] >= 0) coarse.sink[size_t(parent[size_t(q)])] += fine.sink[size_t(q)];
            std::vector<Coupling> records;
            records.reserve(fine.couplings.size());
            for (const Coupling& c : fine.couplings)
            {
                const int a = parent[size_t(c.lo)], b = parent[size_t(c.hi)];
                if (a >= 0 && b >= 0 && a != b) records.push_back({std::min(a, b), std::max(a, b), c.weight});
            }
            assemble(coarse, records);
            return coarse;
        }

        // Block aggregation of a lattice level: cells of one 2x2x2 block of lattice coordinates
        // that are connected through couplings inside the block form one coarse cell, found by a
        // depth-first walk from each unvisited cell in index order (so coarse cells are numbered by
        // their lowest member).  Cells with a zero diagonal are not aggregated.  Each coarse cell
        // sits at its block's coordinate.  Returns the number of coarse cells.
        using Lattice = std::array<int, 3>;
        int block_aggregates(const GraphLevel& level, const std::vector<Lattice>& at, std::vector<int>& parent,
                             std::vector<Lattice>& coarse_at)
        {
            parent.assign(size_t(level.cells), -1);
            coarse_at.clear();
            auto block = [&](int q) { return Lattice{at[size_t(q)][0] >> 1, at[size_t(q)][1] >> 1, at[size_t(q)][2] >> 1}; };
            std::vector<int> pending;
            for (int seed = 0; seed < level.cells; ++seed)
            {
                if (parent[size_t(seed)] >= 0 || !(level.diagonal[size_t(seed)] > 0)) continue;
                const int id = int(coarse_at.size());
                const Lattice home = block(seed);
                coarse_at.push_back(home);
                parent[size_t(seed)] = id;
                pending.push_back(seed);
                while (!pending.empty())
                {
                    const int a = pending.back();
                    pending.pop_back();
                    for (int e = level.row_offset[size_t(a)]; e < level.row_offset[size_t(a) + 1]; ++e)
                    {
                        const int b = level.neighbour[size_t(e)];
                        if (parent[size_t(b)] < 0 && level.diagonal[size_t(b)] > 0 && block(b) == home)
                        {
                            parent[size_t(b)] = id;
                            pending.push_back(b);
                        }
                    }
                }
            }
            return int(coarse_at.size());
        }
    }

    namespace
    {
        constexpr double kOmega = 2.0 / 3.0;
        constexpr int kCoarsestSweeps = 96;
    }

    std::vector<std::pair<double, double>> smoothing_steps(int chebyshev, int sweeps)
    {
        std::vector<std::pair<double, double>> steps(size_t(sweeps), {0.0, kOmega});
        if (chebyshev < 2) return steps;
        // Chebyshev polynomial smoothing on [2 / ratio, 2] (D^-1 A of a diagonally dominant Galerkin
        // level has its spectrum in (0, 2])
        const double hi = 2.0, lo = hi / chebyshev, theta = 0.5 * (hi + lo), delta = 0.5 * (hi - lo), sigma = theta / delta;
        double rho = 1.0 / sigma;
        for (int k = 0; k < sweeps; ++k)
        {
            if (k == 0) { steps[0] = {0.0, 1.0 / theta}; continue; }
            const double next = 1.0 / (2.0 * sigma - rho);
            steps[size_t(k)] = {next * rho, 2.0 * next / delta};
            rho = next;
        }
        return steps;
    }

    // The reference's lattice multigrid (its setup: amr_pressure.cu:915-1069), built here as
    // Galerkin levels: the active DOFs summed into their level-0 Cartesian cells
    // (preconditioner_aggregate), then block aggregates of 2x2x2 lattice cells while the level
    // keeps more than 512 live cells (at most 8 levels above the coarsest) and aggregation still
    // shrinks it.
    void build_multigrid(System& s, const pcfd_topology& t, const std::vector<double>& diagonal)
    {
        (void)diagonal;
        const int bs = t.brick_size, c3 = bs * bs * bs;
        const pcfd_level& base = t.levels[0];
        s.base_offset = base.level_offset;
        s.base_cells = base.brick_count * c3;
        const int n = t.storage_size;

        // active DOF -> level-0 lattice cell; restriction CSR over the lattice cells
        std::vector<int> lattice(size_t(n), -1);
        for (int q = 0; q < n; ++q)
        {
            const int c = t.preconditioner_aggregate[q] - s.base_offset;
            if (t.active[q] && c >= 0 && c < s.base_cells) lattice[size_t(q)] = c;
        }
        {
            std::vector<int> offset, member;
            group_members(lattice, s.base_cells, offset, member);
            s.base_restrict_offset.upload(offset);
            s.base_restrict_dof.upload(member);
        }

        std::vector<Lattice> at(size_t(s.base_cells));
        for (int brick = 0; brick < base.brick_count; ++brick)
            for (int c = 0; c < c3; ++c)
                at[size_t(brick) * c3 + c] = {base.coord[3 * brick] * bs + c % bs, base.coord[3 * brick + 1] * bs + (c / bs) % bs,
                                              base.coord[3 * brick + 2] * bs + c / (bs * bs)};
        std::vector<GraphLevel> levels;
        GraphLevel current = galerkin_level(t, lattice, s.base_cells, s.outlet);
        for (;;)
        {
            const int live = int(std::count_if(current.diagonal.begin(), current.diagonal.end(), [](double v) { return v > 0; }));
            if (live <= 512 || levels.size() >= 8) break;
            std::vector<int> parent;
            std::vector<Lattice> coarse_at;
            const int cells = block_aggregates(current, at, parent, coarse_at);
            if (cells <= 0 || cells >= live) break;
            GraphLevel coarse = coarsen(current, parent, cells);
            current.parent = std::move(parent);
            group_members(current.parent, cells, current.member_offset, current.member);
            levels.push_back(std::move(current));
            current = std::move(coarse);
            at = std::move(coarse_at);
        }
        levels.push_back(std::move(current));
        s.mg64.clear();
        s.mg32.clear();
        // all of a level is set before the small ones are planned as one launch, which copies from them
        s.mg64.resize(levels.size());
        for (size_t l = 0; l < levels.size(); ++l)
        {
            upload_level(s.mg64[l], levels[l]);
            s.mg64[l].prolong = s.mg_lattice_scale;
        }
        if (s.mg_precision == PCFD_MG_FP32)
        {
            s.mg32.resize(levels.size());
            for (size_t l = 0; l < levels.size(); ++l)
            {
                upload_level(s.mg32[l], levels[l]);
                s.mg32[l].prolong = s.mg_lattice_scale;
            }
            plan_tail(s.mg32, host_rows(levels), kCoarsestSweeps, kOmega, s.mg_tail32);
        }
        plan_tail(s.mg64, host_rows(levels), kCoarsestSweeps, kOmega, s.mg_tail64);
    }

    // ==================================================================================
    // composite-grid levels (PCFD_MG_CYCLE_COMPOSITE)
    // ==================================================================================
    // The reference aggregates every DOF of a level-l brick straight into its level-0 cell (8^l
    // fine cells per aggregate on the finest level), so the coarse space misses every scale
    // between 2 h_l and h_0.  The composite cycle replaces that hierarchy with stages that
    // coarsen every AMR level by 2x2x2 at once: stage k holds one cell per 2^k x 2^k x 2^k block
    // of same-level cells (cells of different levels never merge; the levels stay coupled
    // through the Galerkin coarse-fine couplings), down to 512 cells or fewer.  Stage operators
    // are Galerkin products of the fine orthogonal operator with the piecewise-constant stage
    // map; every prolongation is weighted 2, as the 2x2x2 Galerkin coarse operator of a uniform
    // Laplacian is twice the rediscretised one.  Each stage takes mg_stage_sweeps damped-Jacobi
    // sweeps before and after its coarse correction, the coarsest 96.
    namespace
    {
        // Explicit inverse of a coarsest level of at most 512 cells (Gauss-Jordan with partial
        // pivoting in FP64) over its cells with a positive diagonal; rows and columns of the other
        // cells stay zero, as the Jacobi sweeps leave them.  Empty when the level is larger or the
        // matrix is numerically singular (the 96 Jacobi sweeps are used then).
        std::vector<double> dense_inverse(const GraphLevel& level)
        {
            const int n = level.cells;
            if (n <= 0 || n > 512) return {};
            std::vector<int> live;
            std::vector<int> index(size_t(n), -1);
            for (int q = 0; q < n; ++q)
                if (level.diagonal[q] > 0) { index[q] = int(live.size()); live.push_back(q); }
            const int m = int(live.size());
            if (!m) return {};
            std::vector<double> a(size_t(m) * m, 0.0), inv(size_t(m) * m, 0.0);
            double scale = 0.0;
            for (int i = 0; i < m; ++i)
            {
                a[size_t(i) * m + i] = level.diagonal[live[i]];
                inv[size_t(i) * m + i] = 1.0;
                scale = std::max(scale, std::abs(level.diagonal[live[i]]));
            }
            for (const Coupling& e : level.couplings)
            {
                const int i = index[e.lo], j = index[e.hi];
                if (i < 0 || j < 0) continue;
                a[size_t(i) * m + j] -= e.weight;
                a[size_t(j) * m + i] -= e.weight;
            }
            for (int c = 0; c < m; ++c)
            {
                int p = c;
                for (int r = c + 1; r < m; ++r)
                    if (std::abs(a[size_t(r) * m + c]) > std::abs(a[size_t(p) * m + c])) p = r;
                if (!(std::abs(a[size_t(p) * m + c]) > 1e-12 * scale)) return {};
                if (p != c)
                    for (int j = 0; j < m; ++j)
                    {
                        std::swap(a[size_t(p) * m + j], a[size_t(c) * m + j]);
                        std::swap(inv[size_t(p) * m + j], inv[size_t(c) * m + j]);
                    }
                const double d = 1.0 / a[size_t(c) * m + c];
                for (int j = 0; j < m; ++j) { a[size_t(c) * m + j] *= d; inv[size_t(c) * m + j] *= d; }
                for (int r = 0; r < m; ++r)
                {
                    if (r == c) continue;
                    const double f = a[size_t(r) * m + c];
                    if (f == 0.0) continue;
                    for (int j = 0; j < m; ++j)
                    {
                        a[size_t(r) * m + j] -= f * a[size_t(c) * m + j];
                        inv[size_t(r) * m + j] -= f * inv[size_t(c) * m + j];
                    }
                }
            }
            std::vector<double> out(size_t(n) * n, 0.0);
            for (int i = 0; i < m; ++i)
                for (int j = 0; j < m; ++j)
                {
                    const double v = inv[size_t(i) * m + j];
                    if (!std::isfinite(v)) return {};
                    out[size_t(live[i]) * n + live[j]] = v;
                }
            return out;
        }
    }

    void build_composite(System& s, const pcfd_topology& t)
    {
        const int bs = t.brick_size, c3 = bs * bs * bs, S = t.storage_size;
        // every active structured DOF: level and global cell coordinates at that level, and the
        // brick slot that holds the cell
        std::vector<int8_t> dof_level(size_t(S), -1);
        std::vector<std::array<int64_t, 3>> gcoord(static_cast<size_t>(S));
        std::vector<int> dof_slot(size_t(S), -1), level_slot(size_t(t.level_count) + 1, 0);
        for (int l = 0; l < t.level_count; ++l) level_slot[size_t(l) + 1] = level_slot[size_t(l)] + t.levels[l].brick_count;
        for (int l = 0; l < t.level_count; ++l)
        {
            const pcfd_level& lev = t.levels[l];
            for (int b = 0; b < lev.brick_count; ++b)
            {
                if (lev.flags[b] & PCFD_BRICK_COVERED) continue;
                for (int c = 0; c < c3; ++c)
                {
                    const int q = lev.level_offset + b * c3 + c;
                    if (!t.active[q]) continue;
                    dof_level[q] = int8_t(l);
                    dof_slot[q] = level_slot[size_t(l)] + b;
                    gcoord[q] = {int64_t(lev.coord[3 * b]) * bs + c % bs, int64_t(lev.coord[3 * b + 1]) * bs + (c / bs) % bs,
                            int64_t(lev.coord[3 * b + 2]) * bs + c / (bs * bs)};
                }
            }
        }
        // EB fragments (DOFs after the structured slots) join the stages through the cell that
        // contains their centroid (a fragment is a piece of its cut cell, and a cell box is convex,
        // so the centroid lies in that cell): the finest non-covered brick at the centroid, the
        // cell index inside it clamped to the brick.  Without them the stages carry no coarse
        // correction for the cut cells, and on cut-cell grids the cycle loses its coarse space
        // exactly where the solution varies most.
        {
            const auto brick_key = [](int64_t x, int64_t y, int64_t z) {
                return (uint64_t(x & 0x1fffff) << 42) | (uint64_t(y & 0x1fffff) << 21) | uint64_t(z & 0x1fffff);
            };
            std::vector<std::unordered_map<uint64_t, int>> bricks(static_cast<size_t>(t.level_count));
            for (int l = 0; l < t.level_count; ++l)
                for (int b = 0; b < t.levels[l].brick_count; ++b)
                    bricks[size_t(l)][brick_key(t.levels[l].coord[3 * b], t.levels[l].coord[3 * b + 1], t.levels[l].coord[3 * b + 2])] = b;
            for (int q = s.structured; q < S; ++q)
            {
                if (!t.active[q]) continue;
                const double* c = t.centroid + 3 * size_t(q);
                for (int l = t.level_count - 1; l >= 0; --l)
                {
                    const pcfd_level& lev = t.levels[l];
                    const double width = bs * lev.h;
                    int64_t at[3];
                    for (int a = 0; a < 3; ++a) at[a] = int64_t(std::floor((c[a] - t.domain_lo[a]) / width));
                    const auto it = bricks[size_t(l)].find(brick_key(at[0], at[1], at[2]));
                    if (it == bricks[size_t(l)].end() || (lev.flags[it->second] & PCFD_BRICK_COVERED)) continue;
                    const int b = it->second;
                    std::array<int64_t, 3> cell;
                    for (int a = 0; a < 3; ++a)
                        cell[size_t(a)] = int64_t(lev.coord[3 * b + a]) * bs +
                                          std::min<int64_t>(bs - 1, std::max<int64_t>(0, int64_t(std::floor((c[a] - lev.origin[3 * b + a]) / lev.h))));
                    dof_level[size_t(q)] = int8_t(l);
                    dof_slot[size_t(q)] = level_slot[size_t(l)] + b;
                    gcoord[size_t(q)] = cell;
                    break;
                }
            }
        }
        auto key = [](int m, int64_t x, int64_t y, int64_t z) {
            return (uint64_t(m) << 60) | (uint64_t(x & 0xfffff) << 40) | (uint64_t(y & 0xfffff) << 20) | uint64_t(z & 0xfffff);
        };
        // stage maps: stage k merges the level-l cells at global cell coordinates g into the cell
        // (l, g >> k) of the same level, so the maps nest (stage k -> k + 1 halves every index);
        // stages stop at 512 cells or when a coarsening no longer shrinks the grid.
        // With 8^3 bricks a stage-1 cell never leaves its brick, so stage 1 is numbered as 64 rows
        // per non-covered brick (brick rank * 64 + x + 4 y + 16 z of the 4^3 block, rows without a
        // member stay empty): the brick-structured smoothing kernels find a row's face neighbours
        // from its index.  Later stages are numbered in order of first appearance.
        std::vector<int> slot_rank(size_t(level_slot.back()), -1), brick_neighbour;
        int ranks = 0;
        if (bs == 8)
            for (int l = 0; l < t.level_count; ++l)
                for (int b = 0; b < t.levels[l].brick_count; ++b)
                    if (!(t.levels[l].flags[b] & PCFD_BRICK_COVERED)) slot_rank[size_t(level_slot[size_t(l)] + b)] = ranks++;
        if (bs == 8)
        {
            brick_neighbour.assign(size_t(ranks) * 6, -1);
            for (int l = 0; l < t.level_count; ++l)
            {
                const pcfd_level& lev = t.levels[l];
                for (int b = 0; b < lev.brick_count; ++b)
                {
                    const int r = slot_rank[size_t(level_slot[size_t(l)] + b)];
                    if (r < 0) continue;
                    for (int f = 0; f < 6; ++f)
                    {
                        const int n = lev.neighbors[b * 6 + f];
                        if (n >= 0 && !(lev.flags[n] & PCFD_BRICK_COVERED))
                            brick_neighbour[size_t(r) * 6 + f] = slot_rank[size_t(level_slot[size_t(l)] + n)];
                    }
                }
            }
        }
        std::vector<std::vector<int>> map;
        std::vector<int> stage_cells;
        if (bs == 8 && ranks > 0)
        {
            std::vector<int> m(size_t(S), -1);
            for (int q = 0; q < S; ++q)
            {
                const int l = dof_level[q];
                if (l < 0) continue;
                const int slot = dof_slot[q], b = slot - level_slot[size_t(l)];
                const int* coord = t.levels[l].coord + 3 * b;
                int local[3];
                for (int a = 0; a < 3; ++a) local[a] = int(gcoord[q][size_t(a)] - int64_t(coord[a]) * bs) >> 1;
                if (slot_rank[size_t(slot)] < 0 || local[0] < 0 || local[0] > 3 || local[1] < 0 || local[1] > 3 || local[2] < 0 ||
                    local[2] > 3)
                    throw Error(PCFD_INTERNAL, "composite cycle: a stage-1 cell outside its brick");
                m[q] = slot_rank[size_t(slot)] * 64 + local[0] + 4 * local[1] + 16 * local[2];
            }
            map.push_back(std::move(m));
            stage_cells.push_back(ranks * 64);
            // the fused fine level computes stage-1 rows from brick ranks (its active bricks are the
            // non-covered bricks in the same order)
            if (ranks != s.active_bricks) throw Error(PCFD_INTERNAL, "composite cycle: brick ranks do not match the active bricks");
            s.fine.stage_neighbour.upload(brick_neighbour);
        }
        const bool first_is_coarsest = !stage_cells.empty() && stage_cells.front() <= 512;
        for (int k = int(map.size()) + 1; k <= 16 && !first_is_coarsest; ++k)
        {
            std::vector<int> m(size_t(S), -1);
            std::unordered_map<uint64_t, int> index;
            index.reserve(stage_cells.empty() ? size_t(S) / 6 : size_t(stage_cells.back()) / 6 + 16);
            for (int q = 0; q < S; ++q)
            {
                const int l = dof_level[q];
                if (l < 0) continue;
                const uint64_t kq = key(l, gcoord[q][0] >> k, gcoord[q][1] >> k, gcoord[q][2] >> k);
                auto it = index.find(kq);
                if (it == index.end()) it = index.emplace(kq, int(index.size())).first;
                m[q] = it->second;
            }
            const int cells = int(index.size());
            if (cells == 0 || (!stage_cells.empty() && cells >= stage_cells.back())) break;
            map.push_back(std::move(m));
            stage_cells.push_back(cells);
            if (cells <= 512) break;
        }
        if (map.empty()) throw Error(PCFD_INTERNAL, "composite cycle: no active structured cells");
        const int K = int(map.size());
        // Galerkin stage operators through map[k]; stage k -> stage k + 1 parents (consistent for
        // every DOF of a cell) and restriction CSR; the last stage is the coarsest and keeps none
        std::vector<GraphLevel> stages;
        stages.reserve(size_t(K));
        for (int k = 0; k < K; ++k) stages.push_back(galerkin_level(t, map[size_t(k)], stage_cells[size_t(k)], s.outlet));
        for (int k = 0; k + 1 < K; ++k)
        {
            GraphLevel& level = stages[size_t(k)];
            level.parent.assign(size_t(level.cells), -1);
            for (int q = 0; q < S; ++q)
            {
                const int here = map[size_t(k)][size_t(q)];
                if (here < 0) continue;
                int& p = level.parent[size_t(here)];
                if (p < 0) p = map[size_t(k) + 1][size_t(q)];
                else if (p != map[size_t(k) + 1][size_t(q)]) throw Error(PCFD_INTERNAL, "composite stage maps are not nested");
            }
            group_members(level.parent, stage_cells[size_t(k) + 1], level.member_offset, level.member);
        }
        // fine -> stage 1 map and restriction CSR (DOF order kept).  With stage 1 numbered by brick
        // rank, a row's structured members follow from its index and only the EB fragments
        // mapped to it are listed.
        const std::vector<int>& first = map[0];
        std::vector<int> roff, rdof;
        s.first_stage_bricks = s.fine.stage_neighbour.p != nullptr;
        if (s.first_stage_bricks)
        {
            std::vector<int> fragments(first);
            std::fill(fragments.begin(), fragments.begin() + std::min<size_t>(fragments.size(), size_t(s.structured)), -1);
            group_members(fragments, stage_cells[0], roff, rdof);
        }
        else
            group_members(first, stage_cells[0], roff, rdof);
        s.fine_map.upload(first);
        s.fine_restrict_offset.upload(roff);
        s.fine_restrict_dof.upload(rdof);
        s.fine_residual.alloc(size_t(S));
        s.inter64.clear();
        s.inter32.clear();
        const std::vector<double> inverse = dense_inverse(stages.back());
        if (s.composite_fp32)
        {
            s.inter32.resize(stages.size());
            for (size_t k = 0; k < stages.size(); ++k)
            {
                upload_level(s.inter32[k], stages[k]);
                s.inter32[k].prolong = 2.0;
                s.inter32[k].sweeps = s.mg_stage_sweeps;
                s.inter32[k].chebyshev = s.mg_stage_chebyshev;
            }
            if (!inverse.empty()) s.inter32.back().inverse.upload(std::vector<float>(inverse.begin(), inverse.end()));
            if (s.mg_stage_fp16)
                // FP16 storage of the stage coefficients (the coarsest keeps FP32 for its own sweeps)
                for (size_t k = 0; k + 1 < stages.size(); ++k)
                {
                    std::vector<uint16_t> bits(stages[k].weight.size());
                    for (size_t e = 0; e < bits.size(); ++e)
                    {
                        const __half hv = __float2half_rn(float(stages[k].weight[e]));
                        std::memcpy(&bits[e], &hv, sizeof(uint16_t));
                    }
                    s.inter32[k].coefficient16.upload(bits);
                }
            if (!brick_neighbour.empty() && stages.size() > 1 && !s.mg_stage_csr)
            {
                MgLevel<float>& first_stage = s.inter32.front();
                if (first_stage.coefficient16.p)
                    upload_brick_rows<float, uint16_t>(first_stage, stages[0], brick_neighbour, [](double w) {
                        const __half hv = __float2half_rn(float(w));
                        uint16_t bits;
                        std::memcpy(&bits, &hv, sizeof(bits));
                        return bits;
                    }, first_stage.rest_coefficient16);
                else
                    upload_brick_rows<float, float>(first_stage, stages[0], brick_neighbour, [](double w) { return float(w); },
                                                    first_stage.rest_coefficient);
            }
        }
        else
        {
            s.inter64.resize(stages.size());
            for (size_t k = 0; k < stages.size(); ++k)
            {
                upload_level(s.inter64[k], stages[k]);
                s.inter64[k].prolong = 2.0;
                s.inter64[k].sweeps = s.mg_stage_sweeps;
                s.inter64[k].chebyshev = s.mg_stage_chebyshev;
            }
            if (!inverse.empty()) s.inter64.back().inverse.upload(inverse);
            if (!brick_neighbour.empty() && stages.size() > 1 && !s.mg_stage_csr)
                upload_brick_rows<double, double>(s.inter64.front(), stages[0], brick_neighbour, [](double w) { return w; },
                                                  s.inter64.front().rest_coefficient);
        }
        if (s.composite_fp32) plan_tail(s.inter32, host_rows(stages), kCoarsestSweeps, kOmega, s.composite_tail);
        else plan_tail(s.inter64, host_rows(stages), kCoarsestSweeps, kOmega, s.composite_tail);
        s.composite = true;
    }

    // ==================================================================================
    // V-cycle kernels
    // ==================================================================================
    namespace
    {
        __global__ void precondition_kernel(const double* r, double* z, const double* diag, const uint8_t* active, int64_t n, double omega)
        {
            const int64_t q = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
            if (q < n) z[q] = active[q] && diag[q] > 0.0 ? omega * r[q] / diag[q] : 0.0;
        }
        __global__ void jacobi_correction_kernel(const double* r, const double* Ax, double* x, const double* diag,
                                                 const uint8_t* active, int64_t n, double omega)
        {
            const int64_t q = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
            if (q < n && active[q] && diag[q] > 0.0) x[q] += omega * (r[q] - Ax[q]) / diag[q];
        }
        template <class T>
        __global__ void restrict_difference_kernel(const int* offset, const int* dof, const double* r, const double* Ax,
                                                   int cells, T* coarse_rhs)
        {
            const int c = blockIdx.x * blockDim.x + threadIdx.x;
            if (c >= cells) return;
            double sum = 0.0;
            for (int q = offset[c]; q < offset[c + 1]; ++q) sum += r[dof[q]] - Ax[dof[q]];
            coarse_rhs[c] = T(sum);
        }
        // CSR coefficients as stored: FP64, FP32 or (mg_stage_fp16) FP16
        __device__ inline double coefficient_value(double c) { return c; }
        __device__ inline double coefficient_value(float c) { return double(c); }
        __device__ inline double coefficient_value(__half c) { return double(__half2float(c)); }

        template <class T, class TK = T>
        __global__ void __launch_bounds__(256) algebraic_jacobi_kernel(const T* __restrict__ rhs, const T* __restrict__ x,
            T* __restrict__ next, const int* __restrict__ row_offset, const int* __restrict__ neighbour,
            const TK* __restrict__ coefficient, const T* __restrict__ diag, int cells, T omega)
        {
            chain_wait();
            chain_release();
            const int q = blockIdx.x * blockDim.x + threadIdx.x;
            if (q >= cells) return;
            const T dq = diag[q], xq = x[q], bq = rhs[q];
            const int e0 = row_offset[q], e1 = row_offset[q + 1];
            if (!(dq > T(0))) { next[q] = T(0); return; }
            double Ax = double(dq) * double(xq);
#pragma unroll 4
            for (int e = e0; e < e1; ++e) Ax -= coefficient_value(coefficient[e]) * double(x[neighbour[e]]);
            next[q] = xq + omega * T((double(bq) - Ax) / double(dq));
        }
        // x = inverse * rhs on a coarsest level (one warp per row, FP64 accumulation)
        template <class T>
        __global__ void dense_apply_kernel(const T* __restrict__ inverse, const T* __restrict__ rhs, T* __restrict__ x, int n)
        {
            chain_wait();
            chain_release();
            const int row = int((int64_t(blockIdx.x) * blockDim.x + threadIdx.x) >> 5), lane = threadIdx.x & 31;
            if (row >= n) return;
            double acc = 0.0;
            for (int j = lane; j < n; j += 32) acc += double(inverse[int64_t(row) * n + j]) * double(rhs[j]);
            for (int o = 16; o > 0; o >>= 1) acc += __shfl_down_sync(0xffffffffu, acc, o);
            if (lane == 0) x[row] = T(acc);
        }

        // One Chebyshev step of a CSR level, fused: r = rhs - A x, d = c1 d + c2 D^-1 r (first step:
        // d = c2 D^-1 r), next = x + d
        // Every per-row load that does not depend on another (diagonal, iterate, right-hand side,
        // direction, both row offsets) is issued before the first one is used, and the row loop is
        // unrolled so that several gathers are in flight; the sums keep the CSR order.
        template <class T, class TK = T>
        __global__ void __launch_bounds__(256) algebraic_chebyshev_kernel(const T* __restrict__ rhs, const T* __restrict__ x,
            T* __restrict__ next, T* __restrict__ d, const int* __restrict__ row_offset, const int* __restrict__ neighbour,
            const TK* __restrict__ coefficient, const T* __restrict__ diag, int cells, T c1, T c2, int first)
        {
            chain_wait();
            chain_release();
            const int q = blockIdx.x * blockDim.x + threadIdx.x;
            if (q >= cells) return;
            const T dq = diag[q], xq = x[q], bq = rhs[q], dold = first ? T(0) : d[q];
            const int e0 = row_offset[q], e1 = row_offset[q + 1];
            if (!(dq > T(0))) { next[q] = T(0); d[q] = T(0); return; }
            double Ax = double(dq) * double(xq);
#pragma unroll 4
            for (int e = e0; e < e1; ++e) Ax -= coefficient_value(coefficient[e]) * double(x[neighbour[e]]);
            const T step = c2 * T((double(bq) - Ax) / double(dq));
            const T dn = first ? step : c1 * dold + step;
            d[q] = dn;
            next[q] = xq + dn;
        }
        // The first step from x = 0 (every pre-smoothing of a correction; damped Jacobi with
        // c2 = omega): the residual is the right-hand side, so d = c2 D^-1 rhs and next = 0 + d without
        // reading the matrix or the iterate; the same values as the general step.
        template <class T>
        __global__ void __launch_bounds__(256) chebyshev_zero_start_kernel(const T* __restrict__ rhs, T* __restrict__ next,
                                                                           T* __restrict__ d, const T* __restrict__ diag, int cells, T c2)
        {
            chain_wait();
            chain_release();
            const int q = blockIdx.x * blockDim.x + threadIdx.x;
            if (q >= cells) return;
            const T dq = diag[q], bq = rhs[q];
            if (!(dq > T(0))) { next[q] = T(0); d[q] = T(0); return; }
            const T step = c2 * T(double(bq) / double(dq));
            d[q] = step;
            next[q] = T(0) + step;
        }

        // ---- brick-structured stage (rows as 4^3 blocks per fine brick) ------------------------
        // A row's face neighbours follow from its index: inside the block at offsets 16, 4, 1, across
        // a block face the facing cell of the neighbour block (BrickStage::neighbour).  Only the
        // couplings that are not face neighbours (coarse/fine, cut-cell) keep a column index.
        template <class TK> struct BrickStage
        {
            const uint4* rows;            // stage_row_words<TK>() 16-byte words per row
            const int* neighbour;         // [blocks][6]: -x, +x, -y, +y, -z, +z
            const int* rest_column;
            const TK* rest_coefficient;
        };
        template <class TK> __host__ __device__ constexpr int stage_row_words() { return (6 * int(sizeof(TK)) + 4 + 15) / 16; }

        // Decodes a row: six coefficients (-z, -y, -x, +x, +y, +z) then the rest descriptor, packed
        // little-endian from the row's first byte.
        __device__ inline void load_stage_row(const uint4* __restrict__ rows, int q, __half (&c)[6], uint32_t& rest)
        {
            const uint4 w = rows[q];
            c[0] = __ushort_as_half(static_cast<unsigned short>(w.x & 0xffffu)); c[1] = __ushort_as_half(static_cast<unsigned short>(w.x >> 16));
            c[2] = __ushort_as_half(static_cast<unsigned short>(w.y & 0xffffu)); c[3] = __ushort_as_half(static_cast<unsigned short>(w.y >> 16));
            c[4] = __ushort_as_half(static_cast<unsigned short>(w.z & 0xffffu)); c[5] = __ushort_as_half(static_cast<unsigned short>(w.z >> 16));
            rest = w.w;
        }
        __device__ inline void load_stage_row(const uint4* __restrict__ rows, int q, float (&c)[6], uint32_t& rest)
        {
            const uint4 w0 = rows[2 * int64_t(q)], w1 = rows[2 * int64_t(q) + 1];
            c[0] = __uint_as_float(w0.x); c[1] = __uint_as_float(w0.y); c[2] = __uint_as_float(w0.z); c[3] = __uint_as_float(w0.w);
            c[4] = __uint_as_float(w1.x); c[5] = __uint_as_float(w1.y);
            rest = w1.z;
        }
        __device__ inline void load_stage_row(const uint4* __restrict__ rows, int q, double (&c)[6], uint32_t& rest)
        {
            const uint4 w0 = rows[4 * int64_t(q)], w1 = rows[4 * int64_t(q) + 1], w2 = rows[4 * int64_t(q) + 2];
            c[0] = __hiloint2double(int(w0.y), int(w0.x)); c[1] = __hiloint2double(int(w0.w), int(w0.z));
            c[2] = __hiloint2double(int(w1.y), int(w1.x)); c[3] = __hiloint2double(int(w1.w), int(w1.z));
            c[4] = __hiloint2double(int(w2.y), int(w2.x)); c[5] = __hiloint2double(int(w2.w), int(w2.z));
            rest = rows[4 * int64_t(q) + 3].x;
        }

        // Ax - (off-diagonal part of row q) x: face neighbours in the order -z, -y, -x, +x, +y, +z,
        // then the rest entries; a face slot with a zero coefficient loads nothing.
        template <class T, class TK>
        __device__ inline double brick_stage_product(int q, double Ax, const TK (&c)[6], uint32_t rest, const T* __restrict__ x,
                                                     const BrickStage<TK>& st)
        {
            const int cell = q & 63, i = cell & 3, j = (cell >> 2) & 3, k = cell >> 4;
            const int* nb = st.neighbour + 6 * (q >> 6);
            const int n[6] = {k > 0 ? q - 16 : nb[4] * 64 + cell + 48, j > 0 ? q - 4 : nb[2] * 64 + cell + 12,
                              i > 0 ? q - 1 : nb[0] * 64 + cell + 3,   i < 3 ? q + 1 : nb[1] * 64 + cell - 3,
                              j < 3 ? q + 4 : nb[3] * 64 + cell - 12,  k < 3 ? q + 16 : nb[5] * 64 + cell - 48};
            double v[6];
#pragma unroll
            for (int f = 0; f < 6; ++f) v[f] = coefficient_value(c[f]) != 0.0 ? double(x[n[f]]) : 0.0;
#pragma unroll
            for (int f = 0; f < 6; ++f) Ax -= coefficient_value(c[f]) * v[f];
            const int r0 = int(rest >> 5), r1 = r0 + int(rest & 31u);
#pragma unroll 2
            for (int e = r0; e < r1; ++e) Ax -= coefficient_value(st.rest_coefficient[e]) * double(x[st.rest_column[e]]);
            return Ax;
        }

        // algebraic_chebyshev_kernel on a brick-structured stage
        template <class T, class TK>
        __global__ void __launch_bounds__(256) brick_stage_chebyshev_kernel(const T* __restrict__ rhs, const T* __restrict__ x,
            T* __restrict__ next, T* __restrict__ d, BrickStage<TK> st, const T* __restrict__ diag, int cells, T c1, T c2, int first)
        {
            chain_wait();
            chain_release();
            const int q = blockIdx.x * blockDim.x + threadIdx.x;
            if (q >= cells) return;
            const T dq = diag[q], xq = x[q], bq = rhs[q], dold = first ? T(0) : d[q];
            TK c[6];
            uint32_t rest;
            load_stage_row(st.rows, q, c, rest);
            if (!(dq > T(0))) { next[q] = T(0); d[q] = T(0); return; }
            const double Ax = brick_stage_product<T, TK>(q, double(dq) * double(xq), c, rest, x, st);
            const T step = c2 * T((double(bq) - Ax) / double(dq));
            const T dn = first ? step : c1 * dold + step;
            d[q] = dn;
            next[q] = xq + dn;
        }
        template <class T, class TK>
        __global__ void __launch_bounds__(256) brick_stage_residual_kernel(const T* __restrict__ rhs, const T* __restrict__ x,
            T* __restrict__ residual, BrickStage<TK> st, const T* __restrict__ diag, int cells)
        {
            chain_wait();
            chain_release();
            const int q = blockIdx.x * blockDim.x + threadIdx.x;
            if (q >= cells) return;
            const T dq = diag[q], xq = x[q], bq = rhs[q];
            TK c[6];
            uint32_t rest;
            load_stage_row(st.rows, q, c, rest);
            if (!(dq > T(0))) { residual[q] = T(0); return; }
            residual[q] = T(double(bq) - brick_stage_product<T, TK>(q, double(dq) * double(xq), c, rest, x, st));
        }

        template <class T, class TK = T>
        __global__ void __launch_bounds__(256) algebraic_residual_kernel(const T* __restrict__ rhs, const T* __restrict__ x,
            T* __restrict__ residual, const int* __restrict__ row_offset, const int* __restrict__ neighbour,
            const TK* __restrict__ coefficient, const T* __restrict__ diag, int cells)
        {
            chain_wait();
            chain_release();
            const int q = blockIdx.x * blockDim.x + threadIdx.x;
            if (q >= cells) return;
            const T dq = diag[q], xq = x[q], bq = rhs[q];
            const int e0 = row_offset[q], e1 = row_offset[q + 1];
            if (!(dq > T(0))) { residual[q] = T(0); return; }
            double Ax = double(dq) * double(xq);
#pragma unroll 4
            for (int e = e0; e < e1; ++e) Ax -= coefficient_value(coefficient[e]) * double(x[neighbour[e]]);
            residual[q] = T(double(bq) - Ax);
        }
        template <class T> BrickStage<T> brick_stage(const MgLevel<T>& l)
        {
            return BrickStage<T>{l.brick_rows, l.brick_neighbour, l.rest_column, l.rest_coefficient};
        }
        template <class T> BrickStage<__half> brick_stage16(const MgLevel<T>& l)
        {
            return BrickStage<__half>{l.brick_rows, l.brick_neighbour, l.rest_column, reinterpret_cast<const __half*>(l.rest_coefficient16.p)};
        }
        template <class T>
        __global__ void restrict_gather_kernel(const int* offset, const int* dof, const T* residual, int cells, T* coarse_rhs)
        {
            chain_wait();
            chain_release();
            const int c = blockIdx.x * blockDim.x + threadIdx.x;
            if (c >= cells) return;
            double sum = 0.0;
            for (int q = offset[c]; q < offset[c + 1]; ++q) sum += double(residual[dof[q]]);
            coarse_rhs[c] = T(sum);
        }
        template <class T>
        __global__ void prolong_add_kernel(const int* aggregate, int cells, const T* coarse_x, T* fine_x, T scale)
        {
            chain_wait();
            chain_release();
            const int q = blockIdx.x * blockDim.x + threadIdx.x;
            if (q < cells && aggregate[q] >= 0) fine_x[q] += scale * coarse_x[aggregate[q]];
        }
        template <class T>
        __global__ void prolong_aggregate_kernel(const int* aggregate, const uint8_t* active, int64_t n, int base_offset,
                                                 int base_cells, const T* coarse_x, double* out, double scale)
        {
            const int64_t q = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
            if (q >= n || !active[q]) return;
            const int c = aggregate[q] - base_offset;
            if (c >= 0 && c < base_cells) out[q] += scale * double(coarse_x[c]);
        }
        // Coarsest-level Jacobi sweeps inside one CTA (cells <= blockDim.x * kPerThread).
        template <class T, int kPerThread>
        __global__ void __launch_bounds__(1024) coarse_jacobi_kernel(const T* rhs, T* x, T* temporary, const int* row_offset,
            const int* neighbour, const T* coefficient, const T* diag, int cells, T omega, int sweeps)
        {
            T* a = x;
            T* b = temporary;
            for (int sweep = 0; sweep < sweeps; ++sweep)
            {
                for (int r = 0; r < kPerThread; ++r)
                {
                    const int q = threadIdx.x + r * blockDim.x;
                    if (q >= cells) continue;
                    if (!(diag[q] > T(0))) { b[q] = T(0); continue; }
                    double Ax = double(diag[q]) * double(a[q]);
                    for (int e = row_offset[q]; e < row_offset[q + 1]; ++e) Ax -= double(coefficient[e]) * double(a[neighbour[e]]);
                    b[q] = a[q] + omega * T((double(rhs[q]) - Ax) / double(diag[q]));
                }
                __syncthreads();
                T* tmp = a; a = b; b = tmp;
            }
            // after an even number of sweeps the result is back in x; copy when odd
            if (sweeps & 1)
                for (int q = threadIdx.x; q < cells; q += blockDim.x) x[q] = temporary[q];
        }

        // One V-cycle from chain[index] down: level.sweeps smoothing steps from x = 0, residual,
        // restriction, the coarser levels, the weighted prolongation (chain[index]->prolong),
        // level.sweeps steps; the last level applies its explicit inverse or takes 96 sweeps (in one CTA
        // when it fits).  Levels from tail.first on run as one cluster launch.
        template <class T>
        void mg_level(System& s, MgLevel<T>* const* chain, int count, int index, const StageTail& tail)
        {
            MgLevel<T>& level = *chain[index];
            if (index == tail.first)
            {
                launch_tail(s, level, tail);
                return;
            }
            const T omega = T(kOmega);
            // from_zero: the pre-smoothing of a correction, whose first step needs neither the matrix
            // nor x; the Chebyshev direction lives in level.residual
            auto smooth = [&](int sweeps, bool from_zero) {
                const std::vector<std::pair<double, double>> steps = smoothing_steps(level.chebyshev, sweeps);
                for (int sweep = 0; sweep < sweeps; ++sweep)
                {
                    const T c1 = T(steps[size_t(sweep)].first), c2 = T(steps[size_t(sweep)].second);
                    if (from_zero && sweep == 0)
                    {
                        launch_chained(s, chebyshev_zero_start_kernel<T>, blocks_for(level.cells), kThreads,
                            level.rhs, level.temporary, level.residual, level.diagonal, level.cells, c2);
                        std::swap(level.x.p, level.temporary.p);
                        continue;
                    }
                    if (level.chebyshev >= 2)
                    {
                        // the first composite stage's full steps are the profiled stage-smoothing region
                        ProfileScope scope(s, index == 0 && s.composite ? PCFD_PROFILE_STAGE_SMOOTH : -1);
                        if (level.brick_rows.p && level.coefficient16.p)
                            launch_chained(s, brick_stage_chebyshev_kernel<T, __half>, blocks_for(level.cells), kThreads,
                                level.rhs, level.x, level.temporary, level.residual, brick_stage16(level), level.diagonal, level.cells,
                                c1, c2, sweep == 0 ? 1 : 0);
                        else if (level.brick_rows.p)
                            launch_chained(s, brick_stage_chebyshev_kernel<T, T>, blocks_for(level.cells), kThreads,
                                level.rhs, level.x, level.temporary, level.residual, brick_stage(level), level.diagonal, level.cells,
                                c1, c2, sweep == 0 ? 1 : 0);
                        else if (level.coefficient16.p)
                            launch_chained(s, algebraic_chebyshev_kernel<T, __half>, blocks_for(level.cells), kThreads,
                                level.rhs, level.x, level.temporary, level.residual, level.row_offset, level.neighbour,
                                reinterpret_cast<const __half*>(level.coefficient16.p), level.diagonal, level.cells, c1, c2,
                                sweep == 0 ? 1 : 0);
                        else
                            launch_chained(s, algebraic_chebyshev_kernel<T, T>, blocks_for(level.cells), kThreads,
                                level.rhs, level.x, level.temporary, level.residual, level.row_offset, level.neighbour, level.coefficient,
                                level.diagonal, level.cells, c1, c2, sweep == 0 ? 1 : 0);
                    }
                    else if (level.coefficient16.p)
                        launch_chained(s, algebraic_jacobi_kernel<T, __half>, blocks_for(level.cells), kThreads,
                            level.rhs, level.x, level.temporary, level.row_offset, level.neighbour,
                            reinterpret_cast<const __half*>(level.coefficient16.p), level.diagonal, level.cells, omega);
                    else
                        launch_chained(s, algebraic_jacobi_kernel<T, T>, blocks_for(level.cells), kThreads,
                            level.rhs, level.x, level.temporary, level.row_offset, level.neighbour, level.coefficient,
                            level.diagonal, level.cells, omega);
                    std::swap(level.x.p, level.temporary.p);
                }
            };
            if (index + 1 == count)
            {
                if (level.inverse.p)
                    launch_chained(s, dense_apply_kernel<T>, blocks_for(int64_t(level.cells) * 32), kThreads, level.inverse, level.rhs,
                                                                                                              level.x, level.cells);
                else if (level.cells <= 4096)
                {
                    cuda_check(cudaMemsetAsync(level.x, 0, size_t(level.cells) * sizeof(T), s.stream), "clear coarse correction");
                    coarse_jacobi_kernel<T, 4><<<1, 1024, 0, launch_stream(s)>>>(level.rhs, level.x, level.temporary, level.row_offset,
                        level.neighbour, level.coefficient, level.diagonal, level.cells, omega, kCoarsestSweeps);
                }
                else
                    smooth(kCoarsestSweeps, true);
                return;
            }
            smooth(level.sweeps, true);
            if (level.brick_rows.p && level.coefficient16.p)
                launch_chained(s, brick_stage_residual_kernel<T, __half>, blocks_for(level.cells), kThreads,
                    level.rhs, level.x, level.residual, brick_stage16(level), level.diagonal, level.cells);
            else if (level.brick_rows.p)
                launch_chained(s, brick_stage_residual_kernel<T, T>, blocks_for(level.cells), kThreads,
                    level.rhs, level.x, level.residual, brick_stage(level), level.diagonal, level.cells);
            else if (level.coefficient16.p)
                launch_chained(s, algebraic_residual_kernel<T, __half>, blocks_for(level.cells), kThreads,
                    level.rhs, level.x, level.residual, level.row_offset, level.neighbour,
                    reinterpret_cast<const __half*>(level.coefficient16.p), level.diagonal, level.cells);
            else
                launch_chained(s, algebraic_residual_kernel<T, T>, blocks_for(level.cells), kThreads,
                    level.rhs, level.x, level.residual, level.row_offset, level.neighbour, level.coefficient, level.diagonal, level.cells);
            MgLevel<T>& coarse = *chain[index + 1];
            launch_chained(s, restrict_gather_kernel<T>, blocks_for(coarse.cells), kThreads,
                level.restrict_offset, level.restrict_dof, level.residual, coarse.cells, coarse.rhs);
            mg_level(s, chain, count, index + 1, tail);
            launch_chained(s, prolong_add_kernel<T>, blocks_for(level.cells), kThreads, level.aggregate, level.cells, coarse.x, level.x,
                                                                                             T(level.prolong));
            smooth(level.sweeps, false);
        }

        // Runs mg_level over `chain` through a CUDA graph captured on first use (the chain and its
        // buffers are fixed for the system's lifetime), or, where it is one cluster launch, as that,
        // chained to its neighbours (65 k cells: 33.1 against 39.1 us an application; the levels of
        // larger grids launched one by one: 840 -> 849 us on 16 M).
        // Returns whether its last launch is a kernel that the next may be chained to.
        template <class T>
        bool run_captured(System& s, std::vector<MgLevel<T>*>& chain, const StageTail& tail, cudaGraphExec_t& exec, int64_t& nodes)
        {
            // uncaptured while the stage-smoothing region is profiled: its launches get event pairs
            // (and a first stage small enough for the cluster launch runs as launches of its own)
            if (!s.stream || s.profile_region == PCFD_PROFILE_STAGE_SMOOTH)
            {
                const bool apart = s.profile_region == PCFD_PROFILE_STAGE_SMOOTH && tail.first == 0;
                mg_level(s, chain.data(), int(chain.size()), 0, apart ? StageTail{} : tail);
                return false;
            }
            if (tail.first == 0)
            {
                mg_level(s, chain.data(), int(chain.size()), 0, tail);
                return true;
            }
            if (!exec)
            {
                const int64_t before = s.launches;
                cuda_check(cudaStreamBeginCapture(s.stream, cudaStreamCaptureModeThreadLocal), "begin hierarchy capture");
                cudaGraph_t graph = nullptr;
                try
                {
                    mg_level(s, chain.data(), int(chain.size()), 0, tail);
                }
                catch (...)
                {
                    cudaStreamEndCapture(s.stream, &graph);
                    if (graph) cudaGraphDestroy(graph);
                    throw;
                }
                cuda_check(cudaStreamEndCapture(s.stream, &graph), "end hierarchy capture");
                const cudaError_t e = cudaGraphInstantiate(&exec, graph, 0);
                cudaGraphDestroy(graph);
                cuda_check(e, "instantiate hierarchy graph");
                nodes = s.launches - before;
                s.launches = before;
            }
            cuda_check(cudaGraphLaunch(exec, s.stream), "launch hierarchy graph");
            s.launches += nodes;
            return false;
        }

        template <class T>
        void coarse_correction(System& s, std::vector<MgLevel<T>>& levels, const StageTail& tail, const double* r, double* z)
        {
            MgLevel<T>& base = levels.front();
            launch_apply(s, z, s.t, true);
            restrict_difference_kernel<T><<<blocks_for(base.cells), kThreads, 0, launch_stream(s)>>>(
                s.base_restrict_offset, s.base_restrict_dof, r, s.t, base.cells, base.rhs);
            std::vector<MgLevel<T>*> chain;
            for (MgLevel<T>& level : levels) chain.push_back(&level);
            mg_level(s, chain.data(), int(chain.size()), 0, tail);
            prolong_aggregate_kernel<T><<<blocks_for(s.S), kThreads, 0, launch_stream(s)>>>(s.aggregate, s.active, s.S, s.base_offset,
                                                                                  s.base_cells, base.x, z, s.mg_prolong_scale);
        }
    }

    void preconditioner_stage(System& s, int stage, const double* r, double* z)
    {
        if (stage == 0)
        {
            precondition_kernel<<<blocks_for(s.S), kThreads, 0, launch_stream(s)>>>(r, z, s.diagonal, s.active, s.S, kOmega);
            launch_apply(s, z, s.t, true);
            jacobi_correction_kernel<<<blocks_for(s.S), kThreads, 0, launch_stream(s)>>>(r, s.t, z, s.diagonal, s.active, s.S, kOmega);
        }
        else if (stage == 1 && !s.mg64.empty())
        {
            if (s.mg_precision == PCFD_MG_FP32 && !s.mg32.empty()) coarse_correction(s, s.mg32, s.mg_tail32, r, z);
            else coarse_correction(s, s.mg64, s.mg_tail64, r, z);
        }
        else if (stage == 2 && !s.mg64.empty())
            for (int sweep = 0; sweep < 2; ++sweep)
            {
                launch_apply(s, z, s.t, true);
                jacobi_correction_kernel<<<blocks_for(s.S), kThreads, 0, launch_stream(s)>>>(r, s.t, z, s.diagonal, s.active, s.S, kOmega);
            }
    }

    // The aggregation hierarchy below the fine level is the same fixed sequence of ~30 small
    // launches on every application (levels of 2.3 M cells down to <= 512), so it is captured
    // once into a CUDA graph on the system stream and replayed; the launch gaps of the coarse
    // levels, not their bytes, dominate it.  Systems on the legacy default stream launch directly.
    template <class T> bool multigrid_levels(System& s, std::vector<MgLevel<T>>& levels)
    {
        const bool fp32 = std::is_same<T, float>::value;
        std::vector<MgLevel<T>*> chain;
        for (MgLevel<T>& level : levels) chain.push_back(&level);
        return run_captured(s, chain, fp32 ? s.mg_tail32 : s.mg_tail64, fp32 ? s.mg_graph32 : s.mg_graph64, fp32 ? s.mg_graph32_launches : s.mg_graph64_launches);
    }

    // composite chain: the stage levels (FP32 or FP64), the last one the coarsest
    bool composite_levels(System& s)
    {
        if (s.composite_fp32)
        {
            std::vector<MgLevel<float>*> chain;
            for (MgLevel<float>& level : s.inter32) chain.push_back(&level);
            return run_captured(s, chain, s.composite_tail, s.mg_graph_composite, s.mg_graph_composite_launches);
        }
        std::vector<MgLevel<double>*> chain;
        for (MgLevel<double>& level : s.inter64) chain.push_back(&level);
        return run_captured(s, chain, s.composite_tail, s.mg_graph_composite, s.mg_graph_composite_launches);
    }

    // Algorithmic bytes of one step of the first composite stage's smoothing, each array read
    // once: per row rhs, x, diagonal, the direction read and written and the next iterate (4 B
    // each in FP32, 8 B in FP64), then in CSR form the row offset (4 B) and per stored coupling
    // its column index and coefficient; in brick-structured form the row's 16-byte words, per rest
    // entry its column and coefficient and per block its six neighbour blocks.
    double stage_smooth_bytes(const System& s)
    {
        auto bytes = [](const auto& l, double value) {
            const double coefficient = l.coefficient16.p ? 2.0 : value;
            if (l.brick_rows.p)
                return 6.0 * value * l.cells + 16.0 * double(l.brick_rows.n) + (4.0 + coefficient) * double(l.rest_column.n) +
                       24.0 * double(l.cells / 64);
            return 6.0 * value * l.cells + 4.0 * l.cells + (4.0 + coefficient) * double(l.neighbour.n);
        };
        if (s.composite_fp32 && !s.inter32.empty()) return bytes(s.inter32.front(), 4.0);
        if (!s.inter64.empty()) return bytes(s.inter64.front(), 8.0);
        return 0.0;
    }

    // One Chebyshev step of the first composite stage on its resident buffers (kernel timing).
    void stage_smooth_once(System& s)
    {
        require(s.composite && (!s.inter32.empty() || !s.inter64.empty()), "stage smoothing step: the composite cycle");
        auto run = [&](auto& level) {
            using T = typename std::remove_reference_t<decltype(level)>::value_type;
            if (level.brick_rows.p && level.coefficient16.p)
                brick_stage_chebyshev_kernel<T, __half><<<blocks_for(level.cells), kThreads, 0, launch_stream(s)>>>(
                    level.rhs, level.x, level.temporary, level.residual, brick_stage16(level), level.diagonal, level.cells, T(0.5),
                    T(0.7), 0);
            else if (level.brick_rows.p)
                brick_stage_chebyshev_kernel<T, T><<<blocks_for(level.cells), kThreads, 0, launch_stream(s)>>>(
                    level.rhs, level.x, level.temporary, level.residual, brick_stage(level), level.diagonal, level.cells, T(0.5),
                    T(0.7), 0);
            else if (level.coefficient16.p)
                algebraic_chebyshev_kernel<T, __half><<<blocks_for(level.cells), kThreads, 0, launch_stream(s)>>>(
                    level.rhs, level.x, level.temporary, level.residual, level.row_offset, level.neighbour,
                    reinterpret_cast<const __half*>(level.coefficient16.p), level.diagonal, level.cells, T(0.5), T(0.7), 0);
            else
                algebraic_chebyshev_kernel<T, T><<<blocks_for(level.cells), kThreads, 0, launch_stream(s)>>>(
                    level.rhs, level.x, level.temporary, level.residual, level.row_offset, level.neighbour, level.coefficient,
                    level.diagonal, level.cells, T(0.5), T(0.7), 0);
        };
        if (s.composite_fp32) run(s.inter32.front());
        else run(s.inter64.front());
        cuda_check(cudaGetLastError(), "stage smoothing step");
    }

    template bool multigrid_levels<double>(System&, std::vector<MgLevel<double>>&);
    template bool multigrid_levels<float>(System&, std::vector<MgLevel<float>>&);

    namespace
    {
        __global__ void jacobi_precondition_kernel(const double* r, double* z, const double* diag, const uint8_t* active, int64_t n)
        {
            const int64_t q = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
            if (q < n) z[q] = active[q] && diag[q] > 0.0 ? r[q] / diag[q] : 0.0;
        }

        void multigrid_preconditioner(System& s, const double* r, double* z)
        {
            if (s.composite && s.fine.enabled && aligned16(r) && aligned16(z))
            {
                composite_preconditioner(s, r, z);
                return;
            }
            if (s.fine.enabled && aligned16(r) && aligned16(z))
            {
                if (s.mg_precision == PCFD_MG_FP32 && !s.mg32.empty()) fine_preconditioner(s, r, z, s.mg32);
                else fine_preconditioner(s, r, z, s.mg64);
                return;
            }
            preconditioner_stage(s, 0, r, z);
            preconditioner_stage(s, 1, r, z);
            preconditioner_stage(s, 2, r, z);
            cuda_check(cudaGetLastError(), "preconditioner");
        }
    }

    void apply_preconditioner(System& s, const double* r, double* z)
    {
        ProfileScope scope(s, PCFD_PROFILE_PRECONDITIONER);
        if (s.preconditioner == PCFD_PRECONDITIONER_LEARNED || s.preconditioner == PCFD_PRECONDITIONER_LEARNED_MULTIGRID)
        {
            const bool coarse = s.preconditioner == PCFD_PRECONDITIONER_LEARNED_MULTIGRID;
            if (s.fine.enabled && aligned16(r) && aligned16(z) && (!coarse || s.composite)) learned_preconditioner(s, r, z, coarse);
            else learned_apply(s, r, z);
            return;
        }
        if (s.preconditioner == PCFD_PRECONDITIONER_JACOBI)
        {
            jacobi_precondition_kernel<<<blocks_for(s.S), kThreads, 0, launch_stream(s)>>>(r, z, s.diagonal, s.active, s.S);
            return;
        }
        multigrid_preconditioner(s, r, z);
        // training pairs for the learned preconditioner: (r, one multigrid application)
        if (learned_harvesting(s)) learned_harvest(s, r, z);
    }

    // ==================================================================================
    // PCG (orthogonal operator) and flexible GCRO/LGMRES (corrected operator)
    // ==================================================================================
    namespace
    {
        pcfd_solve_result solve_orthogonal(System& s, double* x, const double* b, double tolerance, int max_iterations, bool warm)
        {
            pcfd_solve_result result{};
            if (!warm) vec_zero(s, x);
            const double rhs2 = device_dot(s, b, b);
            if (rhs2 == 0) { vec_zero(s, x); result.converged = 1; return result; }
            if (!std::isfinite(rhs2) || rhs2 < 0) { result.relative_residual = std::numeric_limits<double>::infinity(); return result; }
            auto true_residual = [&]() {
                launch_apply(s, x, s.t, true);
                return vec_residual_dot(s, b, s.t, s.r);
            };
            double residual2;
            if (warm) residual2 = true_residual();
            else
            {
                cuda_check(cudaMemcpyAsync(s.r, b, size_t(s.S) * sizeof(double), cudaMemcpyDeviceToDevice, s.stream), "copy rhs");
                residual2 = rhs2;
            }
            result.relative_residual = std::sqrt(residual2 / rhs2);
            if (!std::isfinite(result.relative_residual)) return result;
            if (result.relative_residual <= tolerance) { result.converged = 1; return result; }
            auto restart = [&]() {
                apply_preconditioner(s, s.r, s.z);
                ++result.preconditioner_applications;
                vec_copy_active(s, s.z, s.dvec);
                return device_dot(s, s.r, s.z);
            };
            double rz = restart();
            if (!(rz > 0) || !std::isfinite(rz)) return result;
            constexpr int kReliable = 128;
            for (int it = 0; it < max_iterations; ++it)
            {
                launch_apply(s, s.dvec, s.Ad, true);
                const double pAp = device_dot(s, s.dvec, s.Ad);
                if (!(pAp > 0) || !std::isfinite(pAp)) break;
                const double alpha = rz / pAp;
                if (!std::isfinite(alpha)) break;
                vec_update_solution_residual(s, x, s.r, s.dvec, s.Ad, alpha);
                residual2 = device_dot(s, s.r, s.r);
                result.iterations = it + 1;
                result.relative_residual = std::sqrt(residual2 / rhs2);
                if (!std::isfinite(result.relative_residual)) break;
                const bool reliable = (it + 1) % kReliable == 0;
                if (result.relative_residual <= tolerance || reliable)
                {
                    residual2 = true_residual();
                    result.relative_residual = std::sqrt(residual2 / rhs2);
                    if (result.relative_residual <= tolerance) { result.converged = 1; break; }
                    rz = restart();
                    if (!(rz > 0) || !std::isfinite(rz)) break;
                    continue;
                }
                apply_preconditioner(s, s.r, s.z);
                ++result.preconditioner_applications;
                const double next_rz = device_dot(s, s.r, s.z);
                if (!(next_rz > 0) || !std::isfinite(next_rz)) break;
                const double beta = next_rz / rz;
                if (!std::isfinite(beta)) break;
                vec_update_direction(s, s.z, s.dvec, beta);
                rz = next_rz;
            }
            if (!result.converged)
            {
                residual2 = true_residual();
                result.relative_residual = std::sqrt(residual2 / rhs2);
                result.converged = std::isfinite(result.relative_residual) && result.relative_residual <= tolerance;
            }
            return result;
        }

        bool finite_value(double v) { return std::isfinite(v); }

        pcfd_solve_result solve_gcro(System& s, double* x, const double* b, double tolerance, int max_iterations, bool warm)
        {
            pcfd_solve_result result{};
            const int n = s.S;
            const size_t ld = size_t(s.Sp);   // stride of the multi-vector slots
            if (!warm)
            {
                s.recycle_count = 0;
                if (max_iterations > 0) vec_zero(s, x);
            }
            if (max_iterations <= 0) return result;
            const double rhs2 = device_dot(s, b, b);
            if (rhs2 == 0) { vec_zero(s, x); result.converged = 1; return result; }
            if (!std::isfinite(rhs2) || rhs2 < 0) { result.relative_residual = std::numeric_limits<double>::infinity(); return result; }
            auto true_residual = [&]() {
                launch_apply(s, x, s.Ad, false);
                return vec_residual_dot(s, b, s.Ad, s.defect);
            };
            auto ru = [&](int c) { return s.recycle_u.p + size_t(c) * ld; };
            auto rcv = [&](int c) { return s.recycle_c.p + size_t(c) * ld; };
            // device coefficient blocks of the fused CGS2 passes and their pinned host copies
            constexpr int kStride = kMaxSet + 1;
            double* h1 = s.block_result.p;
            double* h2 = h1 + kStride;
            double* h3 = h2 + kStride;
            const double* host_h1 = s.pinned_block;
            const double* host_h2 = host_h1 + kStride;
            const double* host_h3 = host_h2 + kStride;
            auto read_block = [&](int blocks) {
                cuda_check(cudaMemcpyAsync(s.pinned_block, s.block_result.p, size_t(blocks) * kStride * sizeof(double),
                                           cudaMemcpyDeviceToHost, s.stream), "coefficient readback");
                cuda_check(cudaStreamSynchronize(s.stream), "coefficient synchronize");
            };
            auto recycle_set = [&](double* base) {
                VecSet set{int64_t(ld)};
                for (int c = 0; c < s.recycle_count; ++c) set.push(base + size_t(c) * ld);
                return set;
            };
            double residual2 = true_residual();
            result.relative_residual = std::sqrt(residual2 / rhs2);
            if (result.relative_residual <= tolerance) { result.converged = 1; return result; }
            const int R = s.restart;
            while (result.iterations < max_iterations)
            {
                // minimise over the recycled space first; accept only if the true residual agrees
                const double before2 = residual2;
                const int attempted = s.recycle_count;
                bool valid = true;
                if (attempted)
                {
                    vec_copy_active(s, x, s.correction);
                    vec_copy_active(s, s.defect, s.t);
                    // two projections of the defect off C, correction += U h (CGS2, one readback)
                    const VecSet Cset = recycle_set(s.recycle_c.p), Uset = recycle_set(s.recycle_u.p);
                    block_dot(s, Cset, s.defect, h1);
                    block_update(s, Cset, h1, s.defect, Uset, 1.0, s.correction, 2, h2);
                    block_update(s, Cset, h2, s.defect, Uset, 1.0, s.correction, 0, nullptr);
                    read_block(2);
                    for (int c = 0; c < attempted && valid; ++c)
                        valid = finite_value(host_h1[c]) && finite_value(host_h2[c]);
                }
                double gap2 = 0, true_recycled2 = before2;
                if (attempted && valid)
                {
                    vec_copy_active(s, s.defect, s.r);
                    launch_apply(s, s.correction, s.Ad, false);
                    true_recycled2 = vec_residual_dot(s, b, s.Ad, s.defect);
                    vec_axpy_active(s, s.r, s.defect, -1.0);
                    gap2 = device_dot(s, s.r, s.r);
                }
                const double requested_gap = 0.25 * tolerance * std::sqrt(rhs2);
                const bool accurate = !attempted || (std::isfinite(gap2) && std::sqrt(gap2) <= requested_gap && true_recycled2 < before2);
                if (attempted && valid && accurate)
                {
                    vec_copy_active(s, s.correction, x);
                    residual2 = true_recycled2;
                }
                else if (attempted)
                {
                    s.recycle_count = 0;
                    vec_copy_active(s, s.t, s.defect);
                    residual2 = before2;
                }
                if (attempted && (!valid || !accurate)) ++result.recycle_rejections;
                result.relative_residual = std::sqrt(residual2 / rhs2);
                if (!std::isfinite(result.relative_residual)) break;
                if (result.relative_residual <= tolerance)
                {
                    residual2 = true_residual();
                    result.relative_residual = std::sqrt(residual2 / rhs2);
                    if (result.relative_residual <= tolerance) { result.converged = 1; break; }
                }
                const double beta = std::sqrt(residual2);
                if (!(beta > 0) || !std::isfinite(beta) || !std::isfinite(1.0 / beta)) break;
                const int cycle = std::min(R, max_iterations - result.iterations);
                std::vector<double> H(size_t(cycle + 1) * cycle, 0.0), cs(cycle), sn(cycle), g(cycle + 1, 0.0), y(cycle);
                std::vector<double> zc_recycle(size_t(cycle) * System::recycle_capacity, 0.0);   // deferred U coefficients
                g[0] = beta;
                vec_scaled_copy_active(s, s.gmres_v, s.defect, 1.0 / beta);
                int used = 0;
                // Column col + 1 needs nothing from the host's reading of column col except whether the
                // cycle ends there.  While the residual estimate, falling as it did last, stays at least
                // ten times the tolerance after column col, column col + 1 is enqueued before that wait,
                // so the device does not idle for the host's round trip and launches (a column on 65 k
                // cells: 109 -> 99 us, on 4.2 M: 611 -> 602).  A column enqueued in vain costs its device time and leaves
                // nothing that is read again.  The columns' work and order on the stream stay the
                // same.  Harvesting preconditioners and the learned ones count applications: no
                // column ahead there.
                const bool ahead = (s.preconditioner == PCFD_PRECONDITIONER_MULTIGRID || s.preconditioner == PCFD_PRECONDITIONER_JACOBI) &&
                                   !learned_harvesting(s);
                double estimate_now = beta, estimate_before = 10.0 * beta;   // first column: a fall by ten
                auto stays_above = [&]() {
                    return ahead && estimate_now * std::min(1.0, estimate_now / estimate_before) > 10.0 * tolerance * std::sqrt(rhs2);
                };
                if (s.delayed_orthogonalisation)
                {
                    // Delayed CGS2: column col's single pass pair reorthogonalises V_col (projected
                    // once in the previous column) and projects w = A z_col once; the previous
                    // column's Hessenberg entries and deferred C coefficients are corrected here by
                    // V_col's reorthogonalisation coefficients.  H is kept unrotated and the small
                    // least-squares problem is solved from scratch per column.
                    std::vector<double> Hu(size_t(cycle + 1) * cycle, 0.0);
                    const int cap = System::recycle_capacity;
                    double prev_rho = 0.0;
                    auto least_squares = [&](int cols, bool solve) {
                        std::vector<double> Rm(Hu.begin(), Hu.begin() + size_t(cols + 1) * cycle), gg(size_t(cols) + 1, 0.0);
                        std::vector<double> c_(static_cast<size_t>(cols)), s_(static_cast<size_t>(cols));
                        gg[0] = beta;
                        for (int j = 0; j < cols; ++j)
                        {
                            for (int i = 0; i < j; ++i)
                            {
                                double& a = Rm[size_t(i) * cycle + j];
                                double& bb = Rm[size_t(i + 1) * cycle + j];
                                const double rot = c_[i] * a + s_[i] * bb;
                                bb = -s_[i] * a + c_[i] * bb;
                                a = rot;
                            }
                            double& d = Rm[size_t(j) * cycle + j];
                            double& below = Rm[size_t(j + 1) * cycle + j];
                            const double norm = std::hypot(d, below);
                            if (!(norm > 0) || !std::isfinite(norm)) return std::numeric_limits<double>::quiet_NaN();
                            c_[j] = d / norm;
                            s_[j] = below / norm;
                            d = norm;
                            below = 0;
                            const double old = gg[j];
                            gg[j] = c_[j] * old;
                            gg[j + 1] = -s_[j] * old;
                        }
                        if (solve)
                            for (int row = cols - 1; row >= 0; --row)
                            {
                                double value = gg[row];
                                for (int col = row + 1; col < cols; ++col) value -= Rm[size_t(row) * cycle + col] * y[col];
                                y[row] = value / Rm[size_t(row) * cycle + row];
                                if (!std::isfinite(y[row])) return std::numeric_limits<double>::quiet_NaN();
                            }
                        return std::abs(gg[cols]);
                    };
                    // Column col's work (preconditioner, operator, both passes, which leave the
                    // coefficients in pinned host memory too) is enqueued as one unit.
                    const int k = s.recycle_count;
                    auto enqueue = [&](int col) {
                        double* v = s.gmres_v.p + size_t(col) * ld;
                        double* zc = s.gmres_z.p + size_t(col) * ld;
                        apply_preconditioner(s, v, zc);
                        launch_apply(s, zc, s.Ad, false);
                        VecSet Q = recycle_set(s.recycle_c.p);
                        for (int row = 0; row < col; ++row) Q.push(s.gmres_v.p + size_t(row) * ld);
                        dcgs_pass(s, Q, v, s.Ad, s.gmres_v.p + size_t(col + 1) * ld, s.dcgs_result,
                                  s.pinned_dcgs + size_t(col & 1) * kDcgsCoefficients);
                        cuda_check(cudaEventRecord(s.dcgs_ready[col & 1], s.stream), "coefficient event");
                    };
                    enqueue(0);
                    for (int col = 0, queued = 1; col < cycle; ++col)
                    {
                        if (col + 1 < cycle && stays_above())
                        {
                            enqueue(col + 1);
                            queued = col + 2;
                        }
                        cuda_check(cudaEventSynchronize(s.dcgs_ready[col & 1]), "coefficient synchronize");
                        ++result.preconditioner_applications;
                        const int m = k + col;
                        const double* cf = s.pinned_dcgs + size_t(col & 1) * kDcgsCoefficients;
                        const double* sc = cf + 4 * kMaxSet;
                        const double r = sc[3], c = sc[4], rho = sc[5];
                        bool ok = std::isfinite(r) && std::isfinite(c) && std::isfinite(rho);
                        for (int l = 0; l < m && ok; ++l) ok = std::isfinite(cf[l]) && std::isfinite(cf[kMaxSet + l]);
                        if (!ok) break;
                        if (col > 0)
                        {
                            for (int i = 0; i < col; ++i) Hu[size_t(i) * cycle + col - 1] += prev_rho * cf[k + i];
                            for (int cc = 0; cc < k; ++cc) zc_recycle[size_t(col - 1) * cap + cc] += prev_rho * cf[cc];
                            Hu[size_t(col) * cycle + col - 1] = prev_rho * r;
                        }
                        // V_col inside the span of the earlier vectors: the previous column closed
                        // the Krylov space, and this column is not used
                        if (!(r > 64 * std::numeric_limits<double>::epsilon() * std::sqrt(std::max(sc[0], 0.0))))
                        {
                            if (col > 0) Hu[size_t(col) * cycle + col - 1] = 0.0;
                            break;
                        }
                        for (int i = 0; i < col; ++i) Hu[size_t(i) * cycle + col] = cf[kMaxSet + k + i];
                        Hu[size_t(col) * cycle + col] = c;
                        double next_norm = rho;
                        if (!(next_norm > 64 * std::numeric_limits<double>::epsilon() * std::sqrt(std::max(sc[2], 0.0)))) next_norm = 0;
                        Hu[size_t(col + 1) * cycle + col] = next_norm;
                        for (int cc = 0; cc < k; ++cc) zc_recycle[size_t(col) * cap + cc] = cf[kMaxSet + cc];
                        used = col + 1;
                        ++result.iterations;
                        const double estimate = least_squares(used, false);
                        if (!std::isfinite(estimate)) { --used; --result.iterations; break; }
                        if (estimate / std::sqrt(rhs2) <= tolerance || next_norm == 0) break;
                        if (queued == col + 1 && col + 1 < cycle)
                        {
                            enqueue(col + 1);
                            queued = col + 2;
                        }
                        estimate_before = estimate_now;
                        estimate_now = estimate;
                        prev_rho = rho;
                    }
                    if (used == 0) break;
                    if (!std::isfinite(least_squares(used, true))) break;
                }
                else
                {
                    // Column col's work: CGS2 of w = A z against [C | V_0..V_col].  The matching z -= U h_C
                    // update is deferred: its coefficients are kept per column and applied once when
                    // the cycle's correction is formed (z only enters the solution through Z y).
                    // Coefficients and their host copies alternate between two sets of three blocks.
                    const int k = s.recycle_count;
                    auto enqueue = [&](int col) {
                        double* v = s.gmres_v.p + size_t(col) * ld;
                        double* zc = s.gmres_z.p + size_t(col) * ld;
                        apply_preconditioner(s, v, zc);
                        launch_apply(s, zc, s.Ad, false);
                        VecSet Q = recycle_set(s.recycle_c.p);
                        const VecSet none{int64_t(ld)};
                        for (int row = 0; row <= col; ++row) Q.push(s.gmres_v.p + size_t(row) * ld);
                        const size_t set = size_t(col & 1) * 3 * kStride;
                        double *b1 = h1 + set, *b2 = b1 + kStride, *b3 = b2 + kStride;
                        double* host = s.pinned_block + set;
                        block_dot(s, Q, s.Ad, b1, host);
                        block_update(s, Q, b1, s.Ad, none, -1.0, nullptr, 2, b2, host + kStride);
                        block_update(s, Q, b2, s.Ad, none, -1.0, nullptr, 1, b3, host + 2 * kStride);
                        scale_by_inverse_norm(s, s.gmres_v.p + size_t(col + 1) * ld, s.Ad, b3);
                        cuda_check(cudaEventRecord(s.dcgs_ready[col & 1], s.stream), "coefficient event");
                    };
                    enqueue(0);
                    for (int col = 0, queued = 1; col < cycle; ++col)
                    {
                        if (col + 1 < cycle && stays_above())
                        {
                            enqueue(col + 1);
                            queued = col + 2;
                        }
                        cuda_check(cudaEventSynchronize(s.dcgs_ready[col & 1]), "coefficient synchronize");
                        ++result.preconditioner_applications;
                        const int m = k + col + 1;
                        const double* host_h1 = s.pinned_block + size_t(col & 1) * 3 * kStride;
                        const double* host_h2 = host_h1 + kStride;
                        const double* host_h3 = host_h2 + kStride;
                        bool column_valid = true;
                        for (int j = 0; j < m && column_valid; ++j) column_valid = finite_value(host_h1[j]) && finite_value(host_h2[j]);
                        if (!column_valid) break;
                        double c_part = 0;
                        for (int c = 0; c < k; ++c) c_part += host_h1[c] * host_h1[c];
                        const double scale = std::sqrt(std::max(0.0, host_h1[m] - c_part));
                        if (!(scale > 0) || !std::isfinite(scale)) break;
                        for (int row = 0; row <= col; ++row) H[size_t(row) * cycle + col] = host_h1[k + row] + host_h2[k + row];
                        for (int c = 0; c < k; ++c) zc_recycle[size_t(col) * System::recycle_capacity + c] = host_h1[c] + host_h2[c];
                        double next_norm = std::sqrt(std::max(0.0, host_h3[0]));
                        const double floor = 64 * std::numeric_limits<double>::epsilon() * scale;
                        if (!(next_norm > floor && std::isfinite(1.0 / next_norm))) next_norm = 0;
                        H[size_t(col + 1) * cycle + col] = next_norm;
                        for (int row = 0; row < col; ++row)
                        {
                            double& a = H[size_t(row) * cycle + col];
                            double& bb = H[size_t(row + 1) * cycle + col];
                            const double rot = cs[row] * a + sn[row] * bb;
                            bb = -sn[row] * a + cs[row] * bb;
                            a = rot;
                        }
                        double& diag = H[size_t(col) * cycle + col];
                        double& below = H[size_t(col + 1) * cycle + col];
                        const double norm = std::hypot(diag, below);
                        if (!(norm > 0) || !std::isfinite(norm)) break;
                        cs[col] = diag / norm;
                        sn[col] = below / norm;
                        diag = norm;
                        below = 0;
                        const double old = g[col];
                        g[col] = cs[col] * old;
                        g[col + 1] = -sn[col] * old;
                        used = col + 1;
                        ++result.iterations;
                        if (std::abs(g[col + 1]) / std::sqrt(rhs2) <= tolerance || next_norm == 0) break;
                        if (queued == col + 1 && col + 1 < cycle)
                        {
                            enqueue(col + 1);
                            queued = col + 2;
                        }
                        estimate_before = estimate_now;
                        estimate_now = std::abs(g[col + 1]);
                    }
                    if (used == 0) break;
                    for (int row = used - 1; row >= 0; --row)
                    {
                        double value = g[row];
                        for (int col = row + 1; col < used; ++col) value -= H[size_t(row) * cycle + col] * y[col];
                        const double d = H[size_t(row) * cycle + row];
                        if (!(std::abs(d) > 0) || !std::isfinite(d)) { used = 0; break; }
                        y[row] = value / d;
                        if (!std::isfinite(y[row])) { used = 0; break; }
                    }
                    if (used == 0) break;
                }
                {
                    // correction = sum_j y_j (z_j - U c_j) = Z y - U (sum_j y_j c_j)
                    VecSet Z{int64_t(ld)};
                    Coefficients coefficient;
                    for (int col = 0; col < used; ++col)
                    {
                        Z.push(s.gmres_z.p + size_t(col) * ld);
                        coefficient.value[col] = y[col];
                    }
                    for (int c = 0; c < s.recycle_count; ++c)
                    {
                        double sum = 0.0;
                        for (int col = 0; col < used; ++col) sum += y[col] * zc_recycle[size_t(col) * System::recycle_capacity + c];
                        Z.push(ru(c));
                        coefficient.value[used + c] = -sum;
                    }
                    block_combine(s, Z, coefficient, s.correction, false);
                }
                vec_axpy_active(s, x, s.correction, 1.0);
                residual2 = true_residual();
                result.relative_residual = std::sqrt(residual2 / rhs2);
                if (!std::isfinite(result.relative_residual)) break;
                if (s.recycle_limit <= 0)
                {
                    if (result.relative_residual <= tolerance) { result.converged = 1; break; }
                    continue;
                }
                // store a normalised (U, C = A U) pair when it adds a resolved direction
                launch_apply(s, s.correction, s.Ad, false);
                {
                    const VecSet Cset = recycle_set(s.recycle_c.p), Uset = recycle_set(s.recycle_u.p);
                    block_dot(s, Cset, s.Ad, h1);
                    block_update(s, Cset, h1, s.Ad, Uset, -1.0, s.correction, 2, h2);
                    block_update(s, Cset, h2, s.Ad, Uset, -1.0, s.correction, 1, h3);
                    read_block(3);
                }
                const int kc = s.recycle_count;
                const double cand_before = std::sqrt(std::max(0.0, host_h1[kc]));
                bool cand_valid = cand_before > 0 && std::isfinite(cand_before);
                for (int c = 0; c < kc && cand_valid; ++c) cand_valid = finite_value(host_h1[c]) && finite_value(host_h2[c]);
                const double cand_after = cand_valid ? std::sqrt(std::max(0.0, host_h3[0])) : 0;
                cand_valid = cand_valid && std::isfinite(cand_after) && cand_after > 1e-12 * cand_before && std::isfinite(1.0 / cand_after);
                if (cand_valid)
                {
                    if (s.recycle_count >= s.recycle_limit)
                    {
                        for (int c = 1; c < s.recycle_count; ++c)
                        {
                            cuda_check(cudaMemcpyAsync(ru(c - 1), ru(c), size_t(n) * sizeof(double), cudaMemcpyDeviceToDevice, s.stream), "shift recycle");
                            cuda_check(cudaMemcpyAsync(rcv(c - 1), rcv(c), size_t(n) * sizeof(double), cudaMemcpyDeviceToDevice, s.stream), "shift recycle");
                        }
                        --s.recycle_count;
                    }
                    vec_scaled_copy_active(s, ru(s.recycle_count), s.correction, 1.0 / cand_after);
                    vec_scaled_copy_active(s, rcv(s.recycle_count), s.Ad, 1.0 / cand_after);
                    ++s.recycle_count;
                }
                if (result.relative_residual <= tolerance) { result.converged = 1; break; }
            }
            if (!result.converged)
            {
                residual2 = true_residual();
                result.relative_residual = std::sqrt(residual2 / rhs2);
                result.converged = std::isfinite(result.relative_residual) && result.relative_residual <= tolerance;
            }
            return result;
        }
    }

    pcfd_solve_result solve(System& s, double* x, const double* b, double tolerance, int max_iterations, bool warm)
    {
        // the learned preconditioner is not a fixed linear map: it always runs under the flexible
        // GCRO/LGMRES recurrence, with the multigrid solve from its last iterate as the fallback
        const bool learned = s.preconditioner == PCFD_PRECONDITIONER_LEARNED || s.preconditioner == PCFD_PRECONDITIONER_LEARNED_MULTIGRID;
        if (learned)
        {
            pcfd_solve_result result = solve_gcro(s, x, b, tolerance, max_iterations, warm);
            learned_check(s);
            if (result.converged) return result;
            const int kind = s.preconditioner;
            s.preconditioner = PCFD_PRECONDITIONER_MULTIGRID;
            pcfd_solve_result fallback{};
            try
            {
                fallback = solve(s, x, b, tolerance, max_iterations, true);
            }
            catch (...)
            {
                s.preconditioner = kind;
                throw;
            }
            s.preconditioner = kind;
            fallback.iterations += result.iterations;
            fallback.preconditioner_applications += result.preconditioner_applications;
            fallback.fallback_solves = 1;
            return fallback;
        }
        if (!s.full_nonorthogonal)
        {
            // One continuous MG-PCG solve with a 5x iteration budget, then the final defect
            // (reference amr_pressure.cu:1361-1389).
            const double rhs2 = device_dot(s, b, b);
            const int budget = max_iterations > std::numeric_limits<int>::max() / 5 ? max_iterations : 5 * max_iterations;
            pcfd_solve_result result = solve_orthogonal(s, x, b, tolerance, budget, warm);
            if (!(rhs2 > 0) || !std::isfinite(rhs2)) return result;
            launch_apply(s, x, s.Ad, true);
            result.relative_residual = std::sqrt(vec_residual_dot(s, b, s.Ad, s.defect) / rhs2);
            result.converged = std::isfinite(result.relative_residual) && result.relative_residual <= tolerance;
            return result;
        }
        return solve_gcro(s, x, b, tolerance, max_iterations, warm);
    }
}
