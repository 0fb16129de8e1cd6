// stage_tail.cu -- the small levels of a multigrid hierarchy as one thread-block cluster.
//
// Below some 30 k rows a level's smoothing step is pure latency: launched one after the other (even
// chained with programmatic dependent launch) each step, residual, restriction and prolongation
// costs 2.6 us whatever its size, and a V-cycle makes 20-60 of them per application.  Here the
// smallest levels of the chain run as ONE launch of one cluster (16 CTAs, each on its own SM of
// one GPC).  Every CTA owns a contiguous run of each level's rows and keeps that run's matrix,
// diagonal, right-hand side, iterate and direction in shared memory for the whole cycle;
// neighbours' iterates are read through distributed shared memory, and a hardware cluster barrier
// separates the phases.  Levels of at most kSoloRows rows stay on CTA 0, whose phases need only a
// CTA barrier.  The coarsest level is its explicit inverse, rows spread over the CTAs, or its Jacobi
// sweeps on CTA 0.
//
// Layout, and why:
//   * a CTA's matrix slices are one contiguous image, built at setup and copied with 16-byte loads
//     (gathering them from the CSR arrays took 6 of 39 us);
//   * a row holds six entries in fixed slots (entry-major, so a warp reads consecutive words) whose
//     loads are all in flight together; the few rows with more walk a list.  A CSR loop's
//     remainder iterations each waited for their own neighbour (2.0-2.5 k cycles a step of 512 rows);
//   * matrix and iterate are kept as doubles: the sums are FP64, and converting every FP32 or FP16
//     operand (16 per cycle and SM) costs more than the sums themselves.  The iterate's values
//     are rounded to T as before, so the arithmetic is that of the per-launch kernels (solver.cu), with
//     each level's couplings as that level stores them (the coarsest's never in FP16): FP64 row
//     sums in CSR order (a brick-structured first stage sums its faces first when it is launched
//     alone), d = c1 d + c2 D^-1 (b - A x), x += d (damped Jacobi is c1 = 0, c2 = omega), the first
//     step of a correction from x = 0 without the matrix.
//
// Which levels: the longest run of levels at the coarse end whose rows fit kTailRows and whose
// slices fit the CTAs' shared memory.
//
// Measured, one preconditioner application (CUDA events, back to back), before -> with this launch:
// composite cycle with FP16 stages 70 -> 49 us on 65 k cells (8,192 rows here), 178 -> 164 on
// 1.1 M (19.8 k), 328 -> 295 on 4.2 M (9.0 k), 936 -> 889 on 16 M (4.4 k); reference cycle in FP64
// 258 -> 149 us on 524 k cells and 296 -> 186 on 1.1 M, where the coarsest sweeps were 85.
#include "pcfd_internal.h"

#include <cuda_fp16.h>

#include <algorithm>
#include <cmath>
#include <cstring>

namespace pcfd
{
    namespace
    {
        constexpr int kTailLevels = 10, kTailSteps = 16, kSlots = 6;
        // A level on one CTA needs no cluster barrier (0.25 us) but has only its FP64 units (64 per
        // cycle): with more rows than this the spread-out phase is the shorter one.
        constexpr int kSoloRows = 192;
        // Above, a thread owns more than two rows and a launch on all 148 SMs is the shorter one.
        constexpr int kTailRows = 32768;
        constexpr int kCoarsestRows = 512;               // inverse, or sweeps with a row per thread
        constexpr int kTailShared = 220 * 1024;          // beside the 4 KiB static right-hand side

        // One level's slice of a CTA: byte offsets into its shared memory.  Static arrays (the image):
        // diagonal, slot coefficients and columns, extra entries, parents, members of the rows.
        // Working arrays: right-hand side, iterate (two buffers), direction / residual.
        struct TailLevel
        {
            int cells, chunk;               // rows; rows per CTA (all rows on a solo level)
            int diagonal, coefficient, column, extra, extra_coefficient, extra_column, parent, first, member;
            int b, x, d;
        };
        template <class T> struct TailArgs
        {
            TailLevel level[kTailLevels];
            int count, steps, image, coarsest_sweeps;   // image: static bytes per CTA; sweeps: without an inverse
            const uint4* images;
            const T *rhs, *dense;
            T* x;
            T c1[kTailSteps], c2[kTailSteps], prolong[kTailLevels], omega;
        };

        __device__ inline void cluster_barrier()
        {
            asm volatile("barrier.cluster.arrive.release;\n\tbarrier.cluster.wait.acquire;" ::: "memory");
        }
        // the address in CTA `rank`'s shared memory of what is at `p` in this CTA's
        template <class V> __device__ inline const V* at_rank(const V* p, unsigned rank)
        {
            uint64_t out;
            asm("mapa.u64 %0, %1, %2;" : "=l"(out) : "l"(reinterpret_cast<uint64_t>(p)), "r"(rank));
            return reinterpret_cast<const V*>(out);
        }
        // value of a row packed as (owning CTA << 24) | (row in its slice)
        template <class V> __device__ inline V row_value(const V* slice, unsigned row) { return *at_rank(slice + (row & 0xffffffu), row >> 24); }

        __device__ inline float fused(float a, float b, float c) { return __fmaf_rn(a, b, c); }
        __device__ inline double fused(double a, double b, double c) { return __fma_rn(a, b, c); }
        __device__ inline float product(float a, float b) { return __fmul_rn(a, b); }
        __device__ inline double product(double a, double b) { return __dmul_rn(a, b); }
        __device__ inline float sum(float a, float b) { return __fadd_rn(a, b); }
        __device__ inline double sum(double a, double b) { return __dadd_rn(a, b); }

        // Bound by the latency of a phase: shared-memory and cluster round trips, one FP64 division
        // and the cluster barrier.
        template <class T>
        __global__ void __launch_bounds__(1024, 1) stage_tail_kernel(const __grid_constant__ TailArgs<T> a)
        {
            extern __shared__ __align__(16) unsigned char shared[];
            __shared__ T full[kCoarsestRows];       // the coarsest level's whole right-hand side
            const int me = int(blockIdx.x), tid = int(threadIdx.x), width = int(blockDim.x);
            const int last = a.count - 1;
            auto values = [&](int offset) { return reinterpret_cast<T*>(shared + offset); };
            auto doubles = [&](int offset) { return reinterpret_cast<double*>(shared + offset); };
            auto ints = [&](int offset) { return reinterpret_cast<const int*>(shared + offset); };
            auto rows_of = [&](const TailLevel& l) { return max(0, min(l.chunk, l.cells - me * l.chunk)); };
            auto solo = [&](int l) { return a.level[l].chunk >= a.level[l].cells; };

            // the static part does not depend on the previous kernel
            const uint4* image = a.images + int64_t(me) * (a.image / 16);
            for (int q = tid; q < a.image / 16; q += width) reinterpret_cast<uint4*>(shared)[q] = image[q];
            chain_wait();
            chain_release();
            {
                const TailLevel& level = a.level[0];
                const int rows = rows_of(level), r0 = me * level.chunk;
                for (int r = tid; r < rows; r += width) values(level.b)[r] = a.rhs[r0 + r];
            }
            __syncthreads();

            auto barrier = [&](int l) {
                if (solo(l)) __syncthreads();
                else cluster_barrier();
            };
            // A x of slice row r, x: this CTA's part of the iterate
            auto row_product = [&](const TailLevel& level, const double* x, int r, double dq) {
                const int* column = ints(level.column) + r;
                const double* coefficient = doubles(level.coefficient) + r;
                double v[kSlots];
#pragma unroll
                for (int e = 0; e < kSlots; ++e) v[e] = row_value(x, unsigned(column[e * level.chunk]));
                double Ax = __dmul_rn(dq, x[r]);
#pragma unroll
                for (int e = 0; e < kSlots; ++e) Ax = __fma_rn(-coefficient[e * level.chunk], v[e], Ax);
                const int extra = ints(level.extra)[r];
                for (int e = extra >> 8, e1 = e + (extra & 255); e < e1; ++e)
                    Ax = __fma_rn(-doubles(level.extra_coefficient)[e], row_value(x, unsigned(ints(level.extra_column)[e])), Ax);
                return Ax;
            };
            auto buffer = [&](const TailLevel& level, int which) { return doubles(level.x) + which * level.chunk; };
            // steps [from, to) of a smoothing pass; `which` is the buffer of the current iterate
            auto smooth = [&](int l, int from, int& which) {
                const TailLevel& level = a.level[l];
                const int rows = rows_of(level);
                for (int step = from; step < a.steps; ++step)
                {
                    const T c1 = a.c1[step], c2 = a.c2[step];
                    const double* x = buffer(level, which);
                    double* next = buffer(level, which ^ 1);
                    for (int r = tid; r < rows; r += width)
                    {
                        const double dq = doubles(level.diagonal)[r];
                        T dn = T(0), xn = T(0);
                        if (dq > 0.0)
                        {
                            const T move = T((double(values(level.b)[r]) - row_product(level, x, r, dq)) / dq);
                            if (a.omega > T(0)) xn = fused(a.omega, move, T(x[r]));
                            else
                            {
                                dn = product(c2, move);
                                if (step) dn = fused(c1, values(level.d)[r], dn);
                                xn = sum(T(x[r]), dn);
                            }
                        }
                        values(level.d)[r] = dn;
                        next[r] = double(xn);
                    }
                    which ^= 1;
                    barrier(l);
                }
            };

            unsigned current = 0;            // bit l: buffer of level l's iterate
            for (int l = 0; l < last; ++l)
            {
                const TailLevel& level = a.level[l];
                const int rows = rows_of(level);
                if (!solo(l) || me == 0)
                {
                    // the first step from zero; it writes buffer 1, so that an even number of steps ends in 0
                    double* x = buffer(level, 1);
                    const T c2 = a.omega > T(0) ? a.omega : a.c2[0];
                    for (int r = tid; r < rows; r += width)
                    {
                        const double dq = doubles(level.diagonal)[r];
                        const T move = dq > 0.0 ? product(c2, T(double(values(level.b)[r]) / dq)) : T(0);
                        values(level.d)[r] = move;
                        x[r] = double(move);
                    }
                    int which = 1;
                    barrier(l);
                    smooth(l, 1, which);
                    const double* xs = buffer(level, which);
                    for (int r = tid; r < rows; r += width)
                    {
                        const double dq = doubles(level.diagonal)[r];
                        values(level.d)[r] = dq > 0.0 ? T(double(values(level.b)[r]) - row_product(level, xs, r, dq)) : T(0);
                    }
                    if (which) current |= 1u << l;
                }
                // the next level's right-hand side needs this level's residuals
                if (solo(l) && solo(l + 1)) { if (me == 0) __syncthreads(); }
                else cluster_barrier();
                const TailLevel& coarse = a.level[l + 1];
                const int crows = rows_of(coarse);
                const T* residual = values(level.d);
                for (int r = tid; r < crows; r += width)
                {
                    double total = 0.0;
#pragma unroll 8
                    for (int q = ints(coarse.first)[r], q1 = ints(coarse.first)[r + 1]; q < q1; ++q)
                        total += double(row_value(residual, unsigned(ints(coarse.member)[q])));
                    values(coarse.b)[r] = T(total);
                }
            }
            if (a.dense)
            {
                // coarsest level: x = inverse * b, one warp per row (FP64 sums), rows spread over the CTAs
                const TailLevel& level = a.level[last];
                cluster_barrier();
                for (int q = tid; q < level.cells; q += width)
                    full[q] = row_value(values(level.b), (unsigned(q / level.chunk) << 24) | unsigned(q % level.chunk));
                __syncthreads();
                const int rows = rows_of(level), lane = tid & 31;
                for (int r = tid >> 5; r < rows; r += width / 32)
                {
                    const T* matrix = a.dense + int64_t(me * level.chunk + r) * level.cells;
                    double total = 0.0;
#pragma unroll 4
                    for (int j = lane; j < level.cells; j += 32) total = __fma_rn(double(matrix[j]), double(full[j]), total);
                    for (int o = 16; o > 0; o >>= 1) total += __shfl_down_sync(0xffffffffu, total, o);
                    if (lane == 0) doubles(level.x)[r] = double(T(total));
                }
                cluster_barrier();
            }
            else
            {
                // the coarsest level's damped Jacobi sweeps from zero on CTA 0, a row per thread with its
                // slots in registers (the same sweeps through global memory in one CTA: 85 us for 128 rows)
                const TailLevel& level = a.level[last];
                if (me == 0)
                {
                    const int r = tid;
                    const bool on = r < level.cells;
                    unsigned column[kSlots];
                    double coefficient[kSlots];
                    const double dq = on ? doubles(level.diagonal)[r] : 0.0, bq = on ? double(values(level.b)[r]) : 0.0;
#pragma unroll
                    for (int e = 0; e < kSlots; ++e)
                    {
                        column[e] = on ? unsigned(ints(level.column)[e * level.chunk + r]) : 0u;
                        coefficient[e] = on ? doubles(level.coefficient)[e * level.chunk + r] : 0.0;
                    }
                    const int extra = on ? ints(level.extra)[r] : 0;
                    double xq = 0.0;
                    if (on) buffer(level, 0)[r] = 0.0;
                    __syncthreads();
                    for (int sweep = 0; sweep < a.coarsest_sweeps; ++sweep)
                    {
                        const double* x = buffer(level, sweep & 1);
                        if (on)
                        {
                            double v[kSlots];
#pragma unroll
                            for (int e = 0; e < kSlots; ++e) v[e] = x[column[e]];
                            double Ax = __dmul_rn(dq, xq);
#pragma unroll
                            for (int e = 0; e < kSlots; ++e) Ax = __fma_rn(-coefficient[e], v[e], Ax);
                            for (int e = extra >> 8, e1 = e + (extra & 255); e < e1; ++e)
                                Ax = __fma_rn(-doubles(level.extra_coefficient)[e], x[ints(level.extra_column)[e]], Ax);
                            xq = dq > 0.0 ? double(fused(a.prolong[last], T((bq - Ax) / dq), T(xq))) : 0.0;
                            buffer(level, (sweep & 1) ^ 1)[r] = xq;
                        }
                        __syncthreads();
                    }
                    if (a.coarsest_sweeps & 1)
                    {
                        if (on) buffer(level, 0)[r] = xq;
                        __syncthreads();
                    }
                }
                if (!solo(last - 1)) cluster_barrier();
            }
            for (int l = last - 1; l >= 0; --l)
            {
                const TailLevel& level = a.level[l];
                const TailLevel& coarse = a.level[l + 1];
                const int rows = rows_of(level);
                if (!solo(l) || me == 0)
                {
                    int which = int(current >> l & 1u);
                    double* x = buffer(level, which);
                    // the coarser level's iterate ends in its buffer 0
                    for (int r = tid; r < rows; r += width)
                    {
                        const int p = ints(level.parent)[r];
                        if (p >= 0) x[r] = double(fused(a.prolong[l], T(row_value(doubles(coarse.x), unsigned(p))), T(x[r])));
                    }
                    barrier(l);
                    smooth(l, 0, which);
                }
                // a finer level on all CTAs reads a solo level's iterate after a cluster barrier
                if (l > 0 && solo(l) && !solo(l - 1)) cluster_barrier();
            }
            {
                const TailLevel& level = a.level[0];
                const int rows = rows_of(level), r0 = me * level.chunk;
                for (int r = tid; r < rows; r += width) a.x[r0 + r] = T(doubles(level.x)[r]);
            }
            // no CTA leaves while another may still read its shared memory
            cluster_barrier();
        }

        // CTAs of the cluster that the device schedules for this kernel and shared memory: 16, else the
        // portable 8, else none
        template <class T> int cluster_ranks(int shared, int threads)
        {
            auto kernel = stage_tail_kernel<T>;
            // the same limit for every system, so that planning one never lowers another's
            if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kTailShared) != cudaSuccess ||
                cudaFuncSetAttribute(kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) != cudaSuccess)
            {
                cudaGetLastError();
                return 0;
            }
            for (int ranks : {16, 8})
            {
                cudaLaunchConfig_t config{};
                config.gridDim = dim3(unsigned(ranks));
                config.blockDim = dim3(unsigned(threads));
                config.dynamicSmemBytes = size_t(shared);
                cudaLaunchAttribute attribute{};
                attribute.id = cudaLaunchAttributeClusterDimension;
                attribute.val.clusterDim.x = unsigned(ranks);
                attribute.val.clusterDim.y = attribute.val.clusterDim.z = 1;
                config.attrs = &attribute;
                config.numAttrs = 1;
                int clusters = 0;
                if (cudaOccupancyMaxActiveClusters(&clusters, kernel, &config) == cudaSuccess && clusters > 0) return ranks;
                cudaGetLastError();
            }
            return 0;
        }

        // Slices of levels [first, count) on `ranks` CTAs; false when they do not fit.
        template <class T>
        bool tail_layout(const std::vector<HostRows>& rows, int first, int ranks, bool dense, TailArgs<T>& a, int& bytes)
        {
            const int count = int(rows.size());
            if (count - first < 2 || count - first > kTailLevels || rows[size_t(first)].cells > kTailRows) return false;
            if (rows[size_t(count) - 1].cells > kCoarsestRows) return false;
            a.count = count - first;
            int64_t at = 0;
            bool fits = true;
            auto take = [&](int64_t size) {
                const int64_t offset = at;
                at += (size + 15) & ~int64_t(15);
                fits = fits && at <= kTailShared;
                return fits ? int(offset) : 0;
            };
            for (int k = 0; k < a.count; ++k)
            {
                TailLevel& l = a.level[k];
                const HostRows& h = rows[size_t(first + k)];
                const bool coarsest = k + 1 == a.count, matrix = !coarsest || !dense;
                l.cells = h.cells;
                l.chunk = h.cells <= kSoloRows || (coarsest && !dense) ? h.cells : (h.cells + ranks - 1) / ranks;
                if (coarsest && dense) l.chunk = (h.cells + ranks - 1) / ranks;
                int64_t extra = 0, members = 0;
                for (int r0 = 0; r0 < h.cells; r0 += l.chunk)
                {
                    const int r1 = std::min(h.cells, r0 + l.chunk);
                    int64_t here = 0;
                    for (int r = r0; r < r1; ++r)
                    {
                        const int more = (*h.row_offset)[size_t(r) + 1] - (*h.row_offset)[size_t(r)] - kSlots;
                        if (more > 255) return false;
                        here += std::max(0, more);
                    }
                    extra = std::max(extra, here);
                    if (k > 0)
                    {
                        const std::vector<int>& m = *rows[size_t(first + k) - 1].member_offset;
                        members = std::max<int64_t>(members, m[size_t(r1)] - m[size_t(r0)]);
                    }
                }
                const int64_t n = l.chunk;
                if (matrix)
                {
                    l.diagonal = take(8 * n);
                    l.coefficient = take(8 * kSlots * n);
                    l.column = take(4 * kSlots * n);
                    l.extra = take(4 * n);
                    l.extra_coefficient = take(8 * extra);
                    l.extra_column = take(4 * extra);
                }
                if (!coarsest) l.parent = take(4 * n);
                if (k > 0)
                {
                    l.first = take(4 * (n + 1));
                    l.member = take(4 * members);
                }
            }
            a.image = fits ? int(at) : 0;
            for (int k = 0; k < a.count; ++k)
            {
                TailLevel& l = a.level[k];
                l.b = take(int64_t(sizeof(T)) * l.chunk);
                l.x = take(16 * int64_t(l.chunk));
                l.d = take(int64_t(sizeof(T)) * l.chunk);
            }
            bytes = int(at);
            return fits;
        }

        // a matrix coefficient as the kernels' storage type holds it
        template <class T> double stored(double weight, bool half)
        {
            if (half) return double(__half2float(__float2half_rn(float(weight))));
            return double(T(weight));
        }

        // the CTAs' images.  half_stages: FP16 couplings, on every level but the coarsest, whose sweeps need them
        // to add up to the diagonal (a closed domain's coarsest operator is singular)
        template <class T> std::vector<unsigned char> images(const std::vector<HostRows>& rows, int first, int ranks, bool dense, bool half_stages, const TailArgs<T>& a)
        {
            std::vector<unsigned char> out(size_t(ranks) * size_t(a.image), 0);
            auto put = [&](int rank, int offset, int64_t index, auto value) {
                std::memcpy(out.data() + size_t(rank) * a.image + size_t(offset) + size_t(index) * sizeof(value), &value, sizeof(value));
            };
            auto packed = [](int row, int chunk) { return int((unsigned(row / chunk) << 24) | unsigned(row % chunk)); };
            for (int k = 0; k < a.count; ++k)
            {
                const TailLevel& l = a.level[k];
                const HostRows& h = rows[size_t(first + k)];
                const bool coarsest = k + 1 == a.count, matrix = !coarsest || !dense, half = half_stages && !coarsest;
                for (int r0 = 0, rank = 0; r0 < h.cells; r0 += l.chunk, ++rank)
                {
                    int extras = 0, members = 0;
                    const int r1 = std::min(h.cells, r0 + l.chunk);
                    for (int q = r0; q < r1; ++q)
                    {
                        const int r = q - r0;
                        if (matrix)
                        {
                            put(rank, l.diagonal, r, double(T((*h.diagonal)[size_t(q)])));
                            const int e0 = (*h.row_offset)[size_t(q)], n = (*h.row_offset)[size_t(q) + 1] - e0;
                            for (int e = 0; e < kSlots; ++e)
                            {
                                const bool in = e < n;
                                put(rank, l.coefficient, int64_t(e) * l.chunk + r, in ? stored<T>((*h.weight)[size_t(e0 + e)], half) : 0.0);
                                put(rank, l.column, int64_t(e) * l.chunk + r, packed(in ? (*h.neighbour)[size_t(e0 + e)] : q, l.chunk));
                            }
                            put(rank, l.extra, r, (extras << 8) | std::max(0, n - kSlots));
                            for (int e = kSlots; e < n; ++e, ++extras)
                            {
                                put(rank, l.extra_coefficient, extras, stored<T>((*h.weight)[size_t(e0 + e)], half));
                                put(rank, l.extra_column, extras, packed((*h.neighbour)[size_t(e0 + e)], l.chunk));
                            }
                        }
                        if (!coarsest)
                        {
                            const int p = (*h.parent)[size_t(q)];
                            put(rank, l.parent, r, p >= 0 ? packed(p, a.level[k + 1].chunk) : -1);
                        }
                        if (k > 0)
                        {
                            const HostRows& finer = rows[size_t(first + k) - 1];
                            put(rank, l.first, r, members);
                            for (int m = (*finer.member_offset)[size_t(q)]; m < (*finer.member_offset)[size_t(q) + 1]; ++m, ++members)
                                put(rank, l.member, members, packed((*finer.member)[size_t(m)], a.level[k - 1].chunk));
                        }
                    }
                    if (k > 0) put(rank, l.first, r1 - r0, members);
                }
            }
            return out;
        }
    }

    // A hierarchy's cluster launch: its arguments and images.
    struct TailPlan
    {
        int ranks = 0, threads = 0, shared = 0;
        TailArgs<float> a32{};
        TailArgs<double> a64{};
        DBuf<unsigned char> image;
        template <class T> TailArgs<T>& args();
    };
    template <> TailArgs<float>& TailPlan::args<float>() { return a32; }
    template <> TailArgs<double>& TailPlan::args<double>() { return a64; }

    namespace
    {
        template <class T> void plan(std::vector<MgLevel<T>>& levels, const std::vector<HostRows>& rows, int coarsest_sweeps, double omega, StageTail& tail)
        {
            tail.first = -1;
            if (levels.empty() || levels.front().sweeps < 1 || levels.front().sweeps > kTailSteps) return;
            const MgLevel<T>& front = levels.front();
            const bool dense = levels.back().inverse.p != nullptr;
            for (int first = 0; first + 1 < int(levels.size()); ++first)
                for (int ranks : {16, 8})
                {
                    TailArgs<T> a{};
                    int bytes = 0;
                    if (!tail_layout<T>(rows, first, ranks, dense, a, bytes)) continue;
                    int threads = 128;      // enough for a row per thread, also of a level on one CTA
                    for (int k = 0; k < a.count; ++k) threads = std::max(threads, std::min(1024, (a.level[k].chunk + 31) / 32 * 32));
                    if (cluster_ranks<T>(bytes, threads) < ranks) continue;
                    a.steps = front.sweeps;
                    a.coarsest_sweeps = coarsest_sweeps;
                    a.omega = front.chebyshev >= 2 ? T(0) : T(omega);
                    const std::vector<std::pair<double, double>> steps = smoothing_steps(front.chebyshev, front.sweeps);
                    for (int k = 0; k < a.steps; ++k)
                    {
                        a.c1[k] = T(steps[size_t(k)].first);
                        a.c2[k] = T(steps[size_t(k)].second);
                    }
                    for (int k = 0; k + 1 < a.count; ++k) a.prolong[k] = T(levels[size_t(first + k)].prolong);
                    a.prolong[a.count - 1] = T(omega);      // the coarsest level's sweeps
                    a.dense = levels.back().inverse;
                    auto plan = std::make_shared<TailPlan>();
                    plan->image.upload(images<T>(rows, first, ranks, dense, front.coefficient16.p != nullptr, a));
                    a.images = reinterpret_cast<const uint4*>(plan->image.p);
                    plan->ranks = ranks;
                    plan->threads = threads;
                    plan->shared = bytes;
                    plan->args<T>() = a;
                    tail.first = first;
                    tail.plan = std::move(plan);
                    return;
                }
        }

        template <class T> void launch(System& s, MgLevel<T>& level, const StageTail& tail)
        {
            TailPlan& p = *tail.plan;
            TailArgs<T> a = p.args<T>();
            a.rhs = level.rhs;
            a.x = level.x;
            cudaLaunchConfig_t config{};
            config.gridDim = dim3(unsigned(p.ranks));
            config.blockDim = dim3(unsigned(p.threads));
            config.dynamicSmemBytes = size_t(p.shared);
            config.stream = launch_stream(s);
            cudaLaunchAttribute attribute[2]{};
            attribute[0].id = cudaLaunchAttributeClusterDimension;
            attribute[0].val.clusterDim.x = unsigned(p.ranks);
            attribute[0].val.clusterDim.y = attribute[0].val.clusterDim.z = 1;
            attribute[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
            attribute[1].val.programmaticStreamSerializationAllowed = 1;
            config.attrs = attribute;
            config.numAttrs = 2;
            cuda_check(cudaLaunchKernelEx(&config, stage_tail_kernel<T>, a), "stage tail");
        }
    }

    void plan_tail(std::vector<MgLevel<double>>& levels, const std::vector<HostRows>& rows, int coarsest_sweeps, double omega, StageTail& tail)
    {
        plan(levels, rows, coarsest_sweeps, omega, tail);
    }
    void plan_tail(std::vector<MgLevel<float>>& levels, const std::vector<HostRows>& rows, int coarsest_sweeps, double omega, StageTail& tail)
    {
        plan(levels, rows, coarsest_sweeps, omega, tail);
    }
    void launch_tail(System& s, MgLevel<double>& level, const StageTail& tail) { launch(s, level, tail); }
    void launch_tail(System& s, MgLevel<float>& level, const StageTail& tail) { launch(s, level, tail); }
}
