// pressure.cu -- FP64 composite pressure operator, deterministic reductions, the
// reference-structured multigrid preconditioner and the outer Krylov solvers.
//
// Operator semantics follow CompositeAmrPressureSystem::apply_cpu / diagonal_cpu
// (reference src/core/fluid/amr_pressure.cpp:498-543) with FP64 geometry coefficients, and
// the device operator of src/core/fluid/amr_pressure.cu:72-179, 825-834 (structured 7-point
// FV Laplacian + deterministic per-DOF incidence gather of the compact edges + WLS
// non-orthogonal correction + gauges).  The B200 design differs in how the work is laid out:
// one CTA per active 8^3 brick stages the FP64 pressure tile and its six face halos in shared
// memory (coalesced 16-byte loads), so every brick is read from HBM once per apply and the
// per-level launch loop and the output memset of the reference disappear.
#include "pcfd_internal.h"

#include <algorithm>
#include <array>
#include <cmath>
#include <cstring>
#include <limits>
#include <numeric>
#include <unordered_map>

namespace pcfd
{
    // ==================================================================================
    // structured operator
    // ==================================================================================
    namespace
    {
        // Shared-memory staged 7-point apply for bs = 8.  Tile index (k+1)*100+(j+1)*10+(i+1).
        template <class T>
        __global__ void __launch_bounds__(256) structured_apply8_kernel(
            const int* __restrict__ brick_list, const int* __restrict__ brick_level,
            const int* __restrict__ nbr, const uint32_t* __restrict__ flags,
            const double* __restrict__ level_h, const uint8_t* __restrict__ active,
            const uint8_t* __restrict__ cut, const T* __restrict__ p, T* __restrict__ out, int outlet)
        {
            constexpr int BS = 8, N = 10, C3 = 512;
            __shared__ T tile[N * N * N];
            __shared__ uint8_t act[N * N * N];
            __shared__ uint8_t cm[N * N * N];
            const int slot = brick_list[blockIdx.x];
            const int tid = threadIdx.x;
            const int64_t base = int64_t(slot) * C3;
            // interior: 512 values, 2 per thread
            for (int c = tid; c < C3; c += 256)
            {
                const int i = c & 7, j = (c >> 3) & 7, k = c >> 6;
                const int s = (k + 1) * 100 + (j + 1) * 10 + (i + 1);
                tile[s] = p[base + c];
                act[s] = active[base + c];
                cm[s] = cut[base + c];
            }
            // halos: 6 faces x 64 cells
            for (int e = tid; e < 6 * 64; e += 256)
            {
                const int face = e >> 6, a = e & 7, b = (e >> 3) & 7;
                const int axis = face >> 1, positive = face & 1;
                int i, j, k, hi, hj, hk;   // neighbour-local cell and halo tile position
                const int inner = positive ? 0 : BS - 1, halo = positive ? BS + 1 : 0;
                if (axis == 0) { i = inner; j = a; k = b; hi = halo; hj = a + 1; hk = b + 1; }
                else if (axis == 1) { i = a; j = inner; k = b; hi = a + 1; hj = halo; hk = b + 1; }
                else { i = a; j = b; k = inner; hi = a + 1; hj = b + 1; hk = halo; }
                const int s = hk * 100 + hj * 10 + hi;
                const int n = nbr[slot * 6 + face];
                if (n >= 0)
                {
                    const int64_t q = int64_t(n) * C3 + (k * BS + j) * BS + i;
                    tile[s] = p[q];
                    act[s] = active[q];
                    cm[s] = cut[q];
                }
                else
                {
                    tile[s] = T(0);
                    act[s] = 0;
                    cm[s] = 0;
                }
            }
            __syncthreads();
            const T h = T(level_h[brick_level[slot]]);
            const bool xmax = outlet && (flags[slot] & PCFD_BRICK_XMAX);
            for (int c = tid; c < C3; c += 256)
            {
                const int i = c & 7, j = (c >> 3) & 7, k = c >> 6;
                const int s = (k + 1) * 100 + (j + 1) * 10 + (i + 1);
                T value = T(0);
                if (act[s])
                {
                    const T pa = tile[s];
                    const uint8_t mine = cm[s];
                    // -x, +x, -y, +y, -z, +z ; the lower cell of the face owns its cut bit
                    if (act[s - 1] && !(cm[s - 1] & 1)) value += h * (pa - tile[s - 1]);
                    if (act[s + 1] && !(mine & 1)) value += h * (pa - tile[s + 1]);
                    if (act[s - 10] && !(cm[s - 10] & 2)) value += h * (pa - tile[s - 10]);
                    if (act[s + 10] && !(mine & 2)) value += h * (pa - tile[s + 10]);
                    if (act[s - 100] && !(cm[s - 100] & 4)) value += h * (pa - tile[s - 100]);
                    if (act[s + 100] && !(mine & 4)) value += h * (pa - tile[s + 100]);
                    if (xmax && i == BS - 1) value += T(2) * h * pa;
                }
                out[base + c] = value;
            }
        }

        // Generic brick size (one thread per cell, global loads).
        template <class T>
        __global__ void structured_apply_generic_kernel(
            const int* __restrict__ brick_list, int brick_count, int bs, const int* __restrict__ brick_level,
            const int* __restrict__ nbr, const uint32_t* __restrict__ flags, const double* __restrict__ level_h,
            const uint8_t* __restrict__ active, const uint8_t* __restrict__ cut, const T* __restrict__ p,
            T* __restrict__ out, int outlet)
        {
            const int c3 = bs * bs * bs;
            const int64_t work = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
            if (work >= int64_t(brick_count) * c3) return;
            const int slot = brick_list[int(work) / c3], local = int(work) % c3;
            const int i = local % bs, j = (local / bs) % bs, k = local / (bs * bs);
            const int64_t a = int64_t(slot) * c3 + local;
            if (!active[a]) { out[a] = T(0); return; }
            const T h = T(level_h[brick_level[slot]]);
            T value = T(0);
            const int coord[3] = {i, j, k};
            for (int axis = 0; axis < 3; ++axis)
                for (int sign = -1; sign <= 1; sign += 2)
                {
                    int q[3] = {i, j, k};
                    q[axis] += sign;
                    int64_t b = -1;
                    if (q[axis] >= 0 && q[axis] < bs) b = int64_t(slot) * c3 + (q[2] * bs + q[1]) * bs + q[0];
                    else
                    {
                        const int n = nbr[slot * 6 + 2 * axis + (sign > 0)];
                        if (n >= 0) { q[axis] = sign > 0 ? 0 : bs - 1; b = int64_t(n) * c3 + (q[2] * bs + q[1]) * bs + q[0]; }
                    }
                    const int64_t lower = sign > 0 ? a : b;
                    if (b >= 0 && active[b] && !(cut[lower] & (1u << axis))) value += h * (p[a] - p[b]);
                }
            if (outlet && (flags[slot] & PCFD_BRICK_XMAX) && coord[0] == bs - 1) value += T(2) * h * p[a];
            out[a] = value;
        }

        __global__ void zero_range_kernel(double* x, int64_t begin, int64_t end)
        {
            const int64_t q = begin + int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
            if (q < end) x[q] = 0.0;
        }

        // WLS pressure gradient of every node, a thread per node (FP64 sums in stencil order).  Reads p only,
        // so it may run beside the structured operator that precedes it on the stream
        // (apply_operator); its last CTA waits for that launch, so that what follows this one finds both
        // complete.  Bound by the scattered reads of p (32-byte sectors for 8-byte values) beside 28 B
        // per entry: four entries in flight per thread.  Staging a CTA's entries in shared memory, one per
        // thread, measured slower (88 against 72 us for 1.2 M nodes).
        constexpr int kRowThreads = 128;
        __global__ void __launch_bounds__(kRowThreads) reconstruct_gradient_kernel(const int* __restrict__ dof, const int* __restrict__ offset,
            const int* __restrict__ neighbour, const double* __restrict__ weight, const double* __restrict__ p,
            double* __restrict__ gradient, int nodes)
        {
            chain_release();
            const int node = blockIdx.x * kRowThreads + threadIdx.x;
            if (node < nodes)
            {
                const int q0 = offset[node], q1 = offset[node + 1];
                const double centre = p[dof[node]];
                double gx = 0, gy = 0, gz = 0;
#pragma unroll 4
                for (int q = q0; q < q1; ++q)
                {
                    const double d = p[neighbour[q]] - centre;
                    gx += weight[3 * q] * d;
                    gy += weight[3 * q + 1] * d;
                    gz += weight[3 * q + 2] * d;
                }
                gradient[3 * node] = gx;
                gradient[3 * node + 1] = gy;
                gradient[3 * node + 2] = gz;
            }
            if (blockIdx.x == gridDim.x - 1) chain_wait();
        }

        __device__ inline double face_derivative(const double* gradient, int lower_node, int upper_node,
                                                 const double* correction, double upper_weight)
        {
            const double lw = 1.0 - upper_weight;
            double derivative = 0.0;
            for (int c = 0; c < 3; ++c)
                derivative += correction[c] * (lw * gradient[3 * lower_node + c] + upper_weight * gradient[3 * upper_node + c]);
            return derivative;
        }

        // Fluxes of the compact edges at each incident DOF (reference amr_pressure.cu:105-178), a thread per
        // DOF: with kPart & 1 the two-point sum in the reference's per-DOF order, sign * coefficient *
        // (p[lower] - p[upper]) evaluated as coefficient * (p[dof] - p[other]) (equal bit for bit: negating
        // a difference or a product is exact), with kPart & 2 the WLS affine-exact non-orthogonal
        // corrections, out += each sum.  Entries have active endpoints only (build_operator drops the
        // others) and hold everything but the values, so a row is three loads deep; as two launches
        // over edge-indexed arrays the sums took 30 us against 21 for the 297 k DOFs of a 5.1 M-cell grid.
        template <int kPart>
        __global__ void __launch_bounds__(kRowThreads) irregular_gather_kernel(const int* __restrict__ incident_dof,
            const int* __restrict__ incident_offset, const int* __restrict__ incident_other, const double* __restrict__ incident_coefficient,
            const int2* __restrict__ incident_nodes, const double* __restrict__ incident_correction, int incident_dofs,
            const double* __restrict__ p, const double* __restrict__ gradient, double* __restrict__ out)
        {
            chain_wait();
            chain_release();
            const int node = blockIdx.x * kRowThreads + threadIdx.x;
            if (node >= incident_dofs) return;
            const int dof = incident_dof[node], q0 = incident_offset[node], q1 = incident_offset[node + 1];
            const double centre = p[dof], before = out[dof];
            double two_point = 0.0, correction = 0.0;
#pragma unroll 2
            for (int q = q0; q < q1; ++q)
            {
                if (kPart & 1) two_point += incident_coefficient[q] * (centre - p[incident_other[q]]);
                if (kPart & 2)
                {
                    const int2 n = incident_nodes[q];
                    const double* c = incident_correction + 5 * int64_t(q);
                    const double corr[3] = {c[0], c[1], c[2]}, upper_weight = c[3], signed_area = c[4];
                    correction += n.x >= 0 ? -signed_area * face_derivative(gradient, n.x, n.y, corr, upper_weight) : 0.0;
                }
            }
            out[dof] = kPart == 3 ? (before + two_point) + correction : before + (kPart == 1 ? two_point : correction);
        }

        __global__ void gauge_apply_kernel(const int* dof, const double* coefficient, int count, const double* p, double* out)
        {
            const int q = blockIdx.x * blockDim.x + threadIdx.x;
            if (q < count) out[dof[q]] += coefficient[q] * p[dof[q]];
        }
    }

    namespace
    {
        // The operator with the WLS-gradient scratch at `gradient`.  Its parts: the structured 7-point part
        // (reads p, writes out), the gradient (reads p) and the compact edges (add to out).  The brick
        // kernel's persistent CTAs release their successor at once and the gradient does not read what
        // they write, so the two run side by side; the edges follow when both are complete.  Grids
        // without compact edges need no gradient.  One application, before -> now: 65 k cells on one level
        // 8.2 -> 4.1 us, 1.1 M on three levels 38 -> 28, 5.1 M 88 -> 68, 16 M on four 220 -> 189.
        void apply_operator(System& s, const double* p, double* out, bool orthogonal_only, double* gradient)
        {
            IrregularOperator& o = s.irr;
            if (s.S > s.structured)
                zero_range_kernel<<<blocks_for(s.S - s.structured), kThreads, 0, launch_stream(s)>>>(out, s.structured, s.S);
            bool beside = false;       // the gradient may start while the structured part runs
            if (s.active_bricks)
            {
                ProfileScope scope(s, PCFD_PROFILE_STRUCTURED_APPLY);
                if (s.fine.enabled && aligned16(p) && aligned16(out))
                {
                    brick_apply(s, p, out);
                    beside = !scope.on;
                }
                else if (s.bs == 8)
                    structured_apply8_kernel<double><<<s.active_bricks, 256, 0, launch_stream(s)>>>(
                        s.active_brick_list, s.brick_level, s.brick_nbr, s.brick_flags, s.d_level_h, s.active,
                        s.cut_face_mask, p, out, s.outlet ? 1 : 0);
                else
                    structured_apply_generic_kernel<double><<<blocks_for(int64_t(s.active_bricks) * s.bs3), kThreads, 0, launch_stream(s)>>>(
                        s.active_brick_list, s.active_bricks, s.bs, s.brick_level, s.brick_nbr, s.brick_flags, s.d_level_h,
                        s.active, s.cut_face_mask, p, out, s.outlet ? 1 : 0);
            }
            const bool corrected = !orthogonal_only && o.gradient_nodes && o.incident_dofs;
            if (corrected && beside)
                launch_chained(s, reconstruct_gradient_kernel, unsigned(blocks_for(o.gradient_nodes, kRowThreads)), kRowThreads, o.grad_dof,
                               o.grad_offset, o.grad_neighbour, o.grad_weight, p, gradient, o.gradient_nodes);
            else if (corrected)
                reconstruct_gradient_kernel<<<blocks_for(o.gradient_nodes, kRowThreads), kRowThreads, 0, launch_stream(s)>>>(
                    o.grad_dof, o.grad_offset, o.grad_neighbour, o.grad_weight, p, gradient, o.gradient_nodes);
            auto edges = [&](auto* kernel) {
                if (o.incident_dofs)
                    launch_chained(s, kernel, unsigned(blocks_for(o.incident_dofs, kRowThreads)), kRowThreads, o.incident_dof,
                                   o.incident_offset, o.incident_other, o.incident_coefficient, o.incident_nodes, o.incident_correction,
                                   o.incident_dofs, p, gradient, out);
            };
            // gauges (closed components of the flow region) are added between the two sums of a row
            const bool together = corrected && !o.gauges;
            edges(together ? irregular_gather_kernel<3> : irregular_gather_kernel<1>);
            if (o.gauges)
                gauge_apply_kernel<<<blocks_for(o.gauges), kThreads, 0, launch_stream(s)>>>(o.gauge_dof, o.gauge_coefficient, o.gauges, p, out);
            if (corrected && !together) edges(irregular_gather_kernel<2>);
            cuda_check(cudaGetLastError(), "launch pressure operator");
        }
    }

    void launch_apply(System& s, const double* p, double* out, bool orthogonal_only)
    {
        apply_operator(s, p, out, orthogonal_only, s.irr.gradient);
    }

    // ==================================================================================
    // deterministic FP64 reductions
    // ==================================================================================
    namespace
    {
        constexpr int kDotBlocks = 592;   // 4 x 148 SMs, fixed so the summation order never changes

        __device__ inline double warp_sum(double v)
        {
            for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
            return v;
        }
        __device__ inline double block_sum(double v, double* shared)
        {
            v = warp_sum(v);
            const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
            if (lane == 0) shared[warp] = v;
            __syncthreads();
            v = threadIdx.x < (blockDim.x >> 5) ? shared[threadIdx.x] : 0.0;
            if (warp == 0) v = warp_sum(v);
            return v;
        }
        __global__ void __launch_bounds__(256) dot_partial_kernel(const double* __restrict__ a, const double* __restrict__ b,
            const uint8_t* __restrict__ active, int64_t n, double* __restrict__ partial)
        {
            __shared__ double shared[8];
            double v = 0.0;
            for (int64_t q = int64_t(blockIdx.x) * blockDim.x + threadIdx.x; q < n; q += int64_t(gridDim.x) * blockDim.x)
                if (active[q]) v += a[q] * b[q];
            v = block_sum(v, shared);
            if (threadIdx.x == 0) partial[blockIdx.x] = v;
        }
        // r = b - Ax on the active entries (0 elsewhere) and its dot partials in one pass, in the order of
        // dot_partial_kernel
        __global__ void __launch_bounds__(256) residual_dot_kernel(const double* __restrict__ b, const double* __restrict__ Ax,
            const uint8_t* __restrict__ active, int64_t n, double* __restrict__ r, double* __restrict__ partial)
        {
            __shared__ double shared[8];
            double v = 0.0;
            for (int64_t q = int64_t(blockIdx.x) * blockDim.x + threadIdx.x; q < n; q += int64_t(gridDim.x) * blockDim.x)
            {
                const double value = active[q] ? b[q] - Ax[q] : 0.0;
                r[q] = value;
                if (active[q]) v += value * value;
            }
            v = block_sum(v, shared);
            if (threadIdx.x == 0) partial[blockIdx.x] = v;
        }
        __global__ void __launch_bounds__(256) dot_final_kernel(const double* __restrict__ partial, int count, double* __restrict__ result)
        {
            __shared__ double shared[8];
            double v = 0.0;
            for (int q = threadIdx.x; q < count; q += blockDim.x) v += partial[q];
            v = block_sum(v, shared);
            if (threadIdx.x == 0) *result = v;
        }
    }

    namespace
    {
        double dot_total(System& s)
        {
            dot_final_kernel<<<1, 256, 0, launch_stream(s)>>>(s.dot_partial, kDotBlocks, s.dot_result);
            cuda_check(cudaMemcpyAsync(s.pinned, s.dot_result, sizeof(double), cudaMemcpyDeviceToHost, s.stream), "dot readback");
            cuda_check(cudaStreamSynchronize(s.stream), "dot synchronize");
            return s.pinned[0];
        }
    }

    double device_dot(System& s, const double* a, const double* b)
    {
        dot_partial_kernel<<<kDotBlocks, 256, 0, launch_stream(s)>>>(a, b, s.active, s.S, s.dot_partial);
        return dot_total(s);
    }

    // One pass in place of a copy, a subtraction and a dot: 25 B per entry against 66.
    double vec_residual_dot(System& s, const double* b, const double* Ax, double* r)
    {
        residual_dot_kernel<<<kDotBlocks, 256, 0, launch_stream(s)>>>(b, Ax, s.active, s.S, r, s.dot_partial);
        return dot_total(s);
    }

    // ==================================================================================
    // vector kernels (active-masked, reference amr_pressure.cu:180-199)
    // ==================================================================================
    namespace
    {
        __global__ void copy_active_kernel(const double* src, double* dst, const uint8_t* active, int64_t n)
        {
            const int64_t q = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
            if (q < n) dst[q] = active[q] ? src[q] : 0.0;
        }
        __global__ void axpy_active_kernel(double* y, const double* x, double a, const uint8_t* active, int64_t n)
        {
            const int64_t q = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
            if (q < n && active[q]) y[q] += a * x[q];
        }
        __global__ void scaled_copy_active_kernel(double* dst, const double* src, double a, const uint8_t* active, int64_t n)
        {
            const int64_t q = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
            if (q < n) dst[q] = active[q] ? a * src[q] : 0.0;
        }
        __global__ void update_solution_residual_kernel(double* x, double* r, const double* d, const double* Ad, double alpha,
                                                        const uint8_t* active, int64_t n)
        {
            const int64_t q = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
            if (q < n && active[q]) { x[q] += alpha * d[q]; r[q] -= alpha * Ad[q]; }
        }
        __global__ void update_direction_kernel(const double* z, double* d, double beta, const uint8_t* active, int64_t n)
        {
            const int64_t q = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
            if (q < n) d[q] = active[q] ? z[q] + beta * d[q] : 0.0;
        }
    }
    void vec_copy_active(System& s, const double* src, double* dst)
    {
        copy_active_kernel<<<blocks_for(s.S), kThreads, 0, launch_stream(s)>>>(src, dst, s.active, s.S);
    }
    void vec_axpy_active(System& s, double* y, const double* x, double a)
    {
        axpy_active_kernel<<<blocks_for(s.S), kThreads, 0, launch_stream(s)>>>(y, x, a, s.active, s.S);
    }
    void vec_scaled_copy_active(System& s, double* dst, const double* src, double a)
    {
        scaled_copy_active_kernel<<<blocks_for(s.S), kThreads, 0, launch_stream(s)>>>(dst, src, a, s.active, s.S);
    }
    void vec_update_solution_residual(System& s, double* x, double* r, const double* d, const double* Ad, double alpha)
    {
        update_solution_residual_kernel<<<blocks_for(s.S), kThreads, 0, launch_stream(s)>>>(x, r, d, Ad, alpha, s.active, s.S);
    }
    void vec_update_direction(System& s, const double* z, double* d, double beta)
    {
        update_direction_kernel<<<blocks_for(s.S), kThreads, 0, launch_stream(s)>>>(z, d, beta, s.active, s.S);
    }
    void vec_zero(System& s, double* x)
    {
        cuda_check(cudaMemsetAsync(x, 0, size_t(s.S) * sizeof(double), s.stream), "zero vector");
    }

    // ==================================================================================
    // operator setup (host)
    // ==================================================================================
    namespace
    {
        double gradient_factor(const pcfd_connections& c, int e)
        {
            // pressure_gradient_factor (amr_pressure.h:122-126)
            const double f = c.orthogonal_gradient_factor[e];
            return f > 0 ? f : (c.normal_distance[e] > 0 ? 1.0 / c.normal_distance[e] : 0.0);
        }
    }

    void build_operator(System& s, const pcfd_topology& t)
    {
        IrregularOperator& o = s.irr;
        const int cf = t.coarse_fine.count, eb = t.embedded.count, nc = cf + eb;
        std::vector<int> lower(nc), upper(nc), lnode(nc), unode(nc);
        std::vector<double> coefficient(nc), correction(size_t(nc) * 3), weight(nc), area(nc);
        for (int e = 0; e < nc; ++e)
        {
            const pcfd_connections& c = e < cf ? t.coarse_fine : t.embedded;
            const int q = e < cf ? e : e - cf;
            const bool forward = c.direction[q] > 0;
            lower[e] = forward ? c.coarse_dof[q] : c.fine_dof[q];
            upper[e] = forward ? c.fine_dof[q] : c.coarse_dof[q];
            coefficient[e] = c.open_area[q] * gradient_factor(c, q);
            lnode[e] = c.lower_gradient_node[q];
            unode[e] = c.upper_gradient_node[q];
            for (int a = 0; a < 3; ++a) correction[3 * e + a] = c.nonorthogonal_correction[3 * q + a];
            weight[e] = c.upper_gradient_weight[q];
            area[e] = c.open_area[q];
        }

        const pcfd_regular_corrections& rc = t.regular;
        o.regular_count = rc.count;
        std::vector<int> rl(rc.count), ru(rc.count), rln(rc.count), run(rc.count);
        std::vector<double> rcoef(rc.count), rcorr(size_t(rc.count) * 3), rw(rc.count), ra(rc.count), rd(rc.count);
        for (int e = 0; e < rc.count; ++e)
        {
            rl[e] = rc.lower_dof[e]; ru[e] = rc.upper_dof[e];
            rln[e] = rc.lower_gradient_node[e]; run[e] = rc.upper_gradient_node[e];
            rcoef[e] = rc.open_area[e] * rc.two_point_delta[e];
            for (int a = 0; a < 3; ++a) rcorr[3 * e + a] = rc.nonorthogonal_correction[3 * e + a];
            rw[e] = rc.upper_gradient_weight[e]; ra[e] = rc.open_area[e]; rd[e] = rc.two_point_delta[e];
        }
        o.reg_lower.upload(rl); o.reg_upper.upload(ru); o.reg_lower_node.upload(rln); o.reg_upper_node.upload(run);
        o.reg_correction.upload(rcorr); o.reg_upper_weight.upload(rw); o.reg_delta.upload(rd);

        // Deterministic incidence: (dof, edge, sign) sorted, reference amr_pressure.cu:774-813.
        struct Incident { int dof, edge; int8_t sign; };
        std::vector<Incident> inc;
        inc.reserve(size_t(2) * (nc + rc.count));
        auto add = [&](int a, int b, int encoded) {
            if (a < 0 || b < 0 || a >= s.S || b >= s.S || a == b || !t.active[a] || !t.active[b]) return;
            inc.push_back({a, encoded, 1});
            inc.push_back({b, encoded, -1});
        };
        for (int e = 0; e < nc; ++e) add(lower[e], upper[e], e);
        for (int e = 0; e < rc.count; ++e) add(rl[e], ru[e], nc + e);
        std::sort(inc.begin(), inc.end(), [](const Incident& a, const Incident& b) {
            if (a.dof != b.dof) return a.dof < b.dof;
            if (a.edge != b.edge) return a.edge < b.edge;
            return a.sign < b.sign;
        });
        std::vector<int> idof, ioff, iother;
        std::vector<int2> inodes;
        std::vector<double> icoef, icorr;
        iother.reserve(inc.size()); inodes.reserve(inc.size()); icoef.reserve(inc.size()); icorr.reserve(5 * inc.size());
        for (size_t q = 0; q < inc.size(); ++q)
        {
            if (q == 0 || inc[q].dof != inc[q - 1].dof) { idof.push_back(inc[q].dof); ioff.push_back(int(q)); }
            const int e = inc[q].edge, r = e - nc;
            const bool connection = e < nc;
            const int lo = connection ? lower[e] : rl[r], hi = connection ? upper[e] : ru[r];
            iother.push_back(inc[q].sign > 0 ? hi : lo);
            icoef.push_back(connection ? coefficient[e] : rcoef[r]);
            const int ln = connection ? lnode[e] : rln[r], un = connection ? unode[e] : run[r];
            inodes.push_back(ln >= 0 && un >= 0 ? make_int2(ln, un) : make_int2(-1, -1));
            const double* c = connection ? &correction[3 * size_t(e)] : &rcorr[3 * size_t(r)];
            icorr.insert(icorr.end(), {c[0], c[1], c[2], connection ? weight[e] : rw[r], inc[q].sign * (connection ? area[e] : ra[r])});
        }
        ioff.push_back(int(inc.size()));
        o.incident_dofs = int(idof.size());
        o.incident_dof.upload(idof); o.incident_offset.upload(ioff);
        o.incident_other.upload(iother); o.incident_coefficient.upload(icoef);
        o.incident_nodes.upload(inodes); o.incident_correction.upload(icorr);

        o.gradient_nodes = t.gradient_node_count;
        if (o.gradient_nodes)
        {
            const int nnz = t.gradient_offset[o.gradient_nodes];
            o.grad_dof.upload(std::vector<int>(t.gradient_dof, t.gradient_dof + o.gradient_nodes));
            o.grad_offset.upload(std::vector<int>(t.gradient_offset, t.gradient_offset + o.gradient_nodes + 1));
            o.grad_neighbour.upload(std::vector<int>(t.gradient_neighbour, t.gradient_neighbour + nnz));
            o.grad_weight.upload(std::vector<double>(t.gradient_weight, t.gradient_weight + size_t(nnz) * 3));
            o.gradient.alloc(size_t(o.gradient_nodes) * 3);
        }
        o.gauges = t.gauge_count;
        if (o.gauges)
        {
            o.gauge_dof.upload(std::vector<int>(t.gauge_dof, t.gauge_dof + o.gauges));
            o.gauge_coefficient.upload(std::vector<double>(t.gauge_coefficient, t.gauge_coefficient + o.gauges));
        }
    }

    // ==================================================================================
    // allocation-free operator apply
    // ==================================================================================
    // The full operator needs FP64 scratch for the WLS pressure gradient at every gradient node
    // (3 doubles per node).  pcfd_pressure_apply_device takes it from the system; this variant
    // takes it from a fixed static device array instead, so a call performs no device or pinned
    // allocation of any kind and never touches the system's own scratch.  It serves callers that
    // cannot allocate at call time -- hosts whose device memory is fully reserved by another
    // pool, latency-bound loops that must not enter the allocator -- and a second user of one
    // system that must not disturb the scratch an in-flight solve on that system is using.
    //
    // Limits and contract:
    //   * at most kNoAllocGradientNodes WLS gradient nodes (262,144 nodes, 6 MiB of scratch);
    //     larger systems are rejected with PCFD_INVALID_ARG before anything is launched;
    //   * the first call through a system that needs the WLS term (not orthogonal-only, gradient
    //     nodes present) looks up the scratch address with cudaGetSymbolAddress, the system's
    //     device current, and keeps it in the system; make that first call before any stream
    //     capture.  Orthogonal-only calls and systems without gradient nodes never look it up.
    //     The address lives as long as the device context, which outlives every system on it (a
    //     cudaDeviceReset invalidates the systems too; they are created again, and look it up
    //     again);
    //   * the scratch is shared by every system on the device: calls that overlap in time (other
    //     threads or other streams) race on it -- serialise them;
    //   * no scratch entry needs to start at zero: the gradient kernel writes all 3 components
    //     of every node before the gather reads them; the output is written exactly where
    //     pcfd_pressure_apply_device writes it (every cell of the non-covered bricks and every
    //     EB fragment).
    namespace
    {
        constexpr int kNoAllocGradientNodes = 1 << 18;
        static __device__ __align__(256) double g_noalloc_gradient[3 * kNoAllocGradientNodes];

        // The static scratch's device address, looked up once per system with its device current.
        double* noalloc_scratch(System& s)
        {
            if (!s.noalloc_gradient)
            {
                int current = 0;
                cuda_check(cudaGetDevice(&current), "cudaGetDevice");
                if (current != s.device) cuda_check(cudaSetDevice(s.device), "cudaSetDevice");
                void* ptr = nullptr;
                const cudaError_t e = cudaGetSymbolAddress(&ptr, g_noalloc_gradient);
                if (current != s.device) cudaSetDevice(current);
                cuda_check(e, "cudaGetSymbolAddress(noalloc gradient scratch)");
                s.noalloc_gradient = static_cast<double*>(ptr);
            }
            return s.noalloc_gradient;
        }
    }

    void launch_apply_noalloc(System& s, const double* p, double* out, bool orthogonal_only)
    {
        IrregularOperator& o = s.irr;
        if (!orthogonal_only && o.gradient_nodes > kNoAllocGradientNodes)
            throw Error(PCFD_INVALID_ARG, "pcfd_pressure_apply_device_noalloc: " + std::to_string(o.gradient_nodes) +
                                              " WLS gradient nodes exceed the static scratch maximum of " +
                                              std::to_string(kNoAllocGradientNodes));
        apply_operator(s, p, out, orthogonal_only, !orthogonal_only && o.gradient_nodes ? noalloc_scratch(s) : nullptr);
    }
}
