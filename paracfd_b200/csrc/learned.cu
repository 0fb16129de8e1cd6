// learned.cu -- brick-local learned preconditioner (no reference counterpart).
//
// A 3-level U-Net per 8^3 brick (levels 8^3/4^3/2^3 with 16/32/64 channels, 3x3x3 convolutions
// with zero padding at the brick boundary, 2x2x2 average pooling, nearest upsampling, skip
// connections by concatenation, ReLU, no biases, a 1x1x1 head).  The input of a brick is
// D^-1 r / s and the active mask, s the RMS of D^-1 r over the brick's active cells; the output is
// z = s * net(...) on the active cells, so the map is positively homogeneous in r.  The
// definition, and the numbers every kernel here is checked against, are the numpy oracle in
// oracle/unet.py.
//
// Convolutions run on the 5th-generation tensor cores: tcgen05.mma kind::f16 (BF16 operands,
// FP32 accumulators in TMEM), M = 128 output positions x N = 3 Cout (the three x taps) x K = 16 input
// channels per instruction.  A CTA stages a group of bricks into shared memory in a K-major layout with
// zero rows around every (z, y) plane ([channel chunk of 8][position][8 x BF16]), so that the A operand
// of every (dz, dy) pair is the same layout shifted by whole rows: each pair is one shared-memory
// descriptor, no im2col copy.  A tile is 128 consecutive positions; rows that fall on padding are
// computed and discarded.  The epilogue adds the three x blocks across neighbouring lanes.
//
// Training (pcfd_learned_train): (residual, multigrid correction) brick pairs harvested from the
// solver's own preconditioner calls, masked mean-square loss on z/s, backward pass with the
// transposed convolutions on the same tensor-core kernel (flipped taps, transposed channels),
// weight gradients on mma.sync tiles (BF16 operands, FP32 sums), Adam on FP32 master weights.
#include "pcfd_internal.h"

#include <cuda_bf16.h>

#include <algorithm>
#include <cmath>
#include <cstring>
#include <random>

namespace pcfd
{
    namespace
    {
        using bf16 = __nv_bfloat16;

        // ---- network shape (must match oracle/unet.py) ----
        // parameter tensors in flat order: enc0.0 enc1.0 bott.0 dec1.0 dec1.1 dec0.0 dec0.1 ([27][cout][cin]
        // each), then the head [16]
        constexpr int kHead = 16;
        enum Tensor { ENC0, ENC1, BOTT, DEC1A, DEC1B, DEC0A, DEC0B };
        __host__ __device__ constexpr int tensor_cout(int k) { return k == 0 ? 16 : k == 1 ? 32 : k == 2 ? 64 : k <= 4 ? 32 : 16; }
        __host__ __device__ constexpr int tensor_cin(int k) { return k <= 1 ? 16 : k == 2 ? 32 : k == 3 ? 64 : k == 4 ? 32 : k == 5 ? 32 : 16; }
        __host__ __device__ constexpr int64_t tensor_size(int k) { return int64_t(27) * tensor_cout(k) * tensor_cin(k); }
        __host__ __device__ constexpr int64_t tensor_offset(int k) { return k == 0 ? 0 : tensor_offset(k - 1) + tensor_size(k - 1); }
        constexpr int64_t kWeights = tensor_offset(7);
        constexpr int64_t kParams = kWeights + kHead;
        static_assert(kParams == 179728, "parameter count must match oracle/unet.py");

        // A tensor-core wait gives up after the system's wait limit (pcfd_learned_set_wait, 2 s by
        // default); after a wait gave up, the kernel drains its last commit with this fixed limit
        // before freeing its tensor memory.
        constexpr uint64_t kMaxWaitNs = 2000000000ull;

        // ---- geometry of one level's staged group of bricks ----
        // NB bricks per CTA; rows (z, y) padded by one on each side, x as it is: position
        // ((b * ROWS + (z + 1) (N + 2) + y + 1) N + x.  A tile is 128 consecutive positions (N = 8: 16 padded
        // rows of 8, five tiles cover a brick's rows 11..90; N = 4: 32 rows of 4, one tile from row 7 covers
        // a brick; N = 2: 64 rows of 2, a tile covers four bricks from row 5).
        template <int N, int NB> struct Geometry
        {
            static constexpr int XP = N + 2, ROWS = XP * XP, P = ROWS * N, FIRST = XP + 1;
            static constexpr int T = N == 8 ? 5 * NB : N == 4 ? NB : NB / 4;
            __host__ __device__ static constexpr int tile_start(int t)
            {
                return N == 8 ? (t / 5) * P + (FIRST + 16 * (t % 5)) * N : N == 4 ? t * P + FIRST * N : FIRST * N + 128 * t;
            }
            // staged positions: the last tile plus the largest shift, in whole 8-position groups
            static constexpr int NPOS = (tile_start(T - 1) + 128 + FIRST * N + 7) / 8 * 8;
        };
        template <int N> __host__ __device__ constexpr int padded(int b, int x, int y, int z)
        {
            return (b * (N + 2) * (N + 2) + (z + 1) * (N + 2) + y + 1) * N + x;
        }
        // shift in positions of the (dz, dy) pair zy = 3 (dz + 1) + dy + 1
        template <int N> __host__ __device__ constexpr int row_shift(int zy) { return ((zy / 3 - 1) * (N + 2) + zy % 3 - 1) * N; }
        // compile-time proof that every descriptor stays inside the staged rows and that the
        // tiles cover every interior voxel of every brick of a group
        template <int N, int NB> constexpr bool geometry_in_bounds()
        {
            using Gm = Geometry<N, NB>;
            bool seen[NB * Gm::P] = {};
            for (int t = 0; t < Gm::T; ++t)
            {
                const int p0 = Gm::tile_start(t);
                if (p0 + row_shift<N>(0) < 0 || p0 + 127 + row_shift<N>(8) >= Gm::NPOS) return false;
                for (int p = p0; p < p0 + 128; ++p)
                    if (p < NB * Gm::P) seen[p] = true;
            }
            for (int b = 0; b < NB; ++b)
                for (int z = 0; z < N; ++z)
                    for (int y = 0; y < N; ++y)
                        for (int x = 0; x < N; ++x)
                            if (!seen[padded<N>(b, x, y, z)]) return false;
            return Gm::NPOS % 8 == 0;
        }
        static_assert(geometry_in_bounds<2, 8>(), "2^3 tiling out of bounds");
        static_assert(geometry_in_bounds<4, 4>() && geometry_in_bounds<4, 2>(), "4^3 tiling out of bounds");
        static_assert(geometry_in_bounds<8, 1>(), "8^3 tiling out of bounds");

        // ---- tcgen05 / mbarrier primitives (inline PTX) ----
        __device__ inline uint32_t smem_u32(const void* p) { return uint32_t(__cvta_generic_to_shared(p)); }

        // K-major, no-swizzle shared-memory matrix descriptor: 8-row core matrices of 16-byte rows,
        // lbo = bytes between the two 8-element K halves, sbo = bytes between 8-row groups.
        __device__ inline uint64_t smem_descriptor(uint32_t address, uint32_t lbo, uint32_t sbo)
        {
            uint64_t d = uint64_t((address >> 4) & 0x3FFFu);
            d |= uint64_t((lbo >> 4) & 0x3FFFu) << 16;
            d |= uint64_t((sbo >> 4) & 0x3FFFu) << 32;
            d |= uint64_t(1) << 46;   // descriptor version (sm_100)
            return d;                 // base offset 0, swizzle none
        }
        // kind::f16 instruction descriptor: BF16 A and B (K-major), FP32 D, M = 128, N = n
        __host__ __device__ constexpr uint32_t instruction_descriptor(int n)
        {
            return (1u << 4) | (1u << 7) | (1u << 10) | (uint32_t(n >> 3) << 17) | (uint32_t(128 >> 4) << 24);
        }
        __device__ inline void mma_bf16(uint32_t tmem_d, uint64_t a, uint64_t b, uint32_t idesc, uint32_t accumulate)
        {
            const uint32_t mask = 0;
            asm volatile(
                "{\n\t.reg .pred p;\n\t"
                "setp.ne.b32 p, %4, 0;\n\t"
                "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, {%5, %5, %5, %5}, p;\n\t}\n"
                :
                : "r"(tmem_d), "l"(a), "l"(b), "r"(idesc), "r"(accumulate), "r"(mask));
        }
        __device__ inline void mma_commit(uint64_t* bar)
        {
            asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_u32(bar)) : "memory");
        }
        __device__ inline void fence_before_sync() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
        __device__ inline void fence_after_sync() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
        __device__ inline void fence_async_shared() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }
        __device__ inline void barrier_init(uint64_t* bar)
        {
            asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_u32(bar)) : "memory");
        }
        __device__ inline uint64_t global_ns()
        {
            uint64_t t;
            asm volatile("mov.u64 %0, %globaltimer;" : "=l"(t));
            return t;
        }
        // polls the barrier phase with the given parity; false after limit_ns nanoseconds
        __device__ inline bool barrier_wait(uint64_t* bar, uint32_t parity, uint64_t limit_ns)
        {
            const uint32_t a = smem_u32(bar);
            const uint64_t start = global_ns();
            for (;;)
            {
                uint32_t done;
                asm volatile(
                    "{\n\t.reg .pred p;\n\t"
                    "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
                    "selp.u32 %0, 1, 0, p;\n\t}\n"
                    : "=r"(done)
                    : "r"(a), "r"(parity)
                    : "memory");
                if (done) return true;
                if (global_ns() - start > limit_ns) return false;
            }
        }
        __device__ inline void tmem_alloc(uint32_t* slot, uint32_t cols)
        {
            asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(slot)), "r"(cols) : "memory");
            asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
        }
        __device__ inline void tmem_dealloc(uint32_t taddr, uint32_t cols)
        {
            asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(cols) : "memory");
        }
        // 16 consecutive FP32 accumulator columns of this thread's TMEM lane
        __device__ inline void tmem_load16(uint32_t taddr, float* v)
        {
            uint32_t r[16];
            asm volatile(
                "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];\n"
                : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
                  "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
                : "r"(taddr));
            asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
            for (int i = 0; i < 16; ++i) v[i] = __uint_as_float(r[i]);
        }

        __device__ inline uint4 pack8(const float* f)
        {
            uint4 u;
            uint32_t* w = reinterpret_cast<uint32_t*>(&u);
            for (int i = 0; i < 4; ++i)
            {
                const __nv_bfloat162 h = __floats2bfloat162_rn(f[2 * i], f[2 * i + 1]);
                w[i] = *reinterpret_cast<const uint32_t*>(&h);
            }
            return u;
        }
        __device__ inline void unpack8(const uint4& u, float* f)
        {
            const uint32_t* w = reinterpret_cast<const uint32_t*>(&u);
            for (int i = 0; i < 4; ++i)
            {
                const __nv_bfloat162 h = *reinterpret_cast<const __nv_bfloat162*>(&w[i]);
                const float2 v = __bfloat1622float2(h);
                f[2 * i] = v.x;
                f[2 * i + 1] = v.y;
            }
        }

        // ---- convolution ----
        constexpr int kConvThreads = 256;
        enum SourceMode { SAME = 0, POOL = 1, UP = 2 };
        struct ConvSource
        {
            const bf16* x;     // [samples][level voxels][channels]
            const bf16* w;     // [27][cout][channels]
            int channels, mode;
        };
        struct ConvParams
        {
            ConvSource src[2];
            int sources, cout, samples, relu, out_fp32;
            int weight_slots;  // staged 16-channel weight blocks: all of the layer's, or two buffers
            void* y;           // [samples][N^3][cout], BF16 or FP32
            int* error;        // set to 1 when a barrier wait gave up
            uint64_t wait_ns;  // limit of each tensor-core wait
            int idle_wait;     // 1: the first wait polls a barrier that no commit completes (fault-path check)
        };

        __host__ __device__ constexpr int tmem_columns(int cols)
        {
            return cols <= 32 ? 32 : cols <= 64 ? 64 : cols <= 128 ? 128 : cols <= 256 ? 256 : 512;
        }

        // 8 channels [c0, c0 + 8) of voxel (x,y,z) of sample b from a source at level N (after
        // its pooling / upsampling), as 8 BF16
        template <int N> __device__ inline uint4 load_source(const ConvSource& s, int64_t b, int x, int y, int z, int c0)
        {
            const int C = s.channels;
            if (s.mode == SAME)
                return *reinterpret_cast<const uint4*>(s.x + ((b * N + z) * N + y) * int64_t(N) * C + int64_t(x) * C + c0);
            if (s.mode == UP)
            {
                constexpr int M = N / 2;
                return *reinterpret_cast<const uint4*>(s.x + ((b * M + z / 2) * M + y / 2) * int64_t(M) * C + int64_t(x / 2) * C + c0);
            }
            constexpr int F = 2 * N;
            float acc[8] = {0, 0, 0, 0, 0, 0, 0, 0}, v[8];
            for (int k = 0; k < 8; ++k)
            {
                const int fx = 2 * x + (k & 1), fy = 2 * y + ((k >> 1) & 1), fz = 2 * z + (k >> 2);
                unpack8(*reinterpret_cast<const uint4*>(s.x + ((b * F + fz) * F + fy) * int64_t(F) * C + int64_t(fx) * C + c0), v);
                for (int i = 0; i < 8; ++i) acc[i] += v[i];
            }
            for (int i = 0; i < 8; ++i) acc[i] *= 0.125f;
            return pack8(acc);
        }

        // address of the 8 channels [c0, c0 + 8) of voxel (x,y,z) of sample b for a SAME or UP source
        template <int N> __device__ inline const bf16* source_address(const ConvSource& s, int64_t b, int x, int y, int z, int c0)
        {
            const int C = s.channels;
            if (s.mode == SAME) return s.x + ((b * N + z) * N + y) * int64_t(N) * C + int64_t(x) * C + c0;
            constexpr int M = N / 2;
            return s.x + ((b * M + z / 2) * M + y / 2) * int64_t(M) * C + int64_t(x / 2) * C + c0;
        }
        __device__ inline void cp_async16(void* dst, const void* src)
        {
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_u32(dst)), "l"(src) : "memory");
        }
        __device__ inline void cp_async_wait_all()
        {
            asm volatile("cp.async.commit_group;\n\tcp.async.wait_group 0;" ::: "memory");
        }

        // One CTA of 256 threads per group of NB bricks (persistent over groups).  The three x taps of a
        // (dz, dy) pair run as ONE MMA of N = 3 cout columns against the same A tile: column block dx of
        // row x holds W[dz, dy, dx] in[z + dz, y + dy, x], and the epilogue adds the blocks of x - 1, x and
        // x + 1, neighbouring lanes of a warp.  An MMA's time is its shared-memory reads (128 B per
        // clock: 4 KiB of A, 32 B per column of B), so 9 MMAs of 48 columns (43 clocks) replace 27 of 16 (36);
        // x needs no padding, and at the 4^3 level a tile holds one brick's rows at half instead of a
        // quarter of its lanes.
        // Two buffers of A (and of B, unless the layer's weights fit whole): the next 16 channels, also of
        // the next group, are staged while the MMAs run.
        // Shared memory: A [2][2][NPOS][16 B] | B [slots][9][2][3 cout][16 B] | barriers | TMEM address.
        template <int N, int NB>
        __global__ void __launch_bounds__(kConvThreads) conv_kernel(ConvParams p)
        {
            using Gm = Geometry<N, NB>;
            extern __shared__ __align__(128) uint8_t smem[];
            uint4* A = reinterpret_cast<uint4*>(smem);
            const int cout = p.cout, n3 = 3 * cout, b_size = 9 * 2 * n3;
            uint4* Bw = A + 4 * Gm::NPOS;
            uint64_t* bar = reinterpret_cast<uint64_t*>(Bw + p.weight_slots * b_size);
            uint32_t* tslot = reinterpret_cast<uint32_t*>(bar + 1);
            uint64_t* idle = bar + 2;      // initialised, never arrived on
            __shared__ int failed;
            const int tid = threadIdx.x, warp = tid >> 5;
            const uint32_t cols = tmem_columns(Gm::T * n3);

            for (int i = tid; i < 4 * Gm::NPOS; i += kConvThreads) A[i] = make_uint4(0, 0, 0, 0);
            if (tid == 0) { barrier_init(bar); barrier_init(idle); failed = 0; }
            if (warp == 0) tmem_alloc(tslot, cols);
            fence_before_sync();
            __syncthreads();
            fence_after_sync();
            const uint32_t tmem = *tslot;
            const uint32_t idesc = instruction_descriptor(n3);
            uint32_t phase = 0;
            const int groups = (p.samples + NB - 1) / NB;
            constexpr int V = N * N * N;
            int chunks = 0;                // of 16 channels, over both sources
            for (int si = 0; si < p.sources; ++si) chunks += p.src[si].channels / 16;
            const bool resident = p.weight_slots >= chunks;

            // stages 16 channels of the group's bricks and the matching weights: copies straight to shared
            // memory (cp.async) for plain and upsampled sources, a register average for pooled ones
            auto stage = [&](int group, int chunk, int slot, bool weights) {
                int si = 0, c0 = 16 * chunk;
                if (c0 >= p.src[0].channels) { si = 1; c0 -= p.src[0].channels; }
                const ConvSource& s = p.src[si];
                const int b0 = group * NB, items = min(NB, p.samples - b0) * V * 2;
                uint4* a = A + slot * 2 * Gm::NPOS;
                for (int i = tid; i < items; i += kConvThreads)
                {
                    const int half = i & 1, v = (i >> 1) % V, b = (i >> 1) / V;
                    const int x = v % N, y = (v / N) % N, z = v / (N * N);
                    uint4* to = &a[half * Gm::NPOS + padded<N>(b, x, y, z)];
                    if (s.mode != POOL) cp_async16(to, source_address<N>(s, b0 + b, x, y, z, c0 + 8 * half));
                    else *to = load_source<N>(s, b0 + b, x, y, z, c0 + 8 * half);
                }
                if (!weights) return;
                uint4* w = Bw + (resident ? chunk : slot) * b_size;
                for (int i = tid; i < b_size; i += kConvThreads)
                {
                    const int n = i % n3, half = (i / n3) & 1, zy = i / (2 * n3);
                    cp_async16(&w[i], s.w + (int64_t(zy) * n3 + n) * s.channels + c0 + 8 * half);
                }
            };

            int slot = 0;
            bool loaded = false;            // resident weights staged
            if (int(blockIdx.x) < groups)
            {
                stage(blockIdx.x, 0, 0, true);
                cp_async_wait_all();
                fence_async_shared();
                __syncthreads();
            }
            for (int group = blockIdx.x; group < groups; group += gridDim.x)
            {
                const int b0 = group * NB, nb = min(NB, p.samples - b0);
                for (int chunk = 0; chunk < chunks; ++chunk, slot ^= 1)
                {
                    if (tid == 0)
                    {
                        fence_after_sync();
                        const uint32_t a_base = smem_u32(A + slot * 2 * Gm::NPOS), b_base = smem_u32(Bw + (resident ? chunk : slot) * b_size);
                        for (int t = 0; t < Gm::T; ++t)
                            for (int zy = 0; zy < 9; ++zy)
                            {
                                const uint64_t a = smem_descriptor(a_base + uint32_t(Gm::tile_start(t) + row_shift<N>(zy)) * 16u,
                                                                   uint32_t(Gm::NPOS) * 16u, 128u);
                                const uint64_t b = smem_descriptor(b_base + uint32_t(zy * 2 * n3) * 16u, uint32_t(n3) * 16u, 128u);
                                mma_bf16(tmem + uint32_t(t * n3), a, b, idesc, (chunk == 0 && zy == 0) ? 0u : 1u);
                            }
                        mma_commit(bar);
                    }
                    // the next chunk goes into the other buffer, whose MMAs have been waited for
                    const bool next_group = chunk + 1 == chunks;
                    const int after = next_group ? group + int(gridDim.x) : group;
                    if (after < groups) stage(after, next_group ? 0 : chunk + 1, slot ^ 1, !(resident && (loaded || next_group)));
                    const bool done = p.idle_wait ? barrier_wait(idle, 0, p.wait_ns) : barrier_wait(bar, phase, p.wait_ns);
                    if (!done) failed = 1;
                    phase ^= 1;
                    cp_async_wait_all();
                    fence_async_shared();
                    __syncthreads();
                    if (failed) break;
                }
                loaded = true;
                if (failed) break;
                // epilogue: TMEM lane = tile row; warps w and w + 4 read lanes 32 (w % 4) .. + 31, alternate tiles
                fence_after_sync();
                const int m = 32 * (warp & 3) + (tid & 31), x = m % N;
                for (int t = warp >> 2; t < Gm::T; t += 2)
                {
                    const int pos = Gm::tile_start(t) + m;
                    const int b = pos / Gm::P, row = (pos % Gm::P) / N, zp = row / Gm::XP, yp = row % Gm::XP;
                    const bool valid = b < nb && zp >= 1 && zp <= N && yp >= 1 && yp <= N;
                    const int64_t voxel = (int64_t(b0 + b) * V + ((zp - 1) * N + (yp - 1)) * N + x);
                    for (int c = 0; c < cout; c += 16)
                    {
                        const uint32_t at = tmem + (uint32_t(32 * (warp & 3)) << 16) + uint32_t(t * n3 + c);
                        float v[16], w[16];
                        tmem_load16(at + uint32_t(cout), v);              // dx = 0
                        tmem_load16(at, w);                               // dx = -1, from x - 1
                        for (int i = 0; i < 16; ++i)
                        {
                            const float left = __shfl_up_sync(0xffffffffu, w[i], 1);
                            v[i] += x > 0 ? left : 0.0f;
                        }
                        tmem_load16(at + uint32_t(2 * cout), w);          // dx = +1, from x + 1
                        for (int i = 0; i < 16; ++i)
                        {
                            const float right = __shfl_down_sync(0xffffffffu, w[i], 1);
                            v[i] += x < N - 1 ? right : 0.0f;
                        }
                        if (!valid) continue;
                        if (p.relu)
                            for (int i = 0; i < 16; ++i) v[i] = fmaxf(v[i], 0.0f);
                        if (p.out_fp32)
                        {
                            float4* o = reinterpret_cast<float4*>(static_cast<float*>(p.y) + voxel * cout + c);
                            for (int i = 0; i < 4; ++i) o[i] = make_float4(v[4 * i], v[4 * i + 1], v[4 * i + 2], v[4 * i + 3]);
                        }
                        else
                        {
                            uint4* o = reinterpret_cast<uint4*>(static_cast<bf16*>(p.y) + voxel * cout + c);
                            o[0] = pack8(v);
                            o[1] = pack8(v + 8);
                        }
                    }
                }
                fence_before_sync();
                __syncthreads();
            }
            if (failed)
            {
                if (tid == 0) atomicExch(p.error, 1);
                // the last commit has not been seen: wait for it (fixed bound) before the tensor
                // memory its MMAs write is freed
                barrier_wait(bar, phase ^ 1, kMaxWaitNs);
            }
            fence_before_sync();
            __syncthreads();
            if (warp == 0) tmem_dealloc(tmem, cols);
        }

        // weights kept whole up to 44 KiB, else two buffers
        inline int weight_slots(int chunks, int cout) { return chunks * 9 * 2 * 3 * cout * 16 <= 44 * 1024 ? std::max(1, chunks) : 2; }
        template <int N, int NB> size_t conv_smem(int cout, int slots)
        {
            const size_t bytes = size_t(4) * Geometry<N, NB>::NPOS * 16 + size_t(slots) * 9 * 2 * 3 * cout * 16 + 32;
            // co-resident CTAs must fit their TMEM allocations into the SM's 512 columns
            const int cols = tmem_columns(Geometry<N, NB>::T * 3 * cout);
            const size_t floor_bytes = cols == 512 ? 116 * 1024 : cols == 256 ? 80 * 1024 : cols == 128 ? 48 * 1024 : 0;
            return std::max(bytes, floor_bytes);
        }

        // ---- elementwise / small kernels ----
        // network input for system bricks: x0 [bricks][512][16], scale [bricks]
        __global__ void prepare_kernel(const int* slots, int bricks, const double* r, const double* diag, const uint8_t* active,
                                       bf16* x0, float* scale)
        {
            const int b = blockIdx.x;
            if (b >= bricks) return;
            const int64_t q0 = int64_t(slots[b]) * 512;
            __shared__ double red[2][8];
            double q[2], ss = 0, cnt = 0;
            for (int k = 0; k < 2; ++k)
            {
                const int v = threadIdx.x + 256 * k;
                const int64_t qq = q0 + v;
                q[k] = active[qq] && diag[qq] > 0 ? r[qq] / diag[qq] : 0.0;
                ss += q[k] * q[k];
                cnt += active[qq] ? 1.0 : 0.0;
            }
            for (int o = 16; o; o >>= 1) { ss += __shfl_xor_sync(0xffffffffu, ss, o); cnt += __shfl_xor_sync(0xffffffffu, cnt, o); }
            if ((threadIdx.x & 31) == 0) { red[0][threadIdx.x >> 5] = ss; red[1][threadIdx.x >> 5] = cnt; }
            __syncthreads();
            double tss = 0, tcnt = 0;
            for (int w = 0; w < 8; ++w) { tss += red[0][w]; tcnt += red[1][w]; }
            double s = std::sqrt(tss / fmax(tcnt, 1.0));
            if (!(s > 0)) s = 1.0;
            if (threadIdx.x == 0) scale[b] = float(s);
            for (int k = 0; k < 2; ++k)
            {
                const int v = threadIdx.x + 256 * k;
                float f[8] = {float(q[k] / s), active[q0 + v] ? 1.0f : 0.0f, 0, 0, 0, 0, 0, 0}, zero[8] = {0, 0, 0, 0, 0, 0, 0, 0};
                uint4* o = reinterpret_cast<uint4*>(x0 + (int64_t(b) * 512 + v) * 16);
                o[0] = pack8(f);
                o[1] = pack8(zero);
            }
        }

        // z = s * head(d0) on the active cells of the system bricks
        __global__ void head_apply_kernel(const int* slots, int bricks, const bf16* d0, const float* head, const float* scale,
                                          const uint8_t* active, double* z)
        {
            const int64_t i = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
            if (i >= int64_t(bricks) * 512) return;
            const int b = int(i / 512), v = int(i % 512);
            const int64_t q = int64_t(slots[b]) * 512 + v;
            float f[16];
            const uint4* src = reinterpret_cast<const uint4*>(d0 + i * 16);
            unpack8(src[0], f);
            unpack8(src[1], f + 8);
            float acc = 0;
            for (int c = 0; c < 16; ++c) acc += f[c] * head[c];
            z[q] = active[q] ? double(scale[b]) * double(acc) : 0.0;
        }

        // EB fragments and other DOFs after the structured slots: one damped Jacobi step
        __global__ void jacobi_tail_kernel(int64_t begin, int64_t end, const double* r, const double* diag, const uint8_t* active, double* z)
        {
            const int64_t q = begin + int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
            if (q < end) z[q] = active[q] && diag[q] > 0 ? (2.0 / 3.0) * r[q] / diag[q] : 0.0;
        }

        // 256-thread block sum
        __device__ inline double block_sum(double v, double* red)
        {
            for (int o = 16; o; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
            __syncthreads();
            if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = v;
            __syncthreads();
            double t = 0;
            for (int w = 0; w < 8; ++w) t += red[w];
            return t;
        }

        // x = A_B^-1 b on one brick by conjugate gradients in shared memory: A_B is the operator's
        // diagonal block of the brick (the full diagonal D, minus h for every open face to a cell of
        // the same brick); 2 cells per thread, to 1e-8 relative or 400 iterations
        __device__ void brick_solve(const double* b, double* x, const uint8_t* code, const double* D, double h, double* ps, double* red)
        {
            double r[2], p[2], Ap[2];
            for (int k = 0; k < 2; ++k)
            {
                const int v = threadIdx.x + 256 * k;
                x[v] = 0;
                r[k] = b[v];
                p[k] = r[k];
                ps[v] = p[k];
            }
            double rr = block_sum(r[0] * r[0] + r[1] * r[1], red);
            const double stop = 1e-16 * rr;
            for (int it = 0; it < 400 && rr > stop; ++it)
            {
                __syncthreads();
                for (int k = 0; k < 2; ++k)
                {
                    const int v = threadIdx.x + 256 * k;
                    const int c[3] = {v & 7, (v >> 3) & 7, v >> 6};
                    double a = D[v] * ps[v];
                    for (int axis = 0; axis < 3; ++axis)
                        for (int pos = 0; pos < 2; ++pos)
                        {
                            const int q = c[axis] + (pos ? 1 : -1);
                            if (q < 0 || q > 7 || !(code[v] & (1u << (2 * axis + pos)))) continue;
                            a -= h * ps[v + (pos ? 1 : -1) * (axis == 0 ? 1 : axis == 1 ? 8 : 64)];
                        }
                    Ap[k] = D[v] > 0 ? a : 0.0;
                }
                const double pAp = block_sum(p[0] * Ap[0] + p[1] * Ap[1], red);
                if (!(pAp > 0)) break;
                const double alpha = rr / pAp;
                for (int k = 0; k < 2; ++k)
                {
                    x[threadIdx.x + 256 * k] += alpha * p[k];
                    r[k] -= alpha * Ap[k];
                }
                const double next = block_sum(r[0] * r[0] + r[1] * r[1], red);
                const double beta = next / rr;
                rr = next;
                __syncthreads();
                for (int k = 0; k < 2; ++k)
                {
                    p[k] = r[k] + beta * p[k];
                    ps[threadIdx.x + 256 * k] = p[k];
                }
            }
            __syncthreads();
        }

        // harvest: brick k of preconditioner call `pair` -> store slot; input D^-1 r / s, mask,
        // target z / s with z the multigrid output (local = 0) or the brick-local solve (local = 1)
        __global__ void harvest_kernel(const int* slots, int bricks, int64_t pair, int per_pair, uint64_t seed, int64_t capacity,
                                       const double* r, const double* z, const double* diag, const uint8_t* active, bf16* hx,
                                       uint8_t* hm, float* ht, int local, const uint8_t* code, const int* brick_level,
                                       const double* level_h)
        {
            const int k = blockIdx.x;
            const int64_t sample = pair * per_pair + k;
            if (sample >= capacity) return;
            uint64_t h = seed ^ (uint64_t(pair) * 0x9E3779B97F4A7C15ull) ^ (uint64_t(k) * 0xC2B2AE3D27D4EB4Full);
            h ^= h >> 33; h *= 0xff51afd7ed558ccdull; h ^= h >> 33; h *= 0xc4ceb9fe1a85ec53ull; h ^= h >> 33;
            const int b = int(h % uint64_t(bricks));
            const int64_t q0 = int64_t(slots[b]) * 512;
            __shared__ double red[2][8];
            double q[2], ss = 0, cnt = 0;
            for (int j = 0; j < 2; ++j)
            {
                const int64_t qq = q0 + threadIdx.x + 256 * j;
                q[j] = active[qq] && diag[qq] > 0 ? r[qq] / diag[qq] : 0.0;
                ss += q[j] * q[j];
                cnt += active[qq] ? 1.0 : 0.0;
            }
            for (int o = 16; o; o >>= 1) { ss += __shfl_xor_sync(0xffffffffu, ss, o); cnt += __shfl_xor_sync(0xffffffffu, cnt, o); }
            if ((threadIdx.x & 31) == 0) { red[0][threadIdx.x >> 5] = ss; red[1][threadIdx.x >> 5] = cnt; }
            __syncthreads();
            double tss = 0, tcnt = 0;
            for (int w = 0; w < 8; ++w) { tss += red[0][w]; tcnt += red[1][w]; }
            double s = std::sqrt(tss / fmax(tcnt, 1.0));
            if (!(s > 0)) s = 1.0;
            __shared__ double bs[512], xs[512], ps[512], Ds[512], red2[8];
            __shared__ uint8_t cs[512];
            if (local)
            {
                for (int j = 0; j < 2; ++j)
                {
                    const int v = threadIdx.x + 256 * j;
                    const int64_t qq = q0 + v;
                    const bool on = active[qq] && diag[qq] > 0;
                    bs[v] = on ? r[qq] : 0.0;
                    Ds[v] = on ? diag[qq] : 0.0;
                    cs[v] = on ? code[qq] : 0;
                }
                __syncthreads();
                brick_solve(bs, xs, cs, Ds, level_h[brick_level[slots[b]]], ps, red2);
            }
            for (int j = 0; j < 2; ++j)
            {
                const int v = threadIdx.x + 256 * j;
                const int64_t qq = q0 + v;
                hx[sample * 512 + v] = __float2bfloat16_rn(float(q[j] / s));
                hm[sample * 512 + v] = active[qq] ? 1 : 0;
                const double target = local ? xs[v] : z[qq];
                ht[sample * 512 + v] = active[qq] ? float(target / s) : 0.0f;
            }
        }

        // sum of squared targets and active count over the harvest store
        __global__ void target_moment_kernel(int64_t n, const uint8_t* hm, const float* ht, double* out)
        {
            double ss = 0, cnt = 0;
            for (int64_t i = int64_t(blockIdx.x) * blockDim.x + threadIdx.x; i < n; i += int64_t(gridDim.x) * blockDim.x)
                if (hm[i]) { ss += double(ht[i]) * ht[i]; cnt += 1; }
            for (int o = 16; o; o >>= 1) { ss += __shfl_xor_sync(0xffffffffu, ss, o); cnt += __shfl_xor_sync(0xffffffffu, cnt, o); }
            if ((threadIdx.x & 31) == 0) { atomicAdd(&out[0], ss); atomicAdd(&out[1], cnt); }
        }

        // training batch: x0 [batch][512][16], target * target_scale, mask; count += active cells
        __global__ void gather_batch_kernel(const int* index, int batch, const bf16* hx, const uint8_t* hm, const float* ht, float target_scale,
                                            bf16* x0, float* target, uint8_t* mask, float* count)
        {
            const int64_t i = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
            if (i >= int64_t(batch) * 512) return;
            const int b = int(i / 512), v = int(i % 512);
            const int64_t src = int64_t(index[b]) * 512 + v;
            float f[8] = {__bfloat162float(hx[src]), float(hm[src]), 0, 0, 0, 0, 0, 0}, zero[8] = {0, 0, 0, 0, 0, 0, 0, 0};
            uint4* o = reinterpret_cast<uint4*>(x0 + i * 16);
            o[0] = pack8(f);
            o[1] = pack8(zero);
            target[i] = ht[src] * target_scale;
            mask[i] = hm[src];
            // one add per warp (a warp's 32 voxels lie in one sample): 49 us for 64 samples with one per voxel
            const unsigned on = __ballot_sync(0xffffffffu, hm[src] != 0);
            if ((threadIdx.x & 31) == 0 && on) atomicAdd(count, float(__popc(on)));
        }

        // head forward + backward: zhat, loss, dhead, G4 = bf16(dz * head * [d0 > 0])
        __global__ void head_backward_kernel(int samples, const bf16* d0, const float* head, const float* target, const uint8_t* mask,
                                             const float* count, float* zhat, bf16* G4, float* dhead, float* loss)
        {
            const int64_t i = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
            float f[16], part[16], l = 0;
            for (int c = 0; c < 16; ++c) part[c] = 0;
            if (i < int64_t(samples) * 512)
            {
                const uint4* src = reinterpret_cast<const uint4*>(d0 + i * 16);
                unpack8(src[0], f);
                unpack8(src[1], f + 8);
                float acc = 0;
                for (int c = 0; c < 16; ++c) acc += f[c] * head[c];
                zhat[i] = acc;
                const float inv = 1.0f / fmaxf(*count, 1.0f);
                const float diff = mask[i] ? acc - target[i] : 0.0f;
                l = diff * diff * inv;
                const float dz = 2.0f * diff * inv;
                float g[16];
                for (int c = 0; c < 16; ++c)
                {
                    part[c] = f[c] * dz;
                    g[c] = f[c] > 0 ? dz * head[c] : 0.0f;
                }
                uint4* o = reinterpret_cast<uint4*>(G4 + i * 16);
                o[0] = pack8(g);
                o[1] = pack8(g + 8);
            }
            for (int o = 16; o; o >>= 1)
            {
                l += __shfl_xor_sync(0xffffffffu, l, o);
                for (int c = 0; c < 16; ++c) part[c] += __shfl_xor_sync(0xffffffffu, part[c], o);
            }
            // a CTA's warps in order, then one add per CTA and sum
            __shared__ float sums[kThreads / 32][17];
            if ((threadIdx.x & 31) == 0)
            {
                for (int c = 0; c < 16; ++c) sums[threadIdx.x >> 5][c] = part[c];
                sums[threadIdx.x >> 5][16] = l;
            }
            __syncthreads();
            if (threadIdx.x < 17)
            {
                float total = 0;
                for (int w = 0; w < kThreads / 32; ++w) total += sums[w][threadIdx.x];
                atomicAdd(threadIdx.x < 16 ? &dhead[threadIdx.x] : loss, total);
            }
        }

        // G = bf16(sum over the 8 children of U (fine level 2n) * [act > 0]) at level n
        __global__ void sum_children_relu_kernel(int samples, int n, int C, const float* U, const bf16* act, bf16* G)
        {
            const int64_t i = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
            const int V = n * n * n;
            if (i >= int64_t(samples) * V * C) return;
            const int c = int(i % C);
            const int64_t vb = i / C;
            const int v = int(vb % V);
            const int64_t b = vb / V;
            const int x = v % n, y = (v / n) % n, z = v / (n * n), F = 2 * n;
            float sum = 0;
            for (int k = 0; k < 8; ++k)
            {
                const int fx = 2 * x + (k & 1), fy = 2 * y + ((k >> 1) & 1), fz = 2 * z + (k >> 2);
                sum += U[((b * F + fz) * F + fy) * int64_t(F) * C + int64_t(fx) * C + c];
            }
            G[i] = __float2bfloat16_rn(__bfloat162float(act[i]) > 0 ? sum : 0.0f);
        }

        // G = bf16((S + P[parent] / 8) * [act > 0]) at level n (P at level n/2)
        __global__ void combine_relu_kernel(int samples, int n, int C, const float* S, const float* P, const bf16* act, bf16* G)
        {
            const int64_t i = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
            const int V = n * n * n;
            if (i >= int64_t(samples) * V * C) return;
            const int c = int(i % C);
            const int64_t vb = i / C;
            const int v = int(vb % V);
            const int64_t b = vb / V;
            const int x = v % n, y = (v / n) % n, z = v / (n * n), M = n / 2;
            const float parent = P[((b * M + z / 2) * M + y / 2) * int64_t(M) * C + int64_t(x / 2) * C + c];
            G[i] = __float2bfloat16_rn(__bfloat162float(act[i]) > 0 ? S[i] + 0.125f * parent : 0.0f);
        }

        // dW[t][co][ci] += sum_b sum_v G[b][v][co] * src[b][v + shift_t][ci]: per tap a (cout x voxels) by
        // (voxels x channels) product with K = the voxels, on m16n8k16 tensor-core tiles (BF16 operands,
        // FP32 sums).  mma.sync rather than tcgen05: the operand rows are voxels shifted by the tap, which
        // ldmatrix gathers row by row from the padded brick as it lies, and M = cout of 16 to 64 would fill
        // an eighth to a half of a 128-row tcgen05 tile.  A CTA stages kStage samples at a time
        // (padded source and G, rows 16 bytes apart from a multiple of the bank width, so that the
        // eight rows of a matrix fall on distinct banks); its eight warps hold two taps
        // each, all of cout x channels in registers, and add them to dW once per CTA.
        // Bound by staging and the final adds: 64 samples of the 8^3 layers take a few us of MMAs.
        // CUDA-core form: 327 us per 8^3 layer and 54 per 4^3 layer at 64 samples (56 to 108 CTAs, one
        // shared-memory read per two FMAs); a whole forward and backward pass on 64 samples went from
        // 1,766 to 600 us with this kernel and the batched counts and sums of the loss kernels.
        __device__ inline void load_matrices(uint32_t (&r)[4], const void* row)
        {
            asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0, %1, %2, %3}, [%4];"
                         : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(smem_u32(row)) : "memory");
        }
        __device__ inline void mma_tile(float (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1)
        {
            asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
                         : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3]) : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
        }
        template <int N> __host__ __device__ constexpr int wgrad_stage() { return N == 8 ? 1 : N == 4 ? 2 : 4; }   // K = 512, 128, 32 voxels
        template <int N, int COUT, int C>
        __global__ void __launch_bounds__(256) weight_grad_kernel(ConvSource s, const bf16* G, int samples, int chunk, float* dW)
        {
            constexpr int XP = N + 2, P = XP * XP * XP, V = N * N * N, kStage = wgrad_stage<N>();
            constexpr int XR = C + 8, GR = COUT + 8;        // row strides
            constexpr int MT = COUT / 16, NT = C / 8;
            extern __shared__ __align__(16) uint8_t wsm[];
            bf16* xs = reinterpret_cast<bf16*>(wsm);        // [kStage][P][XR]
            bf16* gs = xs + kStage * P * XR;                // [kStage * V][GR]
            const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
            for (int i = threadIdx.x; i < kStage * P * XR / 8; i += 256) reinterpret_cast<uint4*>(xs)[i] = make_uint4(0, 0, 0, 0);
            const int first = blockIdx.x * chunk, last = min(samples, first + chunk);
            // blockIdx.y 0: taps 0..15, 1: taps 16..26, two per warp
            constexpr int kTaps = 2;
            const int tap0 = 16 * int(blockIdx.y) + kTaps * warp, taps = min(kTaps, 27 - tap0);
            {
                float acc[kTaps][MT][NT][4] = {};
                int shift[kTaps];
#pragma unroll
                for (int k = 0; k < kTaps; ++k)
                {
                    const int tap = min(26, tap0 + k);
                    shift[k] = ((tap / 9) - 1) * XP * XP + ((tap / 3) % 3 - 1) * XP + (tap % 3) - 1;
                }
                for (int b = first; b < last; b += kStage)
                {
                    __syncthreads();
                    const int here = min(kStage, last - b);
                    for (int i = threadIdx.x; i < kStage * V * (C / 8); i += 256)
                    {
                        const int c0 = 8 * (i % (C / 8)), v = (i / (C / 8)) % V, k = i / (C / 8) / V;
                        const int x = v % N, y = (v / N) % N, z = v / (N * N);
                        reinterpret_cast<uint4*>(xs + (k * P + ((z + 1) * XP + y + 1) * XP + x + 1) * XR + c0)[0] =
                            k < here ? load_source<N>(s, b + k, x, y, z, c0) : make_uint4(0, 0, 0, 0);
                    }
                    for (int i = threadIdx.x; i < kStage * V * (COUT / 8); i += 256)
                    {
                        const int c0 = 8 * (i % (COUT / 8)), v = i / (COUT / 8);
                        reinterpret_cast<uint4*>(gs + v * GR + c0)[0] =
                            v / V < here ? *reinterpret_cast<const uint4*>(G + (int64_t(b) * V + v) * COUT + c0) : make_uint4(0, 0, 0, 0);
                    }
                    __syncthreads();
                    if (taps > 0)
                        for (int k0 = 0; k0 < kStage * V; k0 += 16)
                        {
                            // A (cout x 16 voxels) from G rows, B (16 voxels x channels) from shifted source rows
                            uint32_t a[MT][4];
                            const int ar = k0 + (lane & 7) + ((lane >> 4) << 3), ac = ((lane >> 3) & 1) << 3;
#pragma unroll
                            for (int m = 0; m < MT; ++m) load_matrices(a[m], gs + ar * GR + 16 * m + ac);
                            const int br = k0 + (lane & 7) + (((lane >> 3) & 1) << 3), bc = (lane >> 4) << 3;
                            const int v = br % V, sample = br / V;
                            const int pos = sample * P + ((v / (N * N) + 1) * XP + (v / N) % N + 1) * XP + v % N + 1;
#pragma unroll
                            for (int k = 0; k < kTaps; ++k)
#pragma unroll
                                for (int n = 0; n < NT; n += 2)
                                {
                                    uint32_t bm[4];
                                    load_matrices(bm, xs + (pos + shift[k]) * XR + 8 * n + bc);
#pragma unroll
                                    for (int m = 0; m < MT; ++m)
                                    {
                                        mma_tile(acc[k][m][n], a[m], bm[0], bm[1]);
                                        mma_tile(acc[k][m][n + 1], a[m], bm[2], bm[3]);
                                    }
                                }
                        }
                }
#pragma unroll
                for (int k = 0; k < kTaps; ++k)
                {
                    if (k >= taps) continue;
                    float* out = dW + int64_t(tap0 + k) * COUT * C;
#pragma unroll
                    for (int m = 0; m < MT; ++m)
#pragma unroll
                        for (int n = 0; n < NT; ++n)
                        {
                            const int co = 16 * m + (lane >> 2), ci = 8 * n + 2 * (lane & 3);
                            atomicAdd(out + co * C + ci, acc[k][m][n][0]);
                            atomicAdd(out + co * C + ci + 1, acc[k][m][n][1]);
                            atomicAdd(out + (co + 8) * C + ci, acc[k][m][n][2]);
                            atomicAdd(out + (co + 8) * C + ci + 1, acc[k][m][n][3]);
                        }
                }
            }
        }

        // BF16 forward weights, BF16 transposed weights (taps flipped, channels swapped) and the
        // BF16-rounded head from the FP32 masters
        __global__ void convert_weights_kernel(const float* master, bf16* forward, bf16* transposed, float* head)
        {
            const int64_t i = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
            if (i >= kParams) return;
            if (i >= kWeights)
            {
                head[i - kWeights] = __bfloat162float(__float2bfloat16_rn(master[i]));
                return;
            }
            int k = 0;
            while (k < 6 && i >= tensor_offset(k + 1)) ++k;
            const int64_t local = i - tensor_offset(k);
            const int cout = tensor_cout(k), cin = tensor_cin(k);
            const int tap = int(local / (int64_t(cout) * cin)), co = int((local / cin) % cout), ci = int(local % cin);
            const bf16 w = __float2bfloat16_rn(master[i]);
            forward[i] = w;
            transposed[tensor_offset(k) + (int64_t(26 - tap) * cin + ci) * cout + co] = w;
        }

        __global__ void adam_kernel(float* master, float* m, float* v, const float* grad, float lr, float b1, float b2, float c1, float c2)
        {
            const int64_t i = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
            if (i >= kParams) return;
            const float g = grad[i];
            const float mi = b1 * m[i] + (1 - b1) * g, vi = b2 * v[i] + (1 - b2) * g * g;
            m[i] = mi;
            v[i] = vi;
            master[i] -= lr * (mi / c1) / (sqrtf(vi / c2) + 1e-8f);
        }
    }

    // ==================================================================================
    // state
    // ==================================================================================
    struct Learned
    {
        DBuf<float> master, adam_m, adam_v, grad, head;
        DBuf<bf16> wf, wt;          // forward / transposed BF16 weights, flat parameter order
        bool has_weights = false;
        int64_t adam_step = 0;
        // activations for `capacity` samples
        int capacity = 0;
        DBuf<bf16> x0, e0, e1, bt, d1, d0, G4, G3, G2, G1, G0;
        DBuf<float> U0, S0, U1, S1, P1, P0, scale, zhat, target;
        DBuf<uint8_t> mask;
        DBuf<int> batch_index;
        DBuf<float> scalars;        // [0] count, [1] loss
        DBuf<bf16> eval_x;          // samples handed in by the host (learned_evaluate)
        DBuf<uint8_t> eval_mask;
        DBuf<float> eval_target;
        DBuf<int> error;
        bool harvesting = false;
        uint64_t wait_ns = kMaxWaitNs;   // limit of each tensor-core wait
        bool idle_wait_once = false;     // the next convolution's first wait runs out (fault-path check)
    };

    namespace
    {
        // Harvested training bricks.  One store per process (the device of the first system that
        // harvests), shared by every system, so pairs from several grids accumulate.
        struct Store
        {
            int device = -1, per_pair = 0, local = 1;
            int64_t capacity = 0, pairs = 0;
            uint64_t seed = 0;
            DBuf<bf16> hx;          // [capacity][512] D^-1 r / s
            DBuf<uint8_t> hm;       // [capacity][512] active mask
            DBuf<float> ht;         // [capacity][512] z / s
            int64_t samples() const { return std::min(pairs * per_pair, capacity); }
        };
        Store& store()
        {
            static Store* st = new Store();   // never destroyed: the CUDA context may be gone at exit
            return *st;
        }
    }

    namespace
    {
        bf16* wf(Learned& L, int k) { return L.wf.p + tensor_offset(k); }
        bf16* wt(Learned& L, int k) { return L.wt.p + tensor_offset(k); }

        void ensure_capacity(Learned& L, int samples)
        {
            if (samples <= L.capacity) return;
            L.capacity = 0;          // until all of them are there
            const size_t n = size_t(samples);
            L.x0.alloc(n * 512 * 16); L.e0.alloc(n * 512 * 16); L.e1.alloc(n * 64 * 32); L.bt.alloc(n * 8 * 64);
            L.d1.alloc(n * 64 * 32); L.d0.alloc(n * 512 * 16);
            L.G4.alloc(n * 512 * 16); L.G3.alloc(n * 64 * 32); L.G2.alloc(n * 8 * 64); L.G1.alloc(n * 64 * 32); L.G0.alloc(n * 512 * 16);
            L.U0.alloc(n * 512 * 32); L.S0.alloc(n * 512 * 16); L.U1.alloc(n * 64 * 64); L.S1.alloc(n * 64 * 32);
            L.P1.alloc(n * 8 * 32); L.P0.alloc(n * 64 * 16);
            L.scale.alloc(n); L.zhat.alloc(n * 512); L.target.alloc(n * 512); L.mask.alloc(n * 512); L.batch_index.alloc(n);
            L.capacity = samples;
        }

        Learned& state(System& s)
        {
            if (!s.learned)
            {
                auto fresh = std::make_unique<Learned>();
                Learned& L = *fresh;
                L.master.alloc(kParams); L.adam_m.alloc(kParams); L.adam_v.alloc(kParams); L.grad.alloc(kParams);
                L.head.alloc(kHead); L.wf.alloc(kWeights); L.wt.alloc(kWeights);
                L.scalars.alloc(4); L.error.alloc(1);
                s.learned = fresh.release();
            }
            return *s.learned;
        }

        int sm_count(System& s)
        {
            static int count = 0;
            if (!count) cuda_check(cudaDeviceGetAttribute(&count, cudaDevAttrMultiProcessorCount, s.device), "SM count");
            return count;
        }

        template <int N, int NB>
        void launch_conv(System& s, ConvParams p, int chunks)
        {
            p.weight_slots = weight_slots(chunks, p.cout);
            const size_t smem = conv_smem<N, NB>(p.cout, p.weight_slots);
            require(Geometry<N, NB>::T * 3 * p.cout <= 512 && smem <= 226 * 1024, "learned: output channels");
            // the largest request of any layer, so that one layer never lowers another's
            cuda_check(cudaFuncSetAttribute(conv_kernel<N, NB>, cudaFuncAttributeMaxDynamicSharedMemorySize, 226 * 1024), "conv smem");
            const int groups = (p.samples + NB - 1) / NB;
            const int per_sm = smem > 114 * 1024 ? 1 : smem > 76 * 1024 ? 2 : 3;
            conv_kernel<N, NB><<<std::min(groups, sm_count(s) * per_sm), kConvThreads, smem, launch_stream(s)>>>(p);
            cuda_check(cudaGetLastError(), "conv launch");
        }
        template <int N>
        void conv(System& s, Learned& L, int samples, int cout, ConvSource a, const ConvSource* b, void* y, bool relu, bool fp32)
        {
            if (!samples) return;
            ConvParams p{};
            p.src[0] = a;
            p.sources = 1;
            if (b) { p.src[1] = *b; p.sources = 2; }
            int chunks = 0;
            for (int k = 0; k < p.sources; ++k)
            {
                require(p.src[k].channels % 16 == 0 && p.src[k].channels <= 64, "learned: channel count");
                chunks += p.src[k].channels / 16;
            }
            require(cout % 16 == 0 && cout <= 64, "learned: output channels");
            p.cout = cout;
            p.samples = samples;
            p.relu = relu;
            p.out_fp32 = fp32;
            p.y = y;
            p.error = L.error;
            p.wait_ns = L.wait_ns;
            p.idle_wait = L.idle_wait_once ? 1 : 0;
            L.idle_wait_once = false;
            // bricks per CTA: as many tiles as the 512 TMEM columns hold, but one at the 8^3 level, where two
            // CTAs per SM then overlap their staging, MMAs and epilogues
            if constexpr (N == 8) launch_conv<8, 1>(s, p, chunks);
            else if constexpr (N == 4)
            {
                if (cout <= 32) launch_conv<4, 4>(s, p, chunks);
                else launch_conv<4, 2>(s, p, chunks);
            }
            else launch_conv<2, 8>(s, p, chunks);
        }

        template <int N, int COUT, int C>
        void weight_grad(System& s, ConvSource src, const bf16* G, int samples, float* dW)
        {
            constexpr int P = (N + 2) * (N + 2) * (N + 2), V = N * N * N, kStage = wgrad_stage<N>();
            constexpr int smem = kStage * (P * (C + 8) + V * (COUT + 8)) * 2;
            static_assert(smem <= 200 * 1024 && COUT % 16 == 0 && C % 16 == 0 && (kStage * V) % 16 == 0, "weight-gradient tiles");
            require(src.channels == C, "learned: weight-gradient channels");
            cuda_check(cudaFuncSetAttribute(weight_grad_kernel<N, COUT, C>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem), "wgrad smem");
            // two CTAs (tap halves) per run of samples; runs of whole stages, about one wave of CTAs
            const int runs = std::max(1, sm_count(s) / 2), chunk = (samples + runs * kStage - 1) / (runs * kStage) * kStage;
            weight_grad_kernel<N, COUT, C><<<dim3(unsigned((samples + chunk - 1) / chunk), 2), 256, smem, launch_stream(s)>>>(src, G, samples, chunk, dW);
        }

        ConvSource source(const bf16* x, const bf16* w, int channels, int mode) { return ConvSource{x, w, channels, mode}; }

        // forward from L.x0 through d0 for `samples` samples
        void forward(System& s, Learned& L, int samples)
        {
            conv<8>(s, L, samples, 16, source(L.x0, wf(L, ENC0), 16, SAME), nullptr, L.e0, true, false);
            conv<4>(s, L, samples, 32, source(L.e0, wf(L, ENC1), 16, POOL), nullptr, L.e1, true, false);
            conv<2>(s, L, samples, 64, source(L.e1, wf(L, BOTT), 32, POOL), nullptr, L.bt, true, false);
            const ConvSource skip1 = source(L.e1, wf(L, DEC1B), 32, SAME);
            conv<4>(s, L, samples, 32, source(L.bt, wf(L, DEC1A), 64, UP), &skip1, L.d1, true, false);
            const ConvSource skip0 = source(L.e0, wf(L, DEC0B), 16, SAME);
            conv<8>(s, L, samples, 16, source(L.d1, wf(L, DEC0A), 32, UP), &skip0, L.d0, true, false);
        }

        // backward from the loss on L.target / L.mask; gradients accumulate into L.grad (zeroed here)
        void backward(System& s, Learned& L, int samples)
        {
            cuda_check(cudaMemsetAsync(L.grad, 0, kParams * sizeof(float), s.stream), "zero gradients");
            cuda_check(cudaMemsetAsync(L.scalars.p + 1, 0, sizeof(float), s.stream), "zero loss");
            float* g = L.grad;
            const int64_t V8 = int64_t(samples) * 512;
            head_backward_kernel<<<blocks_for(V8), kThreads, 0, launch_stream(s)>>>(samples, L.d0, L.head, L.target, L.mask, L.scalars.p,
                                                                                     L.zhat, L.G4, g + kWeights, L.scalars.p + 1);
            // dec0
            conv<8>(s, L, samples, 32, source(L.G4, wt(L, DEC0A), 16, SAME), nullptr, L.U0, false, true);
            conv<8>(s, L, samples, 16, source(L.G4, wt(L, DEC0B), 16, SAME), nullptr, L.S0, false, true);
            weight_grad<8, 16, 32>(s, source(L.d1, nullptr, 32, UP), L.G4, samples, g + tensor_offset(DEC0A));
            weight_grad<8, 16, 16>(s, source(L.e0, nullptr, 16, SAME), L.G4, samples, g + tensor_offset(DEC0B));
            sum_children_relu_kernel<<<blocks_for(int64_t(samples) * 64 * 32), kThreads, 0, launch_stream(s)>>>(samples, 4, 32, L.U0, L.d1, L.G3);
            // dec1
            conv<4>(s, L, samples, 64, source(L.G3, wt(L, DEC1A), 32, SAME), nullptr, L.U1, false, true);
            conv<4>(s, L, samples, 32, source(L.G3, wt(L, DEC1B), 32, SAME), nullptr, L.S1, false, true);
            weight_grad<4, 32, 64>(s, source(L.bt, nullptr, 64, UP), L.G3, samples, g + tensor_offset(DEC1A));
            weight_grad<4, 32, 32>(s, source(L.e1, nullptr, 32, SAME), L.G3, samples, g + tensor_offset(DEC1B));
            sum_children_relu_kernel<<<blocks_for(int64_t(samples) * 8 * 64), kThreads, 0, launch_stream(s)>>>(samples, 2, 64, L.U1, L.bt, L.G2);
            // bottleneck
            conv<2>(s, L, samples, 32, source(L.G2, wt(L, BOTT), 64, SAME), nullptr, L.P1, false, true);
            weight_grad<2, 64, 32>(s, source(L.e1, nullptr, 32, POOL), L.G2, samples, g + tensor_offset(BOTT));
            combine_relu_kernel<<<blocks_for(int64_t(samples) * 64 * 32), kThreads, 0, launch_stream(s)>>>(samples, 4, 32, L.S1, L.P1, L.e1, L.G1);
            // enc1
            conv<4>(s, L, samples, 16, source(L.G1, wt(L, ENC1), 32, SAME), nullptr, L.P0, false, true);
            weight_grad<4, 32, 16>(s, source(L.e0, nullptr, 16, POOL), L.G1, samples, g + tensor_offset(ENC1));
            combine_relu_kernel<<<blocks_for(int64_t(samples) * 512 * 16), kThreads, 0, launch_stream(s)>>>(samples, 8, 16, L.S0, L.P0, L.e0, L.G0);
            // enc0
            weight_grad<8, 16, 16>(s, source(L.x0, nullptr, 16, SAME), L.G0, samples, g + tensor_offset(ENC0));
        }

        void convert(System& s, Learned& L)
        {
            convert_weights_kernel<<<blocks_for(kParams), kThreads, 0, launch_stream(s)>>>(L.master, L.wf, L.wt, L.head);
            L.has_weights = true;
        }

        void check_error(System& s, Learned& L)
        {
            int e = 0;
            cuda_check(cudaMemcpyAsync(&e, L.error, sizeof(int), cudaMemcpyDeviceToHost, s.stream), "learned error flag");
            cuda_check(cudaStreamSynchronize(s.stream), "learned sync");
            if (e)
            {
                cuda_check(cudaMemsetAsync(L.error, 0, sizeof(int), s.stream), "reset error flag");
                throw Error(PCFD_TIMEOUT, "learned preconditioner: a tensor-core wait timed out");
            }
        }

        void default_parameters(System& s, Learned& L)
        {
            // He-normal weights from a fixed seed, as oracle/unet.py init_params draws them in shape
            std::vector<float> p(static_cast<size_t>(kParams));
            std::mt19937_64 rng(20261203);
            std::normal_distribution<double> normal(0.0, 1.0);
            for (int k = 0; k < 7; ++k)
            {
                const double sd = std::sqrt(2.0 / (27.0 * tensor_cin(k)));
                for (int64_t i = 0; i < tensor_size(k); ++i) p[size_t(tensor_offset(k) + i)] = float(sd * normal(rng));
            }
            for (int c = 0; c < kHead; ++c) p[size_t(kWeights + c)] = float(0.25 * normal(rng));
            cuda_check(cudaMemcpyAsync(L.master, p.data(), p.size() * sizeof(float), cudaMemcpyHostToDevice, s.stream), "upload parameters");
            convert(s, L);
        }
    }

    // ==================================================================================
    // entry points used by the solver and the C ABI
    // ==================================================================================
    int64_t learned_parameter_count() { return kParams; }

    void learned_destroy(System& s)
    {
        delete s.learned;
        s.learned = nullptr;
    }

    void learned_set_parameters(System& s, const float* host, int64_t count)
    {
        require(count == kParams, "learned: parameter count mismatch");
        Learned& L = state(s);
        cuda_check(cudaMemcpyAsync(L.master, host, size_t(kParams) * sizeof(float), cudaMemcpyHostToDevice, s.stream), "upload parameters");
        cuda_check(cudaMemsetAsync(L.adam_m, 0, size_t(kParams) * sizeof(float), s.stream), "reset adam");
        cuda_check(cudaMemsetAsync(L.adam_v, 0, size_t(kParams) * sizeof(float), s.stream), "reset adam");
        L.adam_step = 0;
        convert(s, L);
        cuda_check(cudaStreamSynchronize(s.stream), "set parameters");
    }

    void learned_get_parameters(System& s, float* host, int64_t count)
    {
        require(count == kParams, "learned: parameter count mismatch");
        Learned& L = state(s);
        if (!L.has_weights) default_parameters(s, L);
        cuda_check(cudaMemcpyAsync(host, L.master, size_t(kParams) * sizeof(float), cudaMemcpyDeviceToHost, s.stream), "download parameters");
        cuda_check(cudaStreamSynchronize(s.stream), "get parameters");
    }

    // z = net(r) on the structured bricks, one damped Jacobi step on the DOFs after them
    void learned_apply(System& s, const double* r, double* z)
    {
        Learned& L = state(s);
        if (!L.has_weights) default_parameters(s, L);
        const int bricks = s.active_bricks;
        ensure_capacity(L, bricks);
        cuda_check(cudaMemsetAsync(z, 0, size_t(s.structured) * sizeof(double), s.stream), "clear z");
        if (bricks)
        {
            prepare_kernel<<<bricks, 256, 0, launch_stream(s)>>>(s.active_brick_list, bricks, r, s.diagonal, s.active, L.x0, L.scale);
            forward(s, L, bricks);
            head_apply_kernel<<<blocks_for(int64_t(bricks) * 512), kThreads, 0, launch_stream(s)>>>(s.active_brick_list, bricks, L.d0, L.head,
                                                                                                   L.scale, s.active, z);
        }
        if (s.Sp > s.structured)
            jacobi_tail_kernel<<<blocks_for(int64_t(s.Sp) - s.structured), kThreads, 0, launch_stream(s)>>>(s.structured, s.S, r, s.diagonal,
                                                                                                          s.active, z);
    }

    void learned_check(System& s)
    {
        if (s.learned) check_error(s, *s.learned);
    }

    void learned_set_wait(System& s, double seconds, bool idle_barrier_once)
    {
        require(seconds > 0 && seconds <= 60, "learned: wait limit must be in (0, 60] s");
        Learned& L = state(s);
        L.wait_ns = uint64_t(seconds * 1e9);
        L.idle_wait_once = idle_barrier_once;
    }

    void learned_harvest_begin(System& s, int capacity_pairs, int per_pair, uint64_t seed, int target)
    {
        require(capacity_pairs > 0 && per_pair > 0 && per_pair <= 4096, "learned: harvest sizes");
        require(target == PCFD_LEARNED_TARGET_MULTIGRID || target == PCFD_LEARNED_TARGET_BRICK_SOLVE, "learned: harvest target");
        require(target == PCFD_LEARNED_TARGET_MULTIGRID || s.fine.enabled, "learned: the brick-solve target needs 8^3 bricks");
        Learned& L = state(s);
        Store& st = store();
        require(st.device < 0 || st.device == s.device, "learned: the harvest store lives on another device");
        const int64_t capacity = int64_t(capacity_pairs) * per_pair;
        if (capacity != st.capacity || per_pair != st.per_pair || target != st.local)
        {
            cuda_check(cudaStreamSynchronize(s.stream), "harvest store");
            st.hx.alloc(size_t(capacity) * 512);
            st.hm.alloc(size_t(capacity) * 512);
            st.ht.alloc(size_t(capacity) * 512);
            st.capacity = capacity;
            st.per_pair = per_pair;
            st.pairs = 0;
            st.device = s.device;
            st.local = target;
        }
        st.seed = seed;
        L.harvesting = true;
    }

    int64_t learned_harvest_stop(System& s)
    {
        if (s.learned) s.learned->harvesting = false;
        return store().samples();
    }

    bool learned_harvesting(const System& s) { return s.learned && s.learned->harvesting; }

    void learned_harvest(System& s, const double* r, const double* z)
    {
        Store& st = store();
        if (!s.active_bricks || st.pairs * st.per_pair >= st.capacity) return;
        harvest_kernel<<<st.per_pair, 256, 0, launch_stream(s)>>>(s.active_brick_list, s.active_bricks, st.pairs, st.per_pair,
                                                                  st.seed, st.capacity, r, z, s.diagonal, s.active, st.hx, st.hm, st.ht,
                                                                  st.local, s.fine.code, s.brick_level, s.d_level_h);
        ++st.pairs;
    }

    namespace
    {
        // head master weights *= factor (and the BF16 copies)
        void scale_head(System& s, Learned& L, double factor)
        {
            float h[kHead];
            cuda_check(cudaMemcpyAsync(h, L.master.p + kWeights, sizeof(h), cudaMemcpyDeviceToHost, s.stream), "head");
            cuda_check(cudaStreamSynchronize(s.stream), "head");
            for (float& v : h) v = float(v * factor);
            cuda_check(cudaMemcpyAsync(L.master.p + kWeights, h, sizeof(h), cudaMemcpyHostToDevice, s.stream), "head");
            cuda_check(cudaStreamSynchronize(s.stream), "head");
            convert(s, L);
        }

        // one optimiser step on L.x0 / target / mask for `batch` samples; returns nothing (loss on device)
        void train_step(System& s, Learned& L, int batch, float lr)
        {
            forward(s, L, batch);
            backward(s, L, batch);
            ++L.adam_step;
            const float b1 = 0.9f, b2 = 0.999f;
            const float c1 = 1.0f - std::pow(b1, float(L.adam_step)), c2 = 1.0f - std::pow(b2, float(L.adam_step));
            adam_kernel<<<blocks_for(kParams), kThreads, 0, launch_stream(s)>>>(L.master, L.adam_m, L.adam_v, L.grad, lr, b1, b2, c1, c2);
            convert(s, L);
        }
    }

    // `steps` Adam steps on random batches of the harvested samples; returns the mean loss of the
    // last min(steps, 50) steps
    double learned_train(System& s, int steps, int batch, double lr, uint64_t seed)
    {
        require(steps >= 0 && batch > 0 && lr > 0, "learned: training arguments");
        Learned& L = state(s);
        if (!L.has_weights) default_parameters(s, L);
        Store& st = store();
        const int64_t samples = st.samples();
        require(samples > 0 && st.device == s.device, "learned: no harvested samples on this device to train on");
        ensure_capacity(L, batch);
        // Targets (multigrid corrections over D^-1 r / s) are 10^2..10^4 in size: train against
        // targets divided by their RMS tau over the store, with the head divided by tau, and fold
        // tau back into the head afterwards (the head is linear, so the trained map is unchanged).
        double tau = 1.0;
        {
            DBuf<double> moment;
            moment.alloc(2);
            target_moment_kernel<<<4 * sm_count(s), 256, 0, launch_stream(s)>>>(samples * 512, st.hm, st.ht, moment);
            double h[2] = {0, 0};
            cuda_check(cudaMemcpyAsync(h, moment.p, sizeof(h), cudaMemcpyDeviceToHost, s.stream), "target moment");
            cuda_check(cudaStreamSynchronize(s.stream), "target moment");
            if (h[1] > 0 && h[0] > 0) tau = std::sqrt(h[0] / h[1]);
        }
        scale_head(s, L, 1.0 / tau);
        cuda_check(cudaMemsetAsync(L.adam_m, 0, size_t(kParams) * sizeof(float), s.stream), "reset adam");
        cuda_check(cudaMemsetAsync(L.adam_v, 0, size_t(kParams) * sizeof(float), s.stream), "reset adam");
        L.adam_step = 0;
        std::mt19937_64 rng(seed);
        std::vector<int> index(static_cast<size_t>(batch));
        std::vector<float> losses;
        const int tail = std::min(steps, 50);
        float* pinned = nullptr;
        cuda_check(cudaMallocHost(&pinned, size_t(std::max(tail, 1)) * sizeof(float)), "pinned losses");
        try
        {
            for (int step = 0; step < steps; ++step)
            {
                for (int& i : index) i = int(rng() % uint64_t(samples));
                cuda_check(cudaMemcpyAsync(L.batch_index, index.data(), index.size() * sizeof(int), cudaMemcpyHostToDevice, s.stream),
                           "batch indices");
                cuda_check(cudaMemsetAsync(L.scalars, 0, sizeof(float), s.stream), "zero count");
                gather_batch_kernel<<<blocks_for(int64_t(batch) * 512), kThreads, 0, launch_stream(s)>>>(L.batch_index, batch, st.hx, st.hm,
                                                                                                        st.ht, float(1.0 / tau), L.x0, L.target,
                                                                                                        L.mask, L.scalars);
                // cosine decay to 10 % of the initial rate
                const double frac = steps > 1 ? double(step) / double(steps - 1) : 0.0;
                const float rate = float(lr * (0.1 + 0.45 * (1.0 + std::cos(M_PI * frac))));
                train_step(s, L, batch, rate);
                if (step >= steps - tail)
                    cuda_check(cudaMemcpyAsync(pinned + (step - (steps - tail)), L.scalars.p + 1, sizeof(float), cudaMemcpyDeviceToHost, s.stream),
                               "loss");
                // the host synchronises every 64 steps so that the batch indices stay in order
                if ((step & 63) == 63) cuda_check(cudaStreamSynchronize(s.stream), "train sync");
            }
            check_error(s, L);
            scale_head(s, L, tau);
        }
        catch (...)
        {
            cudaFreeHost(pinned);
            throw;
        }
        double mean = 0;
        for (int i = 0; i < tail; ++i) mean += pinned[i];
        cudaFreeHost(pinned);
        return tail ? mean / tail : 0.0;
    }

    // forward (and, with gradients != null, backward) on host samples: x [n][512][2] (input
    // channel 0 and mask), target [n][512]; returns the loss, zhat [n][512], gradients [params]
    double learned_evaluate(System& s, int n, const float* x, const float* target, float* zhat, float* gradients)
    {
        require(n > 0 && x && target && zhat, "learned: evaluate arguments");
        Learned& L = state(s);
        if (!L.has_weights) default_parameters(s, L);
        ensure_capacity(L, n);
        std::vector<uint16_t> hx(size_t(n) * 512);
        std::vector<uint8_t> hm(size_t(n) * 512);
        for (size_t i = 0; i < hx.size(); ++i)
        {
            const bf16 b = __float2bfloat16_rn(x[2 * i]);
            std::memcpy(&hx[i], &b, 2);
            hm[i] = x[2 * i + 1] != 0 ? 1 : 0;
        }
        if (L.eval_x.n < hx.size())
        {
            L.eval_x.release();      // the last to be allocated: its size stands for all three
            L.eval_mask.alloc(hm.size(), false);
            L.eval_target.alloc(hx.size(), false);
            L.eval_x.alloc(hx.size(), false);
        }
        cuda_check(cudaMemcpyAsync(L.eval_x, hx.data(), hx.size() * sizeof(bf16), cudaMemcpyHostToDevice, s.stream), "upload inputs");
        cuda_check(cudaMemcpyAsync(L.eval_mask, hm.data(), hm.size(), cudaMemcpyHostToDevice, s.stream), "upload masks");
        cuda_check(cudaMemcpyAsync(L.eval_target, target, hx.size() * sizeof(float), cudaMemcpyHostToDevice, s.stream), "upload targets");
        std::vector<int> index(static_cast<size_t>(n));
        for (int i = 0; i < n; ++i) index[size_t(i)] = i;
        cuda_check(cudaMemcpyAsync(L.batch_index, index.data(), index.size() * sizeof(int), cudaMemcpyHostToDevice, s.stream), "indices");
        cuda_check(cudaMemsetAsync(L.scalars, 0, sizeof(float), s.stream), "zero count");
        gather_batch_kernel<<<blocks_for(int64_t(n) * 512), kThreads, 0, launch_stream(s)>>>(L.batch_index, n, L.eval_x, L.eval_mask, L.eval_target, 1.0f, L.x0,
                                                                                            L.target, L.mask, L.scalars);
        forward(s, L, n);
        backward(s, L, n);
        float loss = 0;
        cuda_check(cudaMemcpyAsync(&loss, L.scalars.p + 1, sizeof(float), cudaMemcpyDeviceToHost, s.stream), "loss");
        cuda_check(cudaMemcpyAsync(zhat, L.zhat, size_t(n) * 512 * sizeof(float), cudaMemcpyDeviceToHost, s.stream), "zhat");
        if (gradients)
            cuda_check(cudaMemcpyAsync(gradients, L.grad, size_t(kParams) * sizeof(float), cudaMemcpyDeviceToHost, s.stream), "gradients");
        check_error(s, L);
        return loss;
    }
}
