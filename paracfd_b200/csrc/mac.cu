// mac.cu -- the staggered MAC momentum mode: semi-Lagrangian MacCormack advection of the face
// velocities with a limited MUSCL update in the near-fabric band, Smagorinsky eddy viscosity and
// explicit face diffusion, on every AMR level at once.
//
// This is the reference's non-default momentum path (DeviceAmrAdvection::advect and
// diffuse_smagorinsky, src/core/fluid/amr_advection.cu:588-720 and 1663-1690), restated on the
// compact per-brick face layout (no ghost rings) in the reference's FP32 arithmetic:
//   forward   each face node is traced back with a two-stage (midpoint) characteristic and the
//             field is sampled trilinearly on the finest brick that owns the foot; faces in the
//             near-fabric band (link bit 6) take a limited MUSCL update along their open
//             same-side links instead (amr_advection.cu:633-647)
//   correct   MacCormack: the forward field is traced forward again and half the round-trip
//             error is added back, clamped to the backward foot's eight samples -- only when the
//             node and both feet lie on the face's own level (amr_advection.cu:653-666)
//   LES       nut = (cs h)^2 |S| from central differences of the sampled velocity (:705-708)
//   diffusion explicit 7-point face Laplacian with nu + mean nut of the two cells across the
//             face; band faces use only their open links and molecular nu (:709-713)
// Samples that leave a brick take the same-level neighbour across one face, else the finest brick
// that contains the lattice node (one-sided linear extension across 2:1 transitions).  That value
// depends on the node alone, so each field is first copied into per-brick lattices with one ghost
// node all round (extend): every sample then reads its eight nodes from one brick's lattice.  One
// launch covers all brick slots of all levels; covered bricks are skipped (their output faces are 0, as
// the reference's scratch commit leaves them).  The link bytes are the caller's preprocessing
// (the fabric band and its open directions come from the caller's surface BVH).
#include "locator.h"

#include <algorithm>
#include <cstring>
#include <vector>

namespace pcfd
{
    namespace
    {
        struct MacView
        {
            LocatorView loc;
            const int* neighbour;       // [B][6] same-level neighbour slot or -1
            const uint32_t* flags;      // [B] brick flags by slot
            const int* slot_level;      // [B]
            int bs;
            const float* ext;           // the sampled field's extended lattices (ext_index), one ghost node all round
        };
        struct Faces
        {
            const float* c[3];
        };

        __device__ inline bool valid_face(int c, int bs, int i, int j, int k)
        {
            return i >= 0 && j >= 0 && k >= 0 && i < (c == 0 ? bs + 1 : bs) && j < (c == 1 ? bs + 1 : bs) && k < (c == 2 ? bs + 1 : bs);
        }
        __device__ inline float4 record_of(const MacView& m, int level, int64_t slot)
        {
            const LocatorLevel lev = m.loc.levels[level];
            return lev.record[slot - lev.slot0];
        }
        __device__ inline bool covered(const MacView& m, int64_t slot) { return (m.flags[slot] & PCFD_BRICK_COVERED) != 0; }

        // face index / value with indices clamped to the component's lattice of the brick
        __device__ inline int64_t clamped_face(int bs, int c, int64_t slot, int i, int j, int k)
        {
            i = max(0, min(c == 0 ? bs : bs - 1, i));
            j = max(0, min(c == 1 ? bs : bs - 1, j));
            k = max(0, min(c == 2 ? bs : bs - 1, k));
            return axis_face(bs, c, slot, i, j, k);
        }
        __device__ inline float clamped(const Faces& f, int bs, int c, int64_t slot, int i, int j, int k)
        {
            return f.c[c][clamped_face(bs, c, slot, i, j, k)];
        }
        // Extended lattice of component c of brick `slot`: its nodes -1 .. n per axis, [slot][c][k][j][i].
        __host__ __device__ inline int ext_size(int bs) { return (bs + 3) * (bs + 2) * (bs + 2); }
        __device__ inline bool in_extended(int c, int bs, int i, int j, int k)
        {
            return i >= -1 && j >= -1 && k >= -1 && i <= (c == 0 ? bs + 1 : bs) && j <= (c == 1 ? bs + 1 : bs) && k <= (c == 2 ? bs + 1 : bs);
        }
        __device__ inline int64_t ext_index(int c, int bs, int64_t slot, int i, int j, int k)
        {
            const int nx = c == 0 ? bs + 3 : bs + 2, ny = c == 1 ? bs + 3 : bs + 2;
            return (slot * 3 + c) * ext_size(bs) + ((k + 1) * ny + j + 1) * nx + i + 1;
        }
        // one-sided linear extension past the lattice ends (weights 2, -1 per axis)
        __device__ float extended(const Faces& f, int bs, int c, int64_t slot, int i, int j, int k)
        {
            const int n[3] = {c == 0 ? bs + 1 : bs, c == 1 ? bs + 1 : bs, c == 2 ? bs + 1 : bs}, want[3] = {i, j, k};
            int at[3][2], count[3];
            float w[3][2];
            for (int a = 0; a < 3; ++a)
            {
                if (want[a] < 0) { at[a][0] = 0; at[a][1] = 1; w[a][0] = 2.0f; w[a][1] = -1.0f; count[a] = 2; }
                else if (want[a] >= n[a]) { at[a][0] = n[a] - 1; at[a][1] = n[a] - 2; w[a][0] = 2.0f; w[a][1] = -1.0f; count[a] = 2; }
                else { at[a][0] = want[a]; w[a][0] = 1.0f; count[a] = 1; }
            }
            float result = 0;
            for (int az = 0; az < count[2]; ++az)
                for (int ay = 0; ay < count[1]; ++ay)
                    for (int ax = 0; ax < count[0]; ++ax)
                        result += w[0][ax] * w[1][ay] * w[2][az] * clamped(f, bs, c, slot, at[0][ax], at[1][ay], at[2][az]);
            return result;
        }
        // trilinear sample of component c at point p inside brick `slot`, with the extension
        __device__ float sample_extended(const Faces& f, int bs, const float4& rec, int c, int64_t slot, float px, float py, float pz)
        {
            float x = (px - rec.x) / rec.w - (c == 0 ? 0.0f : 0.5f);
            float y = (py - rec.y) / rec.w - (c == 1 ? 0.0f : 0.5f);
            float z = (pz - rec.z) / rec.w - (c == 2 ? 0.0f : 0.5f);
            const int i0 = int(floorf(x)), j0 = int(floorf(y)), k0 = int(floorf(z));
            x -= i0;
            y -= j0;
            z -= k0;
            float result = 0;
            for (int dz = 0; dz < 2; ++dz)
                for (int dy = 0; dy < 2; ++dy)
                    for (int dx = 0; dx < 2; ++dx)
                    {
                        const float wx = dx ? x : 1.0f - x, wy = dy ? y : 1.0f - y, wz = dz ? z : 1.0f - z;
                        result += wx * wy * wz * extended(f, bs, c, slot, i0 + dx, j0 + dy, k0 + dz);
                    }
            return result;
        }
        __device__ inline void face_point(const float4& rec, int c, int i, int j, int k, float& x, float& y, float& z)
        {
            x = rec.x + (i + (c == 0 ? 0.0f : 0.5f)) * rec.w;
            y = rec.y + (j + (c == 1 ? 0.0f : 0.5f)) * rec.w;
            z = rec.z + (k + (c == 2 ? 0.0f : 0.5f)) * rec.w;
        }
        __device__ inline int nearest_index(float coordinate, float origin, float h, float offset)
        {
            return int(floorf((coordinate - origin) / h - offset + 0.5f));
        }
        // finest non-covered brick containing the point: level, slot (or -1)
        __device__ inline int locate(const MacView& m, float x, float y, float z, int& level)
        {
            int where[5];
            locate_one(m.loc, x, y, z, where);
            level = where[0];
            return where[0] < 0 ? -1 : m.loc.levels[where[0]].slot0 + where[1];
        }
        // the face on which a brick boundary lies: 0..5, or -1 when outside more than one face
        __device__ inline int outside_face(int nx, int ny, int nz, int i, int j, int k)
        {
            int face = -1, outside = 0;
            if (i < 0) { face = 0; ++outside; } else if (i >= nx) { face = 1; ++outside; }
            if (j < 0) { face = 2; ++outside; } else if (j >= ny) { face = 3; ++outside; }
            if (k < 0) { face = 4; ++outside; } else if (k >= nz) { face = 5; ++outside; }
            return outside == 1 ? face : -1;
        }
        __device__ inline void shift_into(int face, int bs, int& i, int& j, int& k)
        {
            if (face == 0) i += bs; else if (face == 1) i -= bs; else if (face == 2) j += bs;
            else if (face == 3) j -= bs; else if (face == 4) k += bs; else k -= bs;
        }

        // Where the value of lattice node (i,j,k) of component c of brick `slot` (level `level`) comes
        // from, which may lie outside the brick: the index of one face of the component, or -1 when it
        // is interpolated on another level's brick `at` (at the node's position nx, ny, nz).  It
        // depends on the grid only.
        __device__ inline int64_t node_source(const MacView& m, int level, int64_t slot, int c, int i, int j, int k, int& at, int& at_level,
                                              float& nx, float& ny, float& nz)
        {
            const int bs = m.bs;
            if (valid_face(c, bs, i, j, k)) return axis_face(bs, c, slot, i, j, k);
            const int face = outside_face(c == 0 ? bs + 1 : bs, c == 1 ? bs + 1 : bs, c == 2 ? bs + 1 : bs, i, j, k);
            if (face >= 0)
            {
                const int nb = m.neighbour[slot * 6 + face];
                if (nb >= 0 && !covered(m, nb))
                {
                    shift_into(face, bs, i, j, k);
                    return clamped_face(bs, c, nb, i, j, k);
                }
            }
            const float4 rec = record_of(m, level, slot);
            face_point(rec, c, i, j, k, nx, ny, nz);
            const float* lo = m.loc.lo;
            const float* hi = m.loc.hi;
            if (nx < lo[0] || ny < lo[1] || nz < lo[2] || nx > hi[0] || ny > hi[1] || nz > hi[2]) return clamped_face(bs, c, slot, i, j, k);
            const float eps = 1e-5f * rec.w;
            const float px = fminf(hi[0] - eps, fmaxf(lo[0] + eps, nx)), py = fminf(hi[1] - eps, fmaxf(lo[1] + eps, ny)),
                        pz = fminf(hi[2] - eps, fmaxf(lo[2] + eps, nz));
            at = locate(m, px, py, pz, at_level);
            if (at < 0) return clamped_face(bs, c, slot, i, j, k);
            if (at_level != level) return -1;
            const float4 r = record_of(m, at_level, at);
            return clamped_face(bs, c, at, nearest_index(nx, r.x, r.w, c == 0 ? 0.0f : 0.5f), nearest_index(ny, r.y, r.w, c == 1 ? 0.0f : 0.5f),
                                nearest_index(nz, r.z, r.w, c == 2 ? 0.0f : 0.5f));
        }
        __device__ __noinline__ float node_value(const MacView& m, const Faces& f, int level, int64_t slot, int c, int i, int j, int k)
        {
            int at = -1, at_level = -1;
            float nx, ny, nz;
            const int64_t source = node_source(m, level, slot, c, i, j, k, at, at_level, nx, ny, nz);
            if (source >= 0) return f.c[c][source];
            return sample_extended(f, m.bs, record_of(m, at_level, at), c, at, nx, ny, nz);
        }
        // cell i0 (fraction x) moved to the last cell [-1, top] when it is past it by rounding only.  The eddy
        // viscosity's points lie one cell off a centre, on the end nodes exactly unless h rounds; feet and
        // face points lie inside the brick whose lattice they are sampled on and never come here.  The
        // difference, that rounding times a second difference, is no larger than what the
        // rounding of the point makes anyway (a point at 100 m with cells of 6 cm: 1.2e-4 of a cell).
        __device__ inline void settle(float& x, int& i0, int top)
        {
            if (i0 == -2 && x > 0.999f) { i0 = -1; x -= 1.0f; }
            else if (i0 == top + 1 && x < 0.001f) { i0 = top; x += 1.0f; }
        }
        // trilinear sample of component c at p from brick `slot`'s lattice, with the range of the
        // eight node values
        __device__ float sample_bounded(const MacView& m, const Faces& f, int level, int64_t slot, const float4& rec, int c, float px,
                                        float py, float pz, float* lower, float* upper)
        {
            const int bs = m.bs;
            float x = (px - rec.x) / rec.w - (c == 0 ? 0.0f : 0.5f);
            float y = (py - rec.y) / rec.w - (c == 1 ? 0.0f : 0.5f);
            float z = (pz - rec.z) / rec.w - (c == 2 ? 0.0f : 0.5f);
            int i0 = int(floorf(x)), j0 = int(floorf(y)), k0 = int(floorf(z));
            x -= i0;
            y -= j0;
            z -= k0;
            // a sample that rounding put a hair outside the extended lattice's end nodes extends the
            // last cell by that hair instead of reaching for one more node
            settle(x, i0, c == 0 ? bs : bs - 1);
            settle(y, j0, c == 1 ? bs : bs - 1);
            settle(z, k0, c == 2 ? bs : bs - 1);
            float v[8];
            if (in_extended(c, bs, i0, j0, k0) && in_extended(c, bs, i0 + 1, j0 + 1, k0 + 1))
            {
                const float* e = m.ext + ext_index(c, bs, slot, i0, j0, k0);
                const int nx = c == 0 ? bs + 3 : bs + 2, nxy = nx * (c == 1 ? bs + 3 : bs + 2);
#pragma unroll
                for (int q = 0; q < 8; ++q) v[q] = e[(q & 1) + (q >> 1 & 1) * nx + (q >> 2) * nxy];
            }
            else
            {
                // past the extended lattice (not reached by the characteristics of a CFL-limited step)
#pragma unroll
                for (int q = 0; q < 8; ++q) v[q] = node_value(m, f, level, slot, c, i0 + (q & 1), j0 + (q >> 1 & 1), k0 + (q >> 2));
            }
            float result = 0, mn = v[0], mx = v[0];
#pragma unroll
            for (int q = 0; q < 8; ++q)
            {
                const float wx = q & 1 ? x : 1.0f - x, wy = q & 2 ? y : 1.0f - y, wz = q & 4 ? z : 1.0f - z;
                result += wx * wy * wz * v[q];
                mn = fminf(mn, v[q]);
                mx = fmaxf(mx, v[q]);
            }
            if (lower) *lower = mn;
            if (upper) *upper = mx;
            return result;
        }
        __device__ inline float sample(const MacView& m, const Faces& f, int level, int64_t slot, const float4& rec, int c, float px,
                                       float py, float pz)
        {
            return sample_bounded(m, f, level, slot, rec, c, px, py, pz, nullptr, nullptr);
        }
        __device__ inline void clamp_point(const MacView& m, float& x, float& y, float& z)
        {
            x = fminf(m.loc.hi[0] - 1e-5f, fmaxf(m.loc.lo[0] + 1e-5f, x));
            y = fminf(m.loc.hi[1] - 1e-5f, fmaxf(m.loc.lo[1] + 1e-5f, y));
            z = fminf(m.loc.hi[2] - 1e-5f, fmaxf(m.loc.lo[2] + 1e-5f, z));
        }
        // locate() for points near brick `home` (non-covered, level `level`): no finer brick lies in
        // a non-covered one and the level widths are exact halves, so a point whose brick coordinates
        // are the home brick's is in it and needs no search from the finest level down.
        struct Home
        {
            int64_t slot;
            int level;
            float width, bx, by, bz;    // brick width, brick coordinates as locate() rounds them
        };
        __device__ inline Home home_of(const MacView& m, int level, int64_t slot, const float4& rec)
        {
            Home h{slot, level, float(m.bs) * m.loc.levels[level].h, 0.0f, 0.0f, 0.0f};
            const float half = 0.5f * h.width;
            h.bx = floorf((rec.x + half - m.loc.lo[0]) / h.width);
            h.by = floorf((rec.y + half - m.loc.lo[1]) / h.width);
            h.bz = floorf((rec.z + half - m.loc.lo[2]) / h.width);
            return h;
        }
        __device__ inline int locate_near(const MacView& m, const Home& h, float x, float y, float z, int& level)
        {
            const bool inside = x >= m.loc.lo[0] && y >= m.loc.lo[1] && z >= m.loc.lo[2] && x < m.loc.hi[0] && y < m.loc.hi[1] && z < m.loc.hi[2];
            if (inside && floorf((x - m.loc.lo[0]) / h.width) == h.bx && floorf((y - m.loc.lo[1]) / h.width) == h.by &&
                floorf((z - m.loc.lo[2]) / h.width) == h.bz)
            {
                level = h.level;
                return int(h.slot);
            }
            return locate(m, x, y, z, level);
        }
        // two-stage characteristic from p over dt (negative dt traces forward); u: the velocity at p
        __device__ void trace(const MacView& m, const Faces& f, const Home& home, const float u[3], float& x, float& y, float& z, float dt)
        {
            float mx = x - float(0.5f * dt * u[0]), my = y - float(0.5f * dt * u[1]), mz = z - float(0.5f * dt * u[2]);
            clamp_point(m, mx, my, mz);
            int level;
            const int at = locate_near(m, home, mx, my, mz, level);
            float v[3] = {u[0], u[1], u[2]};
            if (at >= 0)
            {
                const float4 rec = record_of(m, level, at);
#pragma unroll
                for (int c = 0; c < 3; ++c) v[c] = sample(m, f, level, at, rec, c, mx, my, mz);
            }
            x = x - float(dt * v[0]);
            y = y - float(dt * v[1]);
            z = z - float(dt * v[2]);
            clamp_point(m, x, y, z);
        }
        __device__ inline void decode(int64_t q, int bs, int& c, int64_t& slot, int& i, int& j, int& k)
        {
            const int per = bs * bs * (bs + 1);
            int local = int(q % per);
            const int64_t r = q / per;
            c = int(r % 3);
            slot = r / 3;
            i = j = k = 0;
            if (c == 0) { i = local % (bs + 1); local /= bs + 1; j = local % bs; k = local / bs; }
            else if (c == 1) { i = local % bs; local /= bs; j = local % (bs + 1); k = local / (bs + 1); }
            else { i = local % bs; local /= bs; j = local % bs; k = local / bs; }
        }
        __device__ inline float minmod(float a, float b) { return a * b <= 0.0f ? 0.0f : (fabsf(a) < fabsf(b) ? a : b); }
        // one step along `axis` from face node (i,j,k) of brick `slot` inside the same level
        __device__ bool step_same_level(const MacView& m, int c, int axis, int direction, int64_t& slot, int& i, int& j, int& k)
        {
            const int bs = m.bs;
            if (axis == 0) i += direction; else if (axis == 1) j += direction; else k += direction;
            if (valid_face(c, bs, i, j, k)) return true;
            const int face = outside_face(c == 0 ? bs + 1 : bs, c == 1 ? bs + 1 : bs, c == 2 ? bs + 1 : bs, i, j, k);
            if (face < 0) return false;
            const int nb = m.neighbour[slot * 6 + face];
            if (nb < 0 || covered(m, nb)) return false;
            shift_into(face, bs, i, j, k);
            slot = nb;
            return valid_face(c, bs, i, j, k);
        }
        // limited MUSCL update of a near-fabric face along its open same-side links
        __device__ float band_update(const MacView& m, const Faces& f, const uint8_t* const* links, int level, int64_t slot,
                                     const float4& rec, int c, int i, int j, int k, float current, uint8_t link, float dt)
        {
            const int bs = m.bs;
            float px, py, pz;
            face_point(rec, c, i, j, k, px, py, pz);
            const float velocity[3] = {sample(m, f, level, slot, rec, 0, px, py, pz), sample(m, f, level, slot, rec, 1, px, py, pz),
                                       sample(m, f, level, slot, rec, 2, px, py, pz)};
            float weighted = 0, weights = 0, lower = current, upper = current;
            for (int axis = 0; axis < 3; ++axis)
            {
                const int up_dir = velocity[axis] >= 0.0f ? -1 : 1, up_bit = 2 * axis + (up_dir > 0), down_bit = 2 * axis + (up_dir < 0);
                if (!(link & (1u << up_bit))) continue;
                int64_t us = slot;
                int ui = i, uj = j, uk = k;
                if (!step_same_level(m, c, axis, up_dir, us, ui, uj, uk)) continue;
                const float upstream = clamped(f, bs, c, us, ui, uj, uk);
                lower = fminf(lower, upstream);
                upper = fmaxf(upper, upstream);
                const float weight = dt * fabsf(velocity[axis]) / rec.w;
                float delta = weight * (upstream - current);
                // the limited linear reconstruction needs all three further segments on same-side
                // links; otherwise the first-order donor update stays
                const uint8_t up_links = links[c][axis_face(bs, c, us, ui, uj, uk)];
                int64_t u2s = us, ds = slot;
                int u2i = ui, u2j = uj, u2k = uk, di = i, dj = j, dk = k;
                const bool second = (link & (1u << down_bit)) && (up_links & (1u << up_bit)) &&
                                    step_same_level(m, c, axis, up_dir, u2s, u2i, u2j, u2k) &&
                                    step_same_level(m, c, axis, -up_dir, ds, di, dj, dk);
                if (second)
                {
                    const float upstream2 = clamped(f, bs, c, u2s, u2i, u2j, u2k), downstream = clamped(f, bs, c, ds, di, dj, dk);
                    lower = fminf(lower, downstream);
                    upper = fmaxf(upper, downstream);
                    const float up_slope = minmod(upstream - upstream2, current - upstream),
                                slope = minmod(current - upstream, downstream - current);
                    const float incoming = upstream + 0.5f * up_slope, outgoing = current + 0.5f * slope;
                    delta = -weight * (outgoing - incoming);
                }
                weighted += delta;
                weights += weight;
            }
            const float scale = weights > 1.0f ? 1.0f / weights : 1.0f;
            return fmaxf(lower, fminf(upper, current + scale * weighted));
        }

        struct Links
        {
            const uint8_t* c[3];
        };
        struct Out
        {
            float* c[3];
        };

        // Source of every node of every extended lattice: the index of a face of the component, -1 for
        // the nodes interpolated on another level (they are counted, and listed when `slow` is
        // given), -2 in covered bricks (never sampled).
        __global__ void mac_source_kernel(MacView m, int64_t total, int* source, int64_t* slow, int* count)
        {
            const int64_t q = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
            if (q >= total) return;
            const int bs = m.bs, per = ext_size(bs);
            const int64_t slot = q / (3 * per);
            const int c = int(q / per % 3);
            int local = int(q % per);
            const int nx = c == 0 ? bs + 3 : bs + 2, ny = c == 1 ? bs + 3 : bs + 2;
            const int i = local % nx - 1;
            local /= nx;
            const int j = local % ny - 1, k = local / ny - 1;
            if (covered(m, slot)) { source[q] = -2; return; }
            int at = -1, at_level = -1;
            float x, y, z;
            const int64_t from = node_source(m, m.slot_level[slot], slot, c, i, j, k, at, at_level, x, y, z);
            source[q] = int(from);
            if (from < 0)
            {
                const int n = atomicAdd(count, 1);
                if (slow) slow[n] = q;
            }
        }
        // Extended lattices of a field: copies, then the listed nodes interpolated on another level.
        // The copy moves 12 B per node (source, value, store; 3 x 1100 nodes per 8^3 brick) in rows of 8 to 10
        // values, bound by L1 and L2 sectors (64 and 49 %): 47 us for 8.2 M nodes.  The interpolation's
        // 64 clamped reads per node (77 us for 0.56 M) run in a launch of their own, so no copying warp
        // waits for them.
        __global__ void mac_extend_kernel(Faces f, int per, int64_t total, const int* __restrict__ source, float* __restrict__ ext)
        {
            const int64_t q = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
            if (q >= total) return;
            const int from = source[q];
            if (from >= 0) ext[q] = f.c[int(q / per % 3)][from];
        }
        __global__ void mac_extend_slow_kernel(MacView m, Faces f, int count, const int64_t* __restrict__ slow, float* __restrict__ ext)
        {
            const int n = blockIdx.x * blockDim.x + threadIdx.x;
            if (n >= count) return;
            const int64_t q = slow[n];
            const int bs = m.bs, per = ext_size(bs);
            const int64_t slot = q / (3 * per);
            const int c = int(q / per % 3);
            int local = int(q % per);
            const int nx = c == 0 ? bs + 3 : bs + 2, ny = c == 1 ? bs + 3 : bs + 2;
            const int i = local % nx - 1;
            local /= nx;
            ext[q] = node_value(m, f, m.slot_level[slot], slot, c, i, local % ny - 1, local / ny - 1);
        }

        // What the correction of a face needs from the forward pass: the forward foot, the range of the
        // backward foot's samples and the brick that owns the forward foot (-1: no correction).
        struct Feet
        {
            float4* foot;               // [3 faces] x, y, z, minimum
            float2* range;              // [3 faces] maximum, brick slot (bits)
        };

        // Forward pass, and both characteristics of the correction: they need the same field and start
        // from the same velocity, so each face is traced back and forth once.  Bound by the latency of ten
        // trilinear samples and four locations per face at two CTAs an SM (110 registers; 44 % of the SM's
        // throughput, 23 % of L1's, 22 % of its warps): 0.57 ms for the 4.3 M faces of a 1.3 M-cell grid on
        // three levels.  With the samples on the extended lattices and the
        // traces shared, a whole advection takes 1.0 instead of 19.8 ms there (correction 0.14,
        // extensions 0.2 ms).
        __global__ void __launch_bounds__(256) mac_forward_kernel(MacView m, Faces f, Links links, int64_t total, float dt, Out out, Feet feet)
        {
            const int64_t q = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
            if (q >= total) return;
            int c, i, j, k;
            int64_t slot;
            decode(q, m.bs, c, slot, i, j, k);
            if (covered(m, slot)) return;
            const int level = m.slot_level[slot];
            const float4 rec = record_of(m, level, slot);
            const int64_t at = axis_face(m.bs, c, slot, i, j, k);
            const float current = f.c[c][at];
            const uint8_t link = links.c[c][at];
            float4 foot = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
            float2 range = make_float2(0.0f, __int_as_float(-1));
            float result;
            if (link & 0x40) result = band_update(m, f, links.c, level, slot, rec, c, i, j, k, current, link, dt);
            else
            {
                float px, py, pz;
                face_point(rec, c, i, j, k, px, py, pz);
                const Home home = home_of(m, level, slot, rec);
                float u[3];
#pragma unroll
                for (int a = 0; a < 3; ++a) u[a] = sample(m, f, level, slot, rec, a, px, py, pz);
                float bx = px, by = py, bz = pz, fx = px, fy = py, fz = pz;
                trace(m, f, home, u, bx, by, bz, dt);
                trace(m, f, home, u, fx, fy, fz, -dt);
                int back_level = -1, forward_level = -1, owner_level = -1;
                const int back = locate_near(m, home, bx, by, bz, back_level);
                float mn = current, mx = current;
                result = current;
                if (back >= 0) result = sample_bounded(m, f, back_level, back, record_of(m, back_level, back), c, bx, by, bz, &mn, &mx);
                // the reverse correction only when the node and both feet are on this level: across a
                // 2:1 transition the forward field mixes independently evolved lattices
                clamp_point(m, px, py, pz);
                locate_near(m, home, px, py, pz, owner_level);
                const int ahead = locate_near(m, home, fx, fy, fz, forward_level);
                foot = make_float4(fx, fy, fz, mn);
                range = make_float2(mx, __int_as_float(owner_level == level && back_level == level && forward_level == level ? ahead : -1));
            }
            out.c[c][at] = result;
            const int64_t n = (at + c * (total / 3));
            feet.foot[n] = foot;
            feet.range[n] = range;
        }

        // MacCormack correction, written over the current field (each face is read by its own thread
        // only); m.ext holds the forward field's lattices.  Covered bricks' faces become 0.
        __global__ void __launch_bounds__(256) mac_correct_kernel(MacView m, Faces forward, int64_t total, Feet feet, Out current)
        {
            const int64_t q = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
            if (q >= total) return;
            int c, i, j, k;
            int64_t slot;
            decode(q, m.bs, c, slot, i, j, k);
            const int64_t at = axis_face(m.bs, c, slot, i, j, k);
            if (covered(m, slot)) { current.c[c][at] = 0.0f; return; }
            const int64_t n = at + c * (total / 3);
            const float2 range = feet.range[n];
            const float phf = forward.c[c][at];
            const int ahead = __float_as_int(range.y);
            float result = phf;
            if (ahead >= 0)
            {
                const int level = m.slot_level[slot];
                const float4 foot = feet.foot[n];
                const float phn = sample(m, forward, level, ahead, record_of(m, level, ahead), c, foot.x, foot.y, foot.z);
                result = fmaxf(foot.w, fminf(range.x, phf + 0.5f * (current.c[c][at] - phn)));
            }
            current.c[c][at] = result;
        }

        // ---- LES and diffusion ----
        __device__ inline float cell_clamped(const float* nut, int bs, int64_t slot, int i, int j, int k)
        {
            i = max(0, min(bs - 1, i));
            j = max(0, min(bs - 1, j));
            k = max(0, min(bs - 1, k));
            return nut[slot * bs * bs * bs + (int64_t(k) * bs + j) * bs + i];
        }
        __device__ float cell_extended(const float* nut, int bs, int64_t slot, int i, int j, int k)
        {
            const int want[3] = {i, j, k};
            int at[3][2], count[3];
            float w[3][2];
            for (int a = 0; a < 3; ++a)
            {
                if (want[a] < 0) { at[a][0] = 0; at[a][1] = 1; w[a][0] = 2.0f; w[a][1] = -1.0f; count[a] = 2; }
                else if (want[a] >= bs) { at[a][0] = bs - 1; at[a][1] = bs - 2; w[a][0] = 2.0f; w[a][1] = -1.0f; count[a] = 2; }
                else { at[a][0] = want[a]; w[a][0] = 1.0f; count[a] = 1; }
            }
            float result = 0;
            for (int az = 0; az < count[2]; ++az)
                for (int ay = 0; ay < count[1]; ++ay)
                    for (int ax = 0; ax < count[0]; ++ax)
                        result += w[0][ax] * w[1][ay] * w[2][az] * cell_clamped(nut, bs, slot, at[0][ax], at[1][ay], at[2][az]);
            return result;
        }
        __device__ float cell_sample_extended(const float* nut, int bs, const float4& rec, int64_t slot, float px, float py, float pz)
        {
            float x = (px - rec.x) / rec.w - 0.5f, y = (py - rec.y) / rec.w - 0.5f, z = (pz - rec.z) / rec.w - 0.5f;
            const int i0 = int(floorf(x)), j0 = int(floorf(y)), k0 = int(floorf(z));
            x -= i0;
            y -= j0;
            z -= k0;
            float result = 0;
            for (int dz = 0; dz < 2; ++dz)
                for (int dy = 0; dy < 2; ++dy)
                    for (int dx = 0; dx < 2; ++dx)
                    {
                        const float wx = dx ? x : 1.0f - x, wy = dy ? y : 1.0f - y, wz = dz ? z : 1.0f - z;
                        result += wx * wy * wz * cell_extended(nut, bs, slot, i0 + dx, j0 + dy, k0 + dz);
                    }
            return result;
        }
        // cell value (i,j,k) of brick `slot`, which may lie outside the brick
        __device__ __noinline__ float cell_node_value(const MacView& m, const float* nut, int level, int64_t slot, int i, int j, int k)
        {
            const int bs = m.bs;
            if (i >= 0 && j >= 0 && k >= 0 && i < bs && j < bs && k < bs) return cell_clamped(nut, bs, slot, i, j, k);
            const int face = outside_face(bs, bs, bs, i, j, k);
            if (face >= 0)
            {
                const int nb = m.neighbour[slot * 6 + face];
                if (nb >= 0 && !covered(m, nb))
                {
                    shift_into(face, bs, i, j, k);
                    return cell_clamped(nut, bs, nb, i, j, k);
                }
            }
            const float4 rec = record_of(m, level, slot);
            const float nx = rec.x + (i + 0.5f) * rec.w, ny = rec.y + (j + 0.5f) * rec.w, nz = rec.z + (k + 0.5f) * rec.w;
            const float* lo = m.loc.lo;
            const float* hi = m.loc.hi;
            if (nx < lo[0] || ny < lo[1] || nz < lo[2] || nx >= hi[0] || ny >= hi[1] || nz >= hi[2]) return cell_clamped(nut, bs, slot, i, j, k);
            int at_level;
            const int at = locate(m, nx, ny, nz, at_level);
            if (at < 0) return cell_clamped(nut, bs, slot, i, j, k);
            const float4 r = record_of(m, at_level, at);
            if (at_level != level) return cell_sample_extended(nut, bs, r, at, nx, ny, nz);
            return cell_clamped(nut, bs, at, nearest_index(nx, r.x, r.w, 0.5f), nearest_index(ny, r.y, r.w, 0.5f),
                                nearest_index(nz, r.z, r.w, 0.5f));
        }

        __global__ void mac_smagorinsky_kernel(MacView m, Faces f, int64_t cells, float cs, float* nut)
        {
            const int64_t q = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
            if (q >= cells) return;
            const int bs = m.bs, c3 = bs * bs * bs;
            const int64_t slot = q / c3;
            const int local = int(q % c3);
            if (covered(m, slot)) return;
            const int i = local % bs, j = (local / bs) % bs, k = local / (bs * bs);
            const int level = m.slot_level[slot];
            const float4 rec = record_of(m, level, slot);
            const float h = rec.w;
            const float cx = rec.x + (i + 0.5f) * h, cy = rec.y + (j + 0.5f) * h, cz = rec.z + (k + 0.5f) * h;
            float g[3][3];
            for (int c = 0; c < 3; ++c)
                for (int axis = 0; axis < 3; ++axis)
                {
                    float lx = cx, ly = cy, lz = cz, ux = cx, uy = cy, uz = cz;
                    if (axis == 0) { lx -= h; ux += h; } else if (axis == 1) { ly -= h; uy += h; } else { lz -= h; uz += h; }
                    g[c][axis] = (sample(m, f, level, slot, rec, c, ux, uy, uz) - sample(m, f, level, slot, rec, c, lx, ly, lz)) / (2.0f * h);
                }
            const float sxx = g[0][0], syy = g[1][1], szz = g[2][2], sxy = 0.5f * (g[0][1] + g[1][0]), sxz = 0.5f * (g[0][2] + g[2][0]),
                        syz = 0.5f * (g[1][2] + g[2][1]);
            const float magnitude = sqrtf(2.0f * (sxx * sxx + syy * syy + szz * szz + 2.0f * (sxy * sxy + sxz * sxz + syz * syz)));
            const float length = cs * h;
            nut[q] = length * length * magnitude;
        }

        // Written over the field: neighbours are read from the extended lattices, the face itself by
        // its own thread only.  Covered bricks' faces become 0.
        __global__ void __launch_bounds__(256) mac_diffuse_kernel(MacView m, Links links, const float* nut, int64_t total, float nu, float dt, Out out)
        {
            const int64_t q = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
            if (q >= total) return;
            int c, i, j, k;
            int64_t slot;
            decode(q, m.bs, c, slot, i, j, k);
            const int bs = m.bs;
            const int64_t at = axis_face(bs, c, slot, i, j, k);
            if (covered(m, slot)) { out.c[c][at] = 0.0f; return; }
            const int level = m.slot_level[slot];
            const float current = out.c[c][at];
            const uint8_t link = links.c[c][at];
            auto face_value = [&](int a, int b, int d) { return m.ext[ext_index(c, bs, slot, a, b, d)]; };
            float laplacian = 0, viscosity = nu;
            if (!(link & 0x40))
            {
                laplacian = face_value(i - 1, j, k) + face_value(i + 1, j, k) + face_value(i, j - 1, k) + face_value(i, j + 1, k) +
                            face_value(i, j, k - 1) + face_value(i, j, k + 1) - 6.0f * current;
                int ci = i, cj = j, ck = k;
                if (c == 0) --ci; else if (c == 1) --cj; else --ck;
                const int ci2 = ci + (c == 0), cj2 = cj + (c == 1), ck2 = ck + (c == 2);
                auto cell_value = [&](int a, int b, int d) {
                    return a >= 0 && b >= 0 && d >= 0 && a < bs && b < bs && d < bs ? cell_clamped(nut, bs, slot, a, b, d)
                                                                                    : cell_node_value(m, nut, level, slot, a, b, d);
                };
                viscosity += 0.5f * (cell_value(ci, cj, ck) + cell_value(ci2, cj2, ck2));
            }
            else
                for (int axis = 0; axis < 3; ++axis)
                    for (int direction = -1; direction <= 1; direction += 2)
                    {
                        const int bit = 2 * axis + (direction > 0);
                        if (!(link & (1u << bit))) continue;
                        int p[3] = {i, j, k};
                        p[axis] += direction;
                        laplacian += face_value(p[0], p[1], p[2]) - current;
                    }
            const float h = m.loc.levels[level].h;
            out.c[c][at] = current + dt * viscosity * laplacian / (h * h);
        }
    }

    namespace
    {
        // max |face velocity| over the faces of non-covered bricks (DeviceAmrFields::
        // max_abs_velocity, amr_fields.cu:65-68, 195-198), as float bits in an unsigned int
        __global__ void mac_max_face_kernel(Faces f, const uint32_t* flags, int64_t per_slot, int64_t per_component, unsigned int* out)
        {
            __shared__ float shared[8];
            float m = 0.0f;
            for (int64_t q = int64_t(blockIdx.x) * blockDim.x + threadIdx.x; q < 3 * per_component; q += int64_t(gridDim.x) * blockDim.x)
            {
                const int c = int(q / per_component);
                const int64_t i = q % per_component;
                if (!(flags[i / per_slot] & PCFD_BRICK_COVERED)) m = fmaxf(m, fabsf(f.c[c][i]));
            }
            for (int o = 16; o > 0; o >>= 1) m = fmaxf(m, __shfl_down_sync(0xffffffffu, m, o));
            if ((threadIdx.x & 31) == 0) shared[threadIdx.x >> 5] = m;
            __syncthreads();
            if (threadIdx.x == 0)
            {
                for (int w = 1; w < int(blockDim.x >> 5); ++w) m = fmaxf(m, shared[w]);
                atomicMax(out, __float_as_uint(m));
            }
        }
    }

    inline float uint_bits_to_float(unsigned int bits)
    {
        float f;
        std::memcpy(&f, &bits, sizeof(f));
        return f;
    }

    // ---- system state and launches ----
    struct MacState
    {
        DBuf<int> neighbour;
        DBuf<uint32_t> flags;
        DBuf<uint8_t> links[3];
        DBuf<float> forward[3], nut;
        DBuf<int> ext_source;                   // extended-lattice nodes: source faces
        DBuf<int64_t> ext_slow;                 // the nodes interpolated on another level
        int slow_count = 0;
        DBuf<float> ext;                        // [B][3][ext_size] extended lattices of the field last extended
        DBuf<float4> foot;                      // [3 faces] forward pass -> correction (Feet)
        DBuf<float2> range;
        DBuf<unsigned int> maximum;
        bool extended = false;                  // ext_source, ext_slow and the buffers above are complete
        bool has_links = false;
    };

    namespace
    {
        MacState& mac_state(System& s)
        {
            require(s.mac != nullptr, "MAC momentum not set up");
            return *static_cast<MacState*>(s.mac);
        }
        MacView mac_view(System& s)
        {
            MacState& st = mac_state(s);
            return MacView{locator_view(s), st.neighbour.p, st.flags.p, s.brick_level, s.bs, st.ext.p};
        }
        int64_t ext_total(const System& s) { return int64_t(s.B) * 3 * ext_size(s.bs); }
        // the lattice nodes' sources (grid only) and the buffers of the extended field
        void build_extension(System& s)
        {
            MacState& st = mac_state(s);
            const int64_t total = ext_total(s);
            require(s.faces < (int64_t(1) << 31), "MAC momentum: grid too large");   // a source is an int (1.9 billion cells)
            st.ext_source.alloc(size_t(total), false);
            st.ext.alloc(size_t(total));
            DBuf<int> count;
            count.alloc(1);
            const MacView m = mac_view(s);
            int64_t* list = nullptr;
            for (int pass = 0; pass < 2; ++pass)
            {
                cuda_check(cudaMemsetAsync(count.p, 0, sizeof(int), s.stream), "clear node count");
                mac_source_kernel<<<blocks_for(total), kThreads, 0, launch_stream(s)>>>(m, total, st.ext_source, list, count);
                cuda_check(cudaMemcpyAsync(&st.slow_count, count.p, sizeof(int), cudaMemcpyDeviceToHost, s.stream), "node count");
                cuda_check(cudaStreamSynchronize(s.stream), "extended lattice nodes");
                if (!st.slow_count) break;
                if (!list) st.ext_slow.alloc(size_t(st.slow_count), false);
                list = st.ext_slow.p;
            }
            st.extended = true;
        }
        void extend(System& s, const Faces& f)
        {
            MacState& st = mac_state(s);
            const int64_t total = ext_total(s);
            mac_extend_kernel<<<blocks_for(total), kThreads, 0, launch_stream(s)>>>(f, ext_size(s.bs), total, st.ext_source, st.ext);
            if (st.slow_count)
                mac_extend_slow_kernel<<<blocks_for(st.slow_count, 64), 64, 0, launch_stream(s)>>>(mac_view(s), f, st.slow_count, st.ext_slow,
                                                                                                  st.ext);
        }
    }

    void build_mac(System& s, const pcfd_topology& t)
    {
        auto* st = new MacState();
        s.mac = st;
        std::vector<int> neighbour(size_t(s.B) * 6, -1);
        std::vector<uint32_t> flags(size_t(s.B), 0);
        for (int l = 0, slot0 = 0; l < t.level_count; ++l)
        {
            const pcfd_level& lev = t.levels[l];
            for (int b = 0; b < lev.brick_count; ++b)
            {
                flags[size_t(slot0 + b)] = lev.flags[b];
                for (int face = 0; face < 6; ++face)
                {
                    const int n = lev.neighbors[b * 6 + face];
                    neighbour[size_t(slot0 + b) * 6 + face] = n >= 0 ? slot0 + n : -1;
                }
            }
            slot0 += lev.brick_count;
        }
        st->neighbour.upload(neighbour);
        st->flags.upload(flags);
        st->maximum.alloc(1);
    }

    void destroy_mac(System& s)
    {
        delete static_cast<MacState*>(s.mac);
        s.mac = nullptr;
    }

    void mac_set_links(System& s, const uint8_t* const host[3])
    {
        MacState& st = mac_state(s);
        st.has_links = false;                   // until everything below is there
        for (int c = 0; c < 3; ++c)
        {
            st.links[c].upload(std::vector<uint8_t>(host[c], host[c] + s.faces));
            if (!st.forward[c].n) st.forward[c].alloc(size_t(s.faces));
        }
        if (!st.nut.n) st.nut.alloc(size_t(s.S));
        if (!st.extended)
        {
            st.foot.alloc(size_t(s.faces) * 3, false);
            st.range.alloc(size_t(s.faces) * 3, false);
            build_extension(s);
        }
        st.has_links = true;
    }

    void mac_advect(System& s, float dt)
    {
        MacState& st = mac_state(s);
        require(st.has_links, "MAC advection: links not set");
        const MacView m = mac_view(s);
        const Faces f{{s.u.p, s.v.p, s.w.p}};
        const Links links{{st.links[0].p, st.links[1].p, st.links[2].p}};
        const int64_t total = int64_t(s.B) * 3 * s.bs * s.bs * (s.bs + 1);
        const Out forward{{st.forward[0].p, st.forward[1].p, st.forward[2].p}};
        const Feet feet{st.foot.p, st.range.p};
        extend(s, f);
        mac_forward_kernel<<<blocks_for(total), kThreads, 0, launch_stream(s)>>>(m, f, links, total, dt, forward, feet);
        const Faces fw{{st.forward[0].p, st.forward[1].p, st.forward[2].p}};
        extend(s, fw);
        const Out out{{s.u.p, s.v.p, s.w.p}};
        mac_correct_kernel<<<blocks_for(total), kThreads, 0, launch_stream(s)>>>(m, fw, total, feet, out);
        cuda_check(cudaGetLastError(), "MAC advection");
    }

    void mac_diffuse_smagorinsky(System& s, float nu, float cs, float dt)
    {
        MacState& st = mac_state(s);
        require(st.has_links, "MAC diffusion: links not set");
        const MacView m = mac_view(s);
        const Faces f{{s.u.p, s.v.p, s.w.p}};
        const Links links{{st.links[0].p, st.links[1].p, st.links[2].p}};
        const int64_t cells = int64_t(s.B) * s.bs * s.bs * s.bs;
        extend(s, f);
        mac_smagorinsky_kernel<<<blocks_for(cells), kThreads, 0, launch_stream(s)>>>(m, f, cells, cs, st.nut.p);
        const int64_t total = int64_t(s.B) * 3 * s.bs * s.bs * (s.bs + 1);
        const Out out{{s.u.p, s.v.p, s.w.p}};
        mac_diffuse_kernel<<<blocks_for(total), kThreads, 0, launch_stream(s)>>>(m, links, st.nut.p, total, nu, dt, out);
        cuda_check(cudaGetLastError(), "MAC diffusion");
    }

    void mac_eddy_viscosity(System& s, float* host_nut)
    {
        MacState& st = mac_state(s);
        require(st.nut.n == size_t(s.S), "MAC eddy viscosity: no diffusion step yet");
        cuda_check(cudaStreamSynchronize(s.stream), "synchronize");
        cuda_check(cudaMemcpy(host_nut, st.nut.p, size_t(s.S) * sizeof(float), cudaMemcpyDeviceToHost), "download eddy viscosity");
    }

    bool mac_ready(const System& s) { return s.mac && static_cast<const MacState*>(s.mac)->has_links; }

    float mac_max_face_speed(System& s)
    {
        MacState& st = mac_state(s);
        const Faces f{{s.u.p, s.v.p, s.w.p}};
        const int64_t per_slot = int64_t(s.bs + 1) * s.bs * s.bs, per_component = int64_t(s.B) * per_slot;
        cuda_check(cudaMemsetAsync(st.maximum.p, 0, sizeof(unsigned int), s.stream), "clear maximum");
        mac_max_face_kernel<<<int(std::min<int64_t>(592, (3 * per_component + kThreads - 1) / kThreads)), kThreads, 0, launch_stream(s)>>>(
            f, st.flags, per_slot, per_component, st.maximum);
        unsigned int bits = 0;
        cuda_check(cudaMemcpyAsync(&bits, st.maximum.p, sizeof(bits), cudaMemcpyDeviceToHost, s.stream), "read maximum");
        cuda_check(cudaStreamSynchronize(s.stream), "face maximum");
        return uint_bits_to_float(bits);
    }
}
