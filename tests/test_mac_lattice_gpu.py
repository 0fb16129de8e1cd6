"""MacCormack advection, band faces, eddy viscosity and diffusion of the staggered faces against a
plain per-face restatement.

mac_advect samples every field on per-brick lattices with one ghost node and shares the two
characteristics between its passes.  The restatement below evaluates randomly chosen faces one by
one from the definition (two-stage characteristics, trilinear samples on the brick that owns the
point, nodes outside a brick from the neighbour, the owning brick or the one-sided extension of
another level's brick), with no ghost storage.  Decisions (which brick, which lattice node) are
taken in FP32 as the kernels take them; the sums in FP64.  Tolerance: a trilinear FP32 sum of
eight values of size U errs by at most ~16 ulp(U), and a foot off by that much times dt moves the
sampled value by less, so 4e-6 U per sample and 1e-5 U over the two passes.
"""
import numpy as np
import pytest

from paracfd_b200 import BuiltTopology, CompositeSystem
from paracfd_b200.geometry import extruded_wing, naca4_section, rotate_section

pytestmark = pytest.mark.gpu

F = np.float32
U = 10.0


def build(levels, brick_size, base=0.125):
    vertices, triangles = extruded_wing(rotate_section(naca4_section(12, 48, 1.0), 4.0), -0.6, 0.6)
    return BuiltTopology(vertices, triangles, (-1.0, -1.0, -1.0), (2.0, 1.0, 1.0), base, levels, brick_size,
                         wing_refinement_distance=0.3, surface_refinement_distance=0.1, wake_length=0.5, wake_radius=0.3)


class Lattice:
    """The grid's bricks and the node / sample / trace definitions on face arrays [3][slot, k, j, i]."""

    def __init__(self, t, bs):
        self.bs, self.level, self.rec, self.nb, self.cov, self.at = bs, [], [], [], [], {}
        self.h, slot0 = [], 0
        for l in range(t.level_count):
            lev = t.levels[l]
            n = lev.brick_count
            flags = np.ctypeslib.as_array(lev.flags, shape=(n,))
            origin = np.ctypeslib.as_array(lev.origin, shape=(3 * n,)).reshape(n, 3)
            coord = np.ctypeslib.as_array(lev.coord, shape=(3 * n,)).reshape(n, 3)
            nb = np.ctypeslib.as_array(lev.neighbors, shape=(6 * n,)).reshape(n, 6)
            self.h.append(F(lev.h))
            for b in range(n):
                self.level.append(l)
                self.rec.append((F(origin[b, 0]), F(origin[b, 1]), F(origin[b, 2])))
                self.nb.append([slot0 + x if x >= 0 else -1 for x in nb[b]])
                self.cov.append(bool(flags[b] & 128))
                self.at[(l,) + tuple(int(x) for x in coord[b])] = slot0 + b
            slot0 += n
        self.lo, self.hi = [F(x) for x in t.domain_lo], [F(x) for x in t.domain_hi]

    def size(self, c):
        return [self.bs + (a == c) for a in range(3)]

    def locate(self, p):
        if any(p[a] < self.lo[a] or p[a] >= self.hi[a] for a in range(3)):
            return -1
        for l in range(len(self.h) - 1, -1, -1):
            width = F(self.bs) * self.h[l]
            s = self.at.get((l,) + tuple(int(np.floor((p[a] - self.lo[a]) / width)) for a in range(3)), -1)
            if s >= 0 and not self.cov[s]:
                return s
        return -1

    def point(self, c, s, ijk):
        h = self.h[self.level[s]]
        return [F(self.rec[s][a] + F(ijk[a] + (0.0 if a == c else 0.5)) * h) for a in range(3)]

    def clamped(self, f, c, s, ijk):
        n = self.size(c)
        i, j, k = (min(max(ijk[a], 0), n[a] - 1) for a in range(3))
        return float(f[c][s, k, j, i])

    def extended(self, f, c, s, ijk):
        n, terms = self.size(c), [((), 1.0)]
        for a in range(3):
            if ijk[a] < 0:
                ends = ((0, 2.0), (1, -1.0))
            elif ijk[a] >= n[a]:
                ends = ((n[a] - 1, 2.0), (n[a] - 2, -1.0))
            else:
                ends = ((ijk[a], 1.0),)
            terms = [(q + (e,), w * v) for q, w in terms for e, v in ends]
        return sum(w * self.clamped(f, c, s, q) for q, w in terms)

    def corners(self, c, s, p):
        h = self.h[self.level[s]]
        x = [F((p[a] - self.rec[s][a]) / h - F(0.0 if a == c else 0.5)) for a in range(3)]
        i0 = [int(np.floor(v)) for v in x]
        for d in np.ndindex(2, 2, 2):
            w = 1.0
            for a in range(3):
                fraction = float(x[a]) - i0[a]
                w *= fraction if d[a] else 1.0 - fraction
            yield [i0[a] + d[a] for a in range(3)], w

    def node(self, f, c, s, ijk):
        n = self.size(c)
        out = [a for a in range(3) if ijk[a] < 0 or ijk[a] >= n[a]]
        if not out:
            return self.clamped(f, c, s, ijk)
        if len(out) == 1:
            a = out[0]
            nb = self.nb[s][2 * a + (ijk[a] >= n[a])]
            if nb >= 0 and not self.cov[nb]:
                q = list(ijk)
                q[a] += self.bs if ijk[a] < 0 else -self.bs
                return self.clamped(f, c, nb, q)
        p = self.point(c, s, ijk)
        if any(p[a] < self.lo[a] or p[a] > self.hi[a] for a in range(3)):
            return self.clamped(f, c, s, ijk)
        eps = F(1e-5) * self.h[self.level[s]]
        at = self.locate([min(self.hi[a] - eps, max(self.lo[a] + eps, p[a])) for a in range(3)])
        if at < 0:
            return self.clamped(f, c, s, ijk)
        if self.level[at] != self.level[s]:
            return sum(w * self.extended(f, c, at, q) for q, w in self.corners(c, at, p))
        h = self.h[self.level[at]]
        return self.clamped(f, c, at, [int(np.floor((p[a] - self.rec[at][a]) / h - F(0.0 if a == c else 0.5) + F(0.5))) for a in range(3)])

    def sample(self, f, c, s, p):
        values = [(self.node(f, c, s, q), w) for q, w in self.corners(c, s, p)]
        return sum(v * w for v, w in values), min(v for v, _ in values), max(v for v, _ in values)

    def clamp(self, p):
        return [min(self.hi[a] - F(1e-5), max(self.lo[a] + F(1e-5), F(p[a]))) for a in range(3)]

    def trace(self, f, s, p, dt):
        u = [self.sample(f, a, s, p)[0] for a in range(3)]
        mid = self.clamp([p[a] - F(0.5 * dt * u[a]) for a in range(3)])
        at = self.locate(mid)
        v = [self.sample(f, a, at, mid)[0] if at >= 0 else u[a] for a in range(3)]
        return self.clamp([p[a] - F(dt * v[a]) for a in range(3)])

    def forward(self, f, c, s, ijk, dt):
        foot = self.trace(f, s, self.point(c, s, ijk), dt)
        at = self.locate(foot)
        current = self.clamped(f, c, s, ijk)
        return (self.sample(f, c, at, foot) if at >= 0 else (current, current, current)) + (at,)


@pytest.mark.parametrize("levels,brick_size", [(1, 8), (3, 8), (2, 4)])
def test_advection_matches_the_per_face_definition(gpu, levels, brick_size):
    built = build(levels, brick_size)
    lattice = Lattice(built.topology, brick_size)
    rng = np.random.default_rng(11 * levels + brick_size)
    with CompositeSystem(built.topology) as s:
        shapes = [(s.bricks, brick_size + (c == 2), brick_size + (c == 1), brick_size + (c == 0)) for c in range(3)]
        before = []
        for c in range(3):
            # a smooth flow of the node positions, the same on both copies of a shared face
            f = np.empty(shapes[c], np.float32)
            k, j, i = np.meshgrid(*[np.arange(n) for n in shapes[c][1:]], indexing="ij")
            for slot in range(s.bricks):
                h = float(lattice.h[lattice.level[slot]])
                x, y, z = (float(lattice.rec[slot][a]) + (q + (0.0 if a == c else 0.5)) * h for a, q in enumerate((i, j, k)))
                f[slot] = U * ((c == 0) + 0.3 * np.sin(2.1 * x + 1.3 * y + c) * np.cos(1.7 * z - 0.9 * y + 0.5 * c))
            before.append(f)
        s.set_faces(*[f.ravel() for f in before])
        s.set_mac_links(*[np.full(s.faces, 0x3F, np.uint8)] * 3)
        dt = float(F(0.5 * float(min(lattice.h)) / (1.4 * U)))
        s.mac_advect(dt)
        after = [f.reshape(shapes[c]) for c, f in enumerate(s.get_faces())]
    kept = [q for q in range(len(lattice.cov)) if not lattice.cov[q]]
    moved = 0.0
    for _ in range(120):
        slot, c = int(rng.choice(kept)), int(rng.integers(3))
        # half of the faces on the brick's rim, where samples leave the lattice
        ijk = [int(rng.choice([0, n - 1])) if rng.random() < 0.5 else int(rng.integers(n)) for n in lattice.size(c)]
        level, p = lattice.level[slot], lattice.point(c, slot, ijk)
        want, low, high, back = lattice.forward(before, c, slot, ijk, dt)
        foot = lattice.trace(before, slot, p, -dt)
        ahead, owner = lattice.locate(foot), lattice.locate(lattice.clamp(p))
        if min(back, ahead, owner) >= 0 and lattice.level[back] == lattice.level[ahead] == lattice.level[owner] == level:
            class Forward:                                    # the forward field, evaluated where it is read
                def __init__(self, axis):
                    self.axis = axis

                def __getitem__(self, q):
                    return lattice.forward(before, self.axis, q[0], [q[3], q[2], q[1]], dt)[0]
            again = lattice.sample([Forward(a) for a in range(3)], c, ahead, foot)[0]
            want = max(low, min(high, want + 0.5 * (lattice.clamped(before, c, slot, ijk) - again)))
        got = float(after[c][slot, ijk[2], ijk[1], ijk[0]])
        moved = max(moved, abs(got - lattice.clamped(before, c, slot, ijk)))
        assert abs(got - want) <= 1e-5 * U, (levels, slot, c, ijk, got, want)
    assert moved > 1e-3 * U                                   # the step moved the field by 100 tolerances
    for c in range(3):                                        # covered bricks' faces end as 0
        assert not np.any(after[c][np.array(lattice.cov)])
    built.close()


class Faces(Lattice):
    """The band update, the eddy viscosity and the diffusion of a face, from their definitions."""

    def cell_point(self, s, ijk):
        return [F(self.rec[s][a] + F(ijk[a] + 0.5) * self.h[self.level[s]]) for a in range(3)]

    def stepped(self, c, axis, direction, s, ijk):
        """(slot, face) one step along axis inside the level, or None."""
        q, n = list(ijk), self.size(c)
        q[axis] += direction
        out = [a for a in range(3) if q[a] < 0 or q[a] >= n[a]]
        if not out:
            return s, q
        nb = self.nb[s][2 * axis + (direction > 0)]
        if len(out) > 1 or nb < 0 or self.cov[nb]:
            return None
        q[axis] -= direction * self.bs
        return nb, q

    def band(self, f, links, c, s, ijk, dt):
        def minmod(a, b):
            return 0.0 if a * b <= 0 else (a if abs(a) < abs(b) else b)

        def opened(at, bit):
            slot, q = at
            return int(links[c][slot, q[2], q[1], q[0]]) >> bit & 1
        here, p, h = (s, list(ijk)), self.point(c, s, ijk), float(self.h[self.level[s]])
        current = low = high = self.clamped(f, c, s, ijk)
        total = weights = 0.0
        for axis in range(3):
            velocity = self.sample(f, axis, s, p)[0]
            up = -1 if velocity >= 0 else 1
            bit, other = 2 * axis + (up > 0), 2 * axis + (up < 0)
            first = self.stepped(c, axis, up, *here) if opened(here, bit) else None
            if first is None:
                continue
            upstream = self.clamped(f, c, *first)
            low, high = min(low, upstream), max(high, upstream)
            weight = dt * abs(velocity) / h
            delta = weight * (upstream - current)
            second, down = self.stepped(c, axis, up, *first), self.stepped(c, axis, -up, *here)
            if opened(here, other) and opened(first, bit) and second and down:
                far, downstream = self.clamped(f, c, *second), self.clamped(f, c, *down)
                low, high = min(low, downstream), max(high, downstream)
                incoming = upstream + 0.5 * minmod(upstream - far, current - upstream)
                delta = -weight * (current + 0.5 * minmod(current - upstream, downstream - current) - incoming)
            total, weights = total + delta, weights + weight
        return max(low, min(high, current + total / max(1.0, weights)))

    def advected(self, f, links, c, s, ijk, dt):
        def first(a, slot, q):
            if int(links[a][slot, q[2], q[1], q[0]]) & 0x40:
                return self.band(f, links, a, slot, q, dt)
            return self.forward(f, a, slot, q, dt)[0]
        if int(links[c][s, ijk[2], ijk[1], ijk[0]]) & 0x40:
            return first(c, s, ijk)
        value, low, high, back = self.forward(f, c, s, ijk, dt)
        p, level = self.point(c, s, ijk), self.level[s]
        foot = self.trace(f, s, p, -dt)
        ahead, owner = self.locate(foot), self.locate(self.clamp(p))
        if min(back, ahead, owner) < 0 or any(self.level[q] != level for q in (back, ahead, owner)):
            return value

        class Forward:                                    # the forward field, evaluated where it is read
            def __init__(self, axis):
                self.axis = axis

            def __getitem__(self, q):
                return first(self.axis, q[0], [q[3], q[2], q[1]])
        again = self.sample([Forward(a) for a in range(3)], c, ahead, foot)[0]
        return max(low, min(high, value + 0.5 * (self.clamped(f, c, s, ijk) - again)))

    def eddy(self, f, s, ijk, cs):
        h, centre = self.h[self.level[s]], self.cell_point(s, ijk)
        g = np.empty((3, 3))
        for c in range(3):
            for axis in range(3):
                lo, hi = list(centre), list(centre)
                lo[axis], hi[axis] = F(lo[axis] - h), F(hi[axis] + h)
                g[c, axis] = (self.sample(f, c, s, hi)[0] - self.sample(f, c, s, lo)[0]) / (2 * float(h))
        strain = 0.5 * (g + g.T)
        return (cs * float(h)) ** 2 * np.sqrt(2 * (strain ** 2).sum())

    def cell(self, nut, s, ijk):
        bs = self.bs

        def clamped(slot, q):
            i, j, k = (min(max(x, 0), bs - 1) for x in q)
            return float(nut[slot, k, j, i])

        def extended(slot, q):
            terms = [((), 1.0)]
            for x in q:
                ends = ((0, 2.0), (1, -1.0)) if x < 0 else ((bs - 1, 2.0), (bs - 2, -1.0)) if x >= bs else ((x, 1.0),)
                terms = [(t + (e,), w * v) for t, w in terms for e, v in ends]
            return sum(w * clamped(slot, t) for t, w in terms)
        out = [a for a in range(3) if ijk[a] < 0 or ijk[a] >= bs]
        if not out:
            return clamped(s, ijk)
        if len(out) == 1:
            a = out[0]
            nb = self.nb[s][2 * a + (ijk[a] >= bs)]
            if nb >= 0 and not self.cov[nb]:
                q = list(ijk)
                q[a] += bs if ijk[a] < 0 else -bs
                return clamped(nb, q)
        p = self.cell_point(s, ijk)
        at = self.locate(p)
        if at < 0:
            return clamped(s, ijk)
        x = [float(F((p[a] - self.rec[at][a]) / self.h[self.level[at]] - F(0.5))) for a in range(3)]
        if self.level[at] == self.level[s]:
            return clamped(at, [int(np.floor(v + 0.5)) for v in x])
        i0, total = [int(np.floor(v)) for v in x], 0.0
        for d in np.ndindex(2, 2, 2):
            w = np.prod([x[a] - i0[a] if d[a] else 1.0 - (x[a] - i0[a]) for a in range(3)])
            total += w * extended(at, [i0[a] + d[a] for a in range(3)])
        return total

    def diffused(self, f, links, nut, c, s, ijk, nu, dt):
        link, current, viscosity, laplacian = int(links[c][s, ijk[2], ijk[1], ijk[0]]), self.clamped(f, c, s, ijk), nu, 0.0
        for axis in range(3):
            for direction in (-1, 1):
                if not link & 0x40 or link >> (2 * axis + (direction > 0)) & 1:
                    q = list(ijk)
                    q[axis] += direction
                    laplacian += self.node(f, c, s, q) - current
        if not link & 0x40:
            lower = list(ijk)
            lower[c] -= 1
            viscosity += 0.5 * (self.cell(nut, s, lower) + self.cell(nut, s, list(ijk)))
        return current + dt * viscosity * laplacian / float(self.h[self.level[s]]) ** 2


def smooth_faces(lattice, bricks):
    """A smooth flow of the node positions, the same on both copies of a shared face."""
    bs, out = lattice.bs, []
    for c in range(3):
        f = np.empty((bricks, bs + (c == 2), bs + (c == 1), bs + (c == 0)), np.float32)
        k, j, i = np.meshgrid(*[np.arange(n) for n in f.shape[1:]], indexing="ij")
        for slot in range(bricks):
            h = float(lattice.h[lattice.level[slot]])
            x, y, z = (float(lattice.rec[slot][a]) + (q + (0.0 if a == c else 0.5)) * h for a, q in enumerate((i, j, k)))
            f[slot] = U * ((c == 0) + 0.3 * np.sin(2.1 * x + 1.3 * y + c) * np.cos(1.7 * z - 0.9 * y + 0.5 * c))
        out.append(f)
    return out


def band_links(faces, rng):
    """Half of the faces in the band, with open directions at random; the others open."""
    return [np.where(rng.random(f.shape) < 0.5, 0x40 | rng.integers(0, 64, f.shape), 0x3F).astype(np.uint8) for f in faces]


def picked(lattice, rng, count):
    """Faces of non-covered bricks, half of the indices on the brick's rim."""
    kept = [q for q in range(len(lattice.cov)) if not lattice.cov[q]]
    for _ in range(count):
        slot, c = int(rng.choice(kept)), int(rng.integers(3))
        yield slot, c, [int(rng.choice([0, n - 1])) if rng.random() < 0.5 else int(rng.integers(n)) for n in lattice.size(c)]


@pytest.mark.parametrize("levels,brick_size", [(1, 8), (3, 8), (2, 4)])
def test_band_faces_match_the_per_face_definition(gpu, levels, brick_size):
    """Advection with half of the faces in the near-surface band: bounds as above."""
    built = build(levels, brick_size)
    lattice = Faces(built.topology, brick_size)
    rng = np.random.default_rng(23 * levels + brick_size)
    with CompositeSystem(built.topology) as s:
        before = smooth_faces(lattice, s.bricks)
        links = band_links(before, rng)
        s.set_faces(*[f.ravel() for f in before])
        s.set_mac_links(*[q.ravel() for q in links])
        dt = float(F(0.5 * float(min(lattice.h)) / (1.4 * U)))
        s.mac_advect(dt)
        after = [f.reshape(b.shape) for f, b in zip(s.get_faces(), before)]
    moved = 0.0
    for slot, c, ijk in picked(lattice, rng, 100):
        want, got = lattice.advected(before, links, c, slot, ijk, dt), float(after[c][slot, ijk[2], ijk[1], ijk[0]])
        moved = max(moved, abs(got - lattice.clamped(before, c, slot, ijk)))
        assert abs(got - want) <= 1e-5 * U, (levels, slot, c, ijk, got, want)
    assert moved > 1e-3 * U
    built.close()


@pytest.mark.parametrize("levels,brick_size,base", [(1, 8, 0.125), (3, 8, 0.125), (2, 4, 0.125), (3, 8, 1 / 12)])
def test_diffusion_matches_the_per_face_definition(gpu, levels, brick_size, base):
    """Eddy viscosity of a cell and diffusion of a face, half of the faces in the band.  A velocity
    gradient is the difference of two samples (4e-6 U each) over 2 h: nine of them leave |S| within
    2e-5 U / h.  The Laplacian's seven values err by 4e-6 U each, times a factor of at most 0.2.  With
    cells of 1/12 the sample points one cell off a centre miss the ghost nodes by a rounding."""
    built = build(levels, brick_size, base)
    lattice = Faces(built.topology, brick_size)
    rng = np.random.default_rng(31 * levels + brick_size)
    nu, cs = 0.2, 0.17
    with CompositeSystem(built.topology) as s:
        before = smooth_faces(lattice, s.bricks)
        links = band_links(before, rng)
        s.set_faces(*[f.ravel() for f in before])
        s.set_mac_links(*[q.ravel() for q in links])
        dt = float(F(0.15 * float(min(lattice.h)) ** 2 / nu))
        s.mac_diffuse_smagorinsky(nu, cs, dt)
        after = [f.reshape(b.shape) for f, b in zip(s.get_faces(), before)]
        nut = s.mac_eddy_viscosity()[:s.bricks * brick_size ** 3].reshape(s.bricks, *[brick_size] * 3)
    moved = 0.0
    for slot, c, ijk in picked(lattice, rng, 100):
        cell = [min(q, brick_size - 1) for q in ijk]
        h = float(lattice.h[lattice.level[slot]])
        assert abs(float(nut[slot, cell[2], cell[1], cell[0]]) - lattice.eddy(before, slot, cell, cs)) <= (cs * h) ** 2 * 2e-5 * U / h, (slot, cell)
        want, got = lattice.diffused(before, links, nut, c, slot, ijk, nu, dt), float(after[c][slot, ijk[2], ijk[1], ijk[0]])
        moved = max(moved, abs(got - lattice.clamped(before, c, slot, ijk)))
        assert abs(got - want) <= 1e-5 * U, (levels, slot, c, ijk, got, want)
    assert moved > 1e-3 * U
    for c in range(3):                                        # covered bricks' faces end as 0
        assert not np.any(after[c][np.array(lattice.cov)])
    built.close()
