"""The culling of the patch distance pass (csrc/m2v_patch.cuh) as a property,
on the CPU: with the kernel's float32 frame, coefficients and margin, no
(voxel, sub-triangle) pair is ever culled against a running minimum equal to
its own float32 distance, neither by its patch's outline nor by its own.
Triangles of every shape, cut into 1 to 40^2 sub-triangles by the reference's
accumulated steps, near the origin and far from it."""
import numpy as np

from tests.test_cull_bound import U, closest_dist2, cross3, cull_coeffs, dot3, fmaf

F = np.float32
INF = F(np.inf)
CULL_FACTOR, SC = F(1.00196), F(22.66)


def grid(p1, p2, p3, n):
    """Vertices at (row, column) of the reference's stepping (mesh_to_volume.rs:75-116)."""
    inv = F(1.0) / F(n)
    s1, s2 = (p2 - p1) * inv, (p3 - p2) * inv
    v = np.zeros((n + 1, n + 1, 3), F)
    if n == 1:
        v[0, 0], v[1, 0], v[1, 1] = p1, p2, p3
        return v, s1, s2
    a = p1
    for r in range(n + 1):
        q = a
        for k in range(r + 1):
            v[r, k] = q
            q = q + s2
        a = a + s1
    return v, s1, s2


def patches(n):
    if n <= 3:
        return [(0, 0, n, n)]
    return [(r, k, min(2, n - r), min(2, n - k)) for r in range(0, n, 2) for k in range(0, r + 1, 2)]


def test_no_pair_is_culled_against_its_own_distance():
    rng = np.random.default_rng(5)
    h = F(0.002)
    tested = near = 0
    for it in range(300):
        n = int(rng.choice([1, 2, 3, 4, 5, 8, 13, 40], p=[.1, .15, .25, .15, .1, .1, .1, .05]))
        centre = rng.uniform(-1, 1, 3) * rng.choice([0.1, 2.0, 40.0])
        t = rng.normal(size=(3, 3))
        if it % 3 == 1:  # slender
            t[2] = t[0] + rng.uniform(0.2, 0.8) * (t[1] - t[0]) + rng.normal(size=3) * 10.0 ** rng.uniform(-2, -0.5)
        side = max(np.linalg.norm(t[i] - t[j]) for i, j in ((0, 1), (0, 2), (1, 2)))
        t = (centre + t * (float(h) * (n + rng.uniform(0.05, 0.95)) / side)).astype(F)
        p1, p2, p3 = t
        v, s1, s2 = grid(p1, p2, p3, n)
        for r0, k0, rows, cols in patches(n) if n < 13 else [patches(n)[i] for i in rng.choice(len(patches(n)), 12)]:
            subs = []
            for r in range(r0, r0 + rows):
                for k in range(k0, min(k0 + cols, r + 1)):
                    subs.append((r, k, 0, v[r, k], v[r + 1, k], v[r + 1, k + 1]))
                    if k < r:
                        subs.append((r, k, 1, v[r, k], v[r + 1, k + 1], v[r, k + 1]))
            A, B, C = (np.array([s[i] for s in subs], F) for i in (3, 4, 5))
            box = np.concatenate([A, B, C])
            lo, hi = np.floor(box.min(0) / h) - 4, np.ceil(box.max(0) / h) + 4
            R = F(h * (np.linalg.norm(hi - lo) + 2))
            M = F(max(np.abs(t).max(), h * (np.abs(np.concatenate([lo, hi])).max() + 1)))
            c2, e0 = cull_coeffs(A, B, C, np.full(len(A), R, F), np.full(len(A), M, F))
            if not np.isfinite(c2).all():
                continue
            ab, ac, cb = B - A, C - A, C - B
            e2 = np.maximum(dot3(ab, ab), np.maximum(dot3(ac, ac), dot3(cb, cb)))
            nn = cross3(ab, ac)
            E1 = e0 - F(1.5) * (F(1024.0) * U * (e2 * np.sqrt(e2) / dot3(nn, nn))) * e2
            # k_patches: the affine frame
            d = s1 + s2
            N = cross3(s1, s2)
            l1, l2, ld = dot3(s1, s1), dot3(s2, s2), dot3(d, d)
            area = np.sqrt(dot3(N, N))
            h1, h2, h3 = area / np.sqrt(l2), area / np.sqrt(l1), area / np.sqrt(ld)
            rm, km = F(r0 + 0.5 * rows), F(k0 + 0.5 * cols)
            ref = p1 + rm * s1 + km * s2
            m1, m2, m3 = (x / (area * np.sqrt(l)) for x, l in ((cross3(s2, N), l2), (cross3(N, s1), l1), (cross3(N, d), ld)))
            delta = (F(4 * n + 8)) * U * M + F(16) * U * np.sqrt(max(l1, l2, ld)) * F(n) + \
                (F(32) + F(64) * max(l1, l2, ld) / area) * U * R
            cs, es = SC * (F(0.25) * c2.max()), SC * (E1.max() + delta)
            # voxels around the patch, many of them over its edges and corners
            w = rng.dirichlet(np.ones(3), 150) * rng.choice([1.0, 1.3], (150, 1))
            at = (w[:, :1] * A[0] + w[:, 1:2] * B[-1] + w[:, 2:] * C[len(A) // 2])
            g = (np.rint((at + rng.normal(size=(150, 3)) * float(h) * rng.choice([0.3, 2.0], (150, 1))) / h).astype(F) * h)
            x = g - ref
            lin = [x @ (N / area), x @ m1, x @ m2, x @ m3 + (km - rm) * h3]
            wd, rho, kap, cc = (y.astype(F) for y in lin)

            def culled(e, cur):
                lb = fmaf(e, e, wd * wd)
                tm = fmaf(np.full_like(lb, cs), lb, np.full_like(lb, es))
                return lb > fmaf(tm, tm, CULL_FACTOR * cur)

            e_patch = np.maximum(np.maximum(np.abs(rho) - F(0.5 * rows) * h1, np.abs(kap) - F(0.5 * cols) * h2),
                                 np.maximum(cc, F(0)))
            for (r, k, down, *_), a, b, c in zip(subs, A, B, C):
                tri = [np.broadcast_to(y, g.shape) for y in (a, b, c)]
                cur = closest_dist2(*tri, g)
                ra = rho + (F(0.5 * rows) - F(r - r0)) * h1
                ka = kap + (F(0.5 * cols) - F(k - k0)) * h2
                cd = F(r - k) * h3 + cc
                e = np.maximum(np.maximum(-ra, ka - h2), -cd) if down else np.maximum(np.maximum(ra - h1, -ka), cd)
                e = np.maximum(e, F(0)).astype(F)
                assert not culled(e_patch.astype(F), cur).any()
                assert not culled(e, cur).any()
                tested += len(cur)
                near += int((fmaf(e, e, wd * wd) > F(0.99) * cur).sum())
    assert tested > 100_000 and near > 0.2 * tested  # the bound is close to the distance on many pairs
