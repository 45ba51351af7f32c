"""grid_spec's classification of random grids against a comparison per axis."""
import numpy as np

from simu_rca_ab_b200.params import grid_spec


def _varying(a):
    return [k for k in range(3) if a.shape[k] > 1 and not np.array_equal(a, np.broadcast_to(np.take(a, [0], k), a.shape))]


def test_grid_classification_matches_the_per_axis_comparison():
    rng = np.random.default_rng(0)
    kinds = set()
    for _ in range(500):
        sh = tuple(int(k) for k in rng.integers(1, 5, 3))
        perm = rng.permutation(3)
        arrs = []
        for c in range(3):
            k = int(perm[c]) if rng.random() < 0.9 else int(rng.integers(3))
            line = rng.normal(size=sh[k]).reshape([-1 if i == k else 1 for i in range(3)])
            a = np.broadcast_to(line, sh).copy(order="F" if rng.random() < 0.3 else "C")
            if rng.random() < 0.15:
                a[tuple(int(rng.integers(0, s)) for s in sh)] += rng.choice([1.0, np.nan, 0.0])
            arrs.append(a)
        v = [_varying(a) for a in arrs]
        used = [x[0] for x in v if len(x) == 1]
        rect = all(len(x) <= 1 for x in v) and len(set(used)) == len(used)
        g = grid_spec(*arrs)
        assert g.kind == (0 if rect else 1) and g.shape == sh
        if rect:
            for a, line, x in zip(arrs, (g.x, g.y, g.z), v):
                if x:
                    assert np.array_equal(line, np.moveaxis(a, x[0], 0)[:, 0, 0], equal_nan=True)
        kinds.add(g.kind)
    assert kinds == {0, 1}
