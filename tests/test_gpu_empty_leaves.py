"""Trees with empty leaves: where all particles of a node share the split
coordinate (sheets, lines, lattices), the rounded mean can fall below every
one of them, and the lower child then holds nothing (as in the reference).

The GPU's mean is a lane-strided sum, the oracle's a sequential one, so on
such input the two mostly round differently and the oracle's tree is
another.  The tree is therefore compared with a replay of the split rule in
the GPU's order of additions, and the forces with a direct sum over all 27
images (theta 0 and a cutoff beyond the images: every leaf pair is
evaluated, so the forces do not depend on the tree).  A few small sets where
both orders give one tree pin the lists, moments and forces to the oracle."""
import numpy as np
import pytest
from scipy.special import erfc

pytestmark = pytest.mark.gpu

L = 100.0


def lane_sums(v):
    """Sums of the rows of v (m, 32 k): lane l adds elements l, l + 32, ..., then the warp's butterfly."""
    a = v.reshape(v.shape[0], -1, 32)
    s = np.zeros((a.shape[0], 32))
    for k in range(a.shape[1]):
        s = s + a[:, k]
    for o in (16, 8, 4, 2, 1):
        s = s + s[:, np.arange(32) ^ o]
    return s[:, 0]


def padded(v, m):
    return np.concatenate([v, np.zeros(-len(v) % m)])


def mean(c):
    """Sums of chunks of 1,024, then the sum of those."""
    chunks = lane_sums(padded(c, 1024).reshape(-1, 1024))
    return lane_sums(padded(chunks, 32)[None])[0] / len(c)


def replay(pos, maxleaf):
    """(permutation, leaf start, leaf size, node size, node children (leaf l
    as ~l)): leaves depth-first, nodes in preorder, axes x, y, z in turn."""
    perm = np.arange(len(pos))
    pos = pos.copy()
    leaves, nodes = [], []
    todo = [(0, len(pos), 0, -1, 0)]
    while todo:
        start, n, depth, parent, side = todo.pop()
        if n <= maxleaf:
            nodes[parent][1 + side] = ~len(leaves)
            leaves.append((start, n))
            continue
        if parent >= 0:
            nodes[parent][1 + side] = len(nodes)
        assert depth < 200
        c = pos[start:start + n, depth % 3].copy()
        left = 1
        if n == 2:
            if c[0] > c[1]:
                pos[start:start + 2] = pos[start:start + 2][::-1].copy()
                perm[start:start + 2] = perm[start:start + 2][::-1].copy()
        else:
            small = c <= mean(c)
            left = int(small.sum())
            if left == n:
                left = n - 1
            else:
                i = start + np.nonzero(~small[:left])[0]
                j = start + left + np.nonzero(small[left:])[0][::-1]
                a, b = np.concatenate([i, j]), np.concatenate([j, i])
                pos[a], perm[a] = pos[b], perm[b]
        todo.append((start + left, n - left, depth + 1, len(nodes), 1))
        todo.append((start, left, depth + 1, len(nodes), 0))
        nodes.append([n, 0, 0])
    leaves, nodes = np.array(leaves), np.array(nodes)
    return perm, leaves[:, 0], leaves[:, 1], nodes[:, 0], nodes[:, 1:]


def sheet(n, z, axis=2, background=0):
    p = np.random.default_rng(n).uniform(0.0, L, (n, 3))
    p[background:, axis] = z
    return p


def lattice(*dims):
    axes = [(np.arange(d) + 0.5) * (L / d) for d in dims]
    return np.stack(np.meshgrid(*axes, indexing="ij"), -1).reshape(-1, 3)


SMALL = [
    (sheet(3000, 1.3), 16),
    (sheet(4096, 0.1, axis=0), 16),
    (sheet(1000, 33.3), 16),
    (sheet(500, 0.3), 2),
    (sheet(3000, 1.3), 64),
    (lattice(7, 11, 13), 5),
    (lattice(3, 50, 21), 8),
]


def check_tree(fp, pos, maxleaf):
    perm, start, size, node, son = replay(pos, maxleaf)
    assert (size == 0).any()
    n = len(pos)
    cap = int(2.0 * n / maxleaf)
    assert max(len(size), len(node)) <= cap
    tr = fp.tree()
    assert np.array_equal(fp.perm(), perm)
    assert np.array_equal(tr["leaf_ipart"], start)
    assert np.array_equal(tr["leaf_npart"], size)
    assert np.array_equal(tr["node_npart"], node)
    assert np.array_equal(tr["node_son"], np.where(son < 0, n + ~son, n + cap + son))


def all_pairs(pos, p, targets):
    out = np.zeros((len(targets), 3))
    shifts = [L * np.array((i, j, k)) for i in (-1, 0, 1) for j in (-1, 0, 1) for k in (-1, 0, 1)]
    for k, t in enumerate(targets):
        for s in shifts:
            d = pos + s - pos[t]
            r = np.sqrt((d ** 2).sum(1))
            u = 0.5 * r / p["rs"]
            f = p["mass"] * (erfc(u) + 2.0 / np.sqrt(np.pi) * u * np.exp(-u * u)) / np.maximum(r, p["eps"]) ** 3
            if not s.any():
                f[t] = 0.0
            out[k] += (f[:, None] * d).sum(0)
    return out


def check_forces(acc, pos, p):
    """FP64 against the direct sum, relative to the largest force of the
    sample (a regular set's forces cancel)."""
    targets = np.arange(0, len(pos), max(1, len(pos) // 60))
    want = all_pairs(pos, p, targets)
    scale = np.linalg.norm(want, axis=1).max() + 1e-2 * p["mass"]
    assert np.abs(acc[targets] - want).max() <= 1e-10 * scale


def direct_params(maxleaf):
    return dict(boxsize=L, theta=0.0, rs=8.0, rcut=4.0 * L, eps=0.1, mass=1.0, maxleaf=maxleaf)


@pytest.fixture(scope="module")
def fp(ph):
    f = ph.ForcePass(0)
    yield f
    f.close()


@pytest.mark.parametrize("case", range(len(SMALL)))
def test_tree_and_forces_with_empty_leaves(ph, fp, case):
    pos, maxleaf = SMALL[case]
    p = direct_params(maxleaf)
    acc = fp.run(pos, p, precision=ph.FP64, flags=ph.F_ONE_WAY)
    check_tree(fp, pos, maxleaf)
    check_forces(acc, pos, p)


@pytest.mark.parametrize("case", range(len(SMALL)))
def test_fp64_mutual_pairs_with_empty_leaves(ph, fp, case):
    pos, maxleaf = SMALL[case]
    p = direct_params(maxleaf)
    check_forces(fp.run(pos, p, precision=ph.FP64), pos, p)


@pytest.mark.parametrize("case", range(len(SMALL)))
@pytest.mark.parametrize("flags", [None, "F_ONE_WAY"])
def test_fp32_pairs_with_empty_leaves(ph, fp, case, flags):
    """Mutual pairs (leaf 64) or one way, long lists by a block, against the
    FP64 pass.  The bars of the clustered inputs (median 1e-5, 99th
    percentile 1e-4), and for lattices, whose forces cancel, that of the
    golden lattice: 1e-5 of one nearest-neighbour pair force."""
    pos, maxleaf = SMALL[case]
    p = direct_params(maxleaf)
    a64 = fp.run(pos, p, precision=ph.FP64, flags=ph.F_ONE_WAY)
    a32 = fp.run(pos, p, precision=ph.FP32_SPLIT, flags=getattr(ph, flags) if flags else 0)
    if case >= 5:
        r = np.linalg.norm(pos[1:] - pos[0], axis=1).min()
        assert np.abs(a32 - a64).max() <= 1e-5 * p["mass"] / r ** 2
        return
    e = np.linalg.norm(a32 - a64, axis=1) / np.linalg.norm(a64, axis=1)
    assert np.median(e) <= 1e-5, np.median(e)
    assert np.percentile(e, 99) <= 1e-4, np.percentile(e, 99)


@pytest.mark.parametrize("n,z,background,maxleaf", [(30000, 0.1, 15000, 24), (2200000, 0.1, 1100000, 48)])
def test_numbering_of_large_trees_with_empty_leaves(ph, fp, n, z, background, maxleaf):
    """Nodes split by the levels, and the scans that take several blocks."""
    pos = sheet(n, z, background=background)
    p = dict(boxsize=L, theta=0.5, rs=0.5, rcut=2.25, eps=0.01, mass=1.0, maxleaf=maxleaf)
    fp.run(pos, p, precision=ph.FP64, flags=ph.F_ONE_WAY)
    check_tree(fp, pos, maxleaf)


@pytest.mark.parametrize("graph", ["1", "0"])
def test_subtree_with_more_leaves_than_one_block_holds(ph, graph, monkeypatch):
    """A line of 1,000 particles whose y and z splits are empty, beside 1,500
    others: 1,240 leaves under a node of 1,000 particles.  Also the pass
    after it (which starts from the small subtrees) and an ordinary one."""
    monkeypatch.setenv("PHOTONS_GRAPH", graph)
    rng = np.random.default_rng(5)
    pos = rng.uniform(0.0, 50.0, (2500, 3)) * (1.0, 2.0, 2.0)
    pos[1500:] = (0.0, 54.723, 56.247)
    pos[1500:, 0] = rng.uniform(90.0, 100.0, 1000)
    p = dict(boxsize=L, theta=0.5, rs=2.0, rcut=9.0, eps=0.1, mass=1.0, maxleaf=2)
    fp = ph.ForcePass(0)
    for _ in range(2):
        fp.run(pos, p, precision=ph.FP64)
        check_tree(fp, pos, 2)
    fp.run(sheet(3000, 1.3), dict(p, maxleaf=16), precision=ph.FP64)
    check_tree(fp, sheet(3000, 1.3), 16)
    fp.close()


@pytest.mark.parametrize("n,maxleaf,z,seed,axis,sheet_only", [
    (342, 2, 89.47, 72207, 2, False), (286, 2, 7.35, 199521, 2, False), (248, 2, 99.85, 905296, 2, False),
    (111, 2, 90.09, 864797, 1, True), (266, 2, 29.37, 523163, 1, False), (355, 2, 53.93, 810033, 1, False),
    (54, 2, 50.42, 939406, 2, True), (369, 2, 30.37, 564142, 0, False)])
def test_lists_and_forces_with_empty_leaves_match_oracle(ph, fp, port, n, maxleaf, z, seed, axis, sheet_only):
    """Sets with empty leaves whose tree is the oracle's: every list, the
    moments and the forces (FP64 bar) as the oracle's, mutual and one way."""
    rng = np.random.default_rng(seed)
    pos = rng.uniform(0.0, 100.0, (n, 3))
    pos[:, axis] = z
    if not sheet_only:
        pos[n // 2:] = rng.uniform(0.0, 100.0, (n - n // 2, 3))
    p = dict(boxsize=100.0, theta=0.7, rs=8.0, rcut=36.0, eps=0.1, mass=1.0, maxleaf=maxleaf)
    r = port.run(pos, p, capture=True, tree=True, nthreads=4)
    assert (r["tree"]["leaf_npart"] == 0).any()
    for flags in (0, ph.F_ONE_WAY):
        acc = fp.run(pos, p, precision=ph.FP64, flags=flags | ph.F_TREE_ORDER | ph.F_KEEP_LISTS | ph.F_MULTIPOLES)
        tr = fp.tree()
        for k in ("leaf_ipart", "leaf_npart", "node_npart", "node_son"):
            assert np.array_equal(tr[k], r["tree"][k]), k
        for kind, (t, s, im) in fp.lists().items():
            a = np.stack([t, s, im], 1)
            b = np.stack([np.asarray(x) for x in r["lists"][kind]], 1)
            assert np.array_equal(a[np.lexsort(a.T)], b[np.lexsort(b.T)]), kind
        for k in ("leaf_M", "node_M"):
            assert np.abs(tr[k] - r["tree"][k]).max() <= 1e-11 * np.abs(r["tree"][k]).max(), k
        scale = np.linalg.norm(r["acc"], axis=1)
        assert (np.linalg.norm(acc - r["acc"], axis=1) <= 1e-10 * scale).all()
