"""Sizes at which the tree, list and direct-sum kernels change tile, launch
shape or code path, against the oracle: trees bit-exact, FP64 direct sums
within 1e-12, FP32 force passes within 1e-6 (the bars of test_gpu_fmm.py)."""
import numpy as np
import pytest
from conftest import rel_l2

import fmmgpu
from fmmgpu import workloads

pytestmark = pytest.mark.gpu


# tiles of 1024 sorted keys (levels, cells) and 2048 items (sorts and lists), and 65,536 items, up to which the sort
# adds its tile histograms up itself
@pytest.mark.parametrize("dim", [2, 3])
@pytest.mark.parametrize("n", [1, 2, 3, 31, 33, 1023, 1024, 1025, 2047, 2049, 65535, 65537])
def test_tree_at_tile_edges(oracle, n, dim):
    gen = workloads.plummer if dim == 3 else workloads.disk_clumps_2d
    pos = gen(n, seed=31)[0]
    want = oracle.tree(pos, 16)
    with fmmgpu.Context(dim=dim, leaf_cap=16) as c:
        got = c.tree(pos, with_pairs=False)
    assert got["depth"] == want["depth"]
    for k in ("leaf_keys", "leaf_start", "perm"):
        np.testing.assert_array_equal(got[k], want[k])
    for a, b in zip(got["level_keys"], want["level_keys"]):
        np.testing.assert_array_equal(a, b)


# the one-launch sort: 1 to 8 blocks of 2, 4, 8 or 16 items per thread, up to 32,768 items
@pytest.mark.parametrize("dim", [2, 3])
@pytest.mark.parametrize("n", [512, 513, 4096, 4097, 8192, 8193, 16384, 16385, 32768, 32769])
def test_tree_at_sort_edges(oracle, n, dim):
    gen = workloads.plummer if dim == 3 else workloads.disk_clumps_2d
    pos = gen(n, seed=32)[0]
    want = oracle.tree(pos, 16, with_pairs=False)
    with fmmgpu.Context(dim=dim, leaf_cap=16) as c:
        got = c.tree(pos, with_pairs=False)
    for k in ("depth", "leaf_keys", "leaf_start", "perm"):
        np.testing.assert_array_equal(got[k], want[k])
    for a, b in zip(got["level_keys"], want["level_keys"]):
        np.testing.assert_array_equal(a, b)


def test_tree_with_many_equal_keys(oracle):
    """More than 512 particles with one key at the maximum depth (the leaf
    order by a sort) next to single ones, and runs across tiles."""
    rng = np.random.default_rng(5)
    pos = np.concatenate([rng.random((40, 3)), np.repeat(rng.random((2, 3)), [700, 2300], axis=0), rng.random((60, 3))])
    rng.shuffle(pos)
    want = oracle.tree(pos, 64)
    with fmmgpu.Context(dim=3, leaf_cap=64) as c:
        got = c.tree(pos, with_pairs=False)
    for k in ("leaf_keys", "leaf_start", "perm"):
        np.testing.assert_array_equal(got[k], want[k])


# boxes far from a cube: whole cell pairs are summed directly, large cells by several warps (32 targets each)
# (adaptive targets need a tree of depth 3: from 6000 particles)
@pytest.mark.parametrize("n,adaptive", [(700, 0), (6000, 0), (20000, 0), (6000, 32), (20000, 32)])
@pytest.mark.parametrize("stretch", [(1.0, 0.7, 1.0), (1.0, 0.45, 0.6)])
def test_elongated_box(oracle, n, adaptive, stretch):
    pos, m = workloads.uniform_cube(n, seed=41)
    pos = pos * np.array(stretch)
    with fmmgpu.Context(dim=3, p=6, leaf_cap=32, direct_max=128, m2l_mode=fmmgpu.FMM_M2L_TC,
                        adaptive_leaf=adaptive) as c:
        acc, pot = c.evaluate(pos, m, want_pot=True)
    if adaptive:
        want = oracle.fmm_adaptive(pos, m, 6, 32, aleaf=adaptive, direct_max=128, w_direct_max=10 ** 18, want_pot=True)
    else:
        want = oracle.fmm(pos, m, 6, 32, direct_max=128, want_pot=True)
    assert rel_l2(acc, want[0]) < 1e-6
    assert rel_l2(pot, want[1]) < 1e-6


def _direct(pos, m, targets, soft, eps2):
    """The sum in FP64, term by term as the kernel's two forms."""
    dim = pos.shape[1]
    acc, pot = np.zeros((len(targets), dim)), np.zeros(len(targets))
    for k, i in enumerate(targets):
        d = pos[i] - pos
        r2 = (d * d).sum(1)
        keep = np.arange(len(pos)) != i
        d, r2, w = d[keep], r2[keep], m[keep]
        if dim == 3 and soft == fmmgpu.FMM_SOFT_NAIVE_REF:
            f, p = w / ((r2 + 1e-4) * np.sqrt(r2)), w / np.sqrt(r2)
        elif dim == 3:
            f, p = w / (r2 + eps2) ** 1.5, w / np.sqrt(r2 + eps2)
        else:
            rr = r2 + (1e-4 if soft == fmmgpu.FMM_SOFT_NAIVE_REF else eps2)
            f, p = w / rr, -0.5 * w * np.log(rr)
        acc[k], pot[k] = -(f[:, None] * d).sum(0), p.sum()
    return acc, pot


# 256 sources per stage, 512 targets per block; distances inside and far outside the range of the one-rsqrt form
@pytest.mark.parametrize("soft", [fmmgpu.FMM_SOFT_PLUMMER, fmmgpu.FMM_SOFT_NAIVE_REF])
@pytest.mark.parametrize("n,dim,scale", [(2, 3, 1.0), (255, 3, 1.0), (257, 3, 1.0), (513, 3, 1.0), (1500, 2, 1.0),
                                         (300, 3, 1e-60), (300, 3, 1e60), (130, 2, 1e-3)])
def test_direct_shapes(n, dim, scale, soft):
    rng = np.random.default_rng(n)
    pos, m = rng.random((n, dim)) * scale, rng.random(n)
    targets = np.array([0, n - 1, n // 2])
    a, p = _direct(pos, m, targets, soft, 0.0)
    with fmmgpu.Context(dim=dim) as c:
        some, some_p = c.direct(pos, m, targets=targets, soft_mode=soft, want_pot=True)
        every = c.direct(pos, m, soft_mode=soft)
    assert rel_l2(some, a) < 1e-12
    assert rel_l2(some_p, p) < 1e-12
    assert rel_l2(every[targets], a) < 1e-12


# blocks of 256 targets, full, with idle warps and with idle threads, over one and many shares of the sources (every
# target checked where there are few, else the ends of the blocks)
@pytest.mark.parametrize("n,nt,dim", [(3000, 1, 3), (3000, 33, 3), (3000, 256, 3), (3000, 257, 3), (450000, 385, 3),
                                      (450000, 384, 3), (120000, 1920, 2), (14000, 14000, 3), (15000, 15000, 3)])
@pytest.mark.parametrize("soft", [fmmgpu.FMM_SOFT_PLUMMER, fmmgpu.FMM_SOFT_NAIVE_REF])
def test_direct_target_blocks(n, nt, dim, soft):
    rng = np.random.default_rng(nt)
    pos, m = rng.random((n, dim)), rng.random(n)
    targets = rng.permutation(n)[:nt]
    look = np.unique(np.clip(np.r_[np.arange(0, nt, max(1, nt // 16)), np.arange(0, nt + 1, 256) - 1, nt - 1], 0, nt - 1))
    a, p = _direct(pos, m, targets[look], soft, 0.0)
    with fmmgpu.Context(dim=dim) as c:
        acc, pot = c.direct(pos, m, targets=targets, soft_mode=soft, want_pot=True)
        plain = c.direct(pos, m, targets=targets, soft_mode=soft)
    assert rel_l2(acc[look], a) < 1e-12
    assert rel_l2(pot[look], p) < 1e-12
    assert rel_l2(plain, acc) < 1e-12


def test_direct_of_few_targets_takes_less_than_of_many():
    """One target, 256 and 512 of 2^20 particles: idle threads cost nothing,
    so 256 take at most three quarters of the time of 512, and one at most
    half (the idle halves of blocks of 512 took as long as full ones)."""
    torch = pytest.importorskip("torch")
    n = 1 << 20
    g = torch.Generator(device="cuda").manual_seed(3)
    pos = torch.rand(n, 3, generator=g, device="cuda", dtype=torch.float64)
    mass = torch.full((n,), 1.0 / n, device="cuda", dtype=torch.float64)
    acc = torch.empty(512, 3, device="cuda", dtype=torch.float64)
    stream = torch.cuda.Stream()
    ms = {}
    with fmmgpu.Context(dim=3) as c, torch.cuda.stream(stream):
        for nt in (1, 256, 512):
            times = []
            for _ in range(8):
                e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
                e0.record()
                c.direct_device(n, pos.data_ptr(), mass.data_ptr(), nt, None, acc.data_ptr(), stream=stream.cuda_stream)
                e1.record()
                torch.cuda.synchronize()
                times.append(e0.elapsed_time(e1))
            ms[nt] = min(times)
    assert ms[256] < 0.75 * ms[512]
    assert ms[1] < 0.5 * ms[512]


# NaiveUpdate's softening with masses at which the force turns subnormal or leaves the FP64 range, the potential not
@pytest.mark.parametrize("scale,mass", [(1e40, 1e-200), (1e-44, 2e261)])
def test_direct_potential_beyond_the_force_range(scale, mass):
    rng = np.random.default_rng(2)
    pos, m = rng.random((30, 3)) * scale, (0.5 + rng.random(30)) * mass
    targets = np.arange(30)
    with np.errstate(all="ignore"):
        _, want = _direct(pos, m, targets, fmmgpu.FMM_SOFT_NAIVE_REF, 0.0)
    with fmmgpu.Context(dim=3) as c:
        _, pot = c.direct(pos, m, soft_mode=fmmgpu.FMM_SOFT_NAIVE_REF, want_pot=True)
    unit = mass / scale  # (the norm's squares would leave the range themselves)
    assert rel_l2(pot / unit, want / unit) < 1e-12


@pytest.mark.parametrize("method", [fmmgpu.FMM_INT_SYMPLECTIC_EULER, fmmgpu.FMM_INT_RK4])
@pytest.mark.parametrize("steps", [1, 2, 5])
def test_integrate_reports_nonfinite_forces(method, steps):
    """Coincident particles in the first step's pass: the call reports the
    non-finite output whether or not it waits for every step, and the context
    works on."""
    pos, m = workloads.uniform_cube(400, seed=3)
    bad = pos.copy()
    bad[7] = bad[11]
    with fmmgpu.Context(dim=3, p=4, leaf_cap=16) as c:
        with pytest.raises(fmmgpu.FmmError) as e:
            c.integrate(method, 1e-3, steps, bad, 0 * bad, m)
        want = fmmgpu.FMM_ERR_NONFINITE_OUTPUT if method == fmmgpu.FMM_INT_SYMPLECTIC_EULER else None
        assert e.value.code in (want, fmmgpu.FMM_ERR_NONFINITE_INPUT) if want is None else e.value.code == want
        acc = c.evaluate(pos, m)
        assert np.all(np.isfinite(acc))
        x, v, a = c.integrate(method, 1e-3, steps, pos, 0 * pos, m)
        assert np.all(np.isfinite(x)) and np.all(np.isfinite(a))


def _clump_in_flat_halo(n, sigma, seed=3):
    """Half of the particles uniform in a box of 1 x 1 x 0.5, the first half
    in a Gaussian clump well inside one cell of the coarse levels."""
    rng = np.random.default_rng(seed)
    pos = rng.random((n, 3)) * np.array([1.0, 1.0, 0.5])
    pos[: n // 2] = np.array([0.3, 0.3, 0.15]) + sigma * rng.normal(size=(n // 2, 3))
    return pos, np.full(n, 1.0 / n)


def test_clump_in_flat_halo(oracle):
    """A flattened box whose largest cells hold half of the particles on ten
    levels: with every cell of a level split as the level's largest, the far
    field had 1.83e8 warps, beyond the 2^27 of a 32-bit thread index.  The
    halo's forces, small beside the clump's, are compared on their own."""
    n = 60000
    pos, m = _clump_in_flat_halo(n, 1e-4)
    with fmmgpu.Context(dim=3, p=6, leaf_cap=64, direct_max=128, m2l_mode=fmmgpu.FMM_M2L_TC) as c:
        acc = c.evaluate(pos, m)
    want = oracle.fmm(pos, m, 6, 64, direct_max=128)
    assert rel_l2(acc[n // 2:], want[n // 2:]) < 1e-6
    assert rel_l2(acc[: n // 2], want[: n // 2]) < 1e-6


def test_clump_in_flat_halo_launches_no_empty_warps():
    """The far field of such a box costs what its pairs cost: here at least
    2e11 pairs/s (a fifth of the rate in boxes without a clump) after 1 ms,
    where warps for every cell as for the largest took 37 ms."""
    n = 60000
    pos, m = _clump_in_flat_halo(n, 1e-4)
    with fmmgpu.Context(dim=3, p=8, leaf_cap=64, m2l_mode=fmmgpu.FMM_M2L_TC) as c:
        ms = []
        for _ in range(4):
            c.evaluate(pos, m)
            st = c.stats()
            ms.append(st["ms_far_direct"])
    assert min(ms) < 1.0 + st["far_direct_pairs"] / 2e11 * 1e3


# 64 and 128 targets per warp, lists of one, a few and hundreds of tiles of 2048 cells (p = 8 truncates to 2e-5 to 6e-5
# here, in FP64 as well)
@pytest.mark.parametrize("n,adaptive", [((1 << 17) + 1, 0), ((1 << 19) + 1, 0), ((1 << 19) + 1, 32)])
def test_flattened_sphere_against_direct(oracle, n, adaptive):
    pos, m = workloads.plummer(n, seed=8)
    pos = pos * np.array([1.0, 1.0, 0.8])
    with fmmgpu.Context(dim=3, p=8, leaf_cap=64, m2l_mode=fmmgpu.FMM_M2L_TC, adaptive_leaf=adaptive) as c:
        acc, pot = c.evaluate(pos, m, want_pot=True)
    some = np.random.default_rng(1).choice(n, 300, replace=False)
    want, want_pot = oracle.direct(pos, m, targets=some, want_pot=True)
    assert rel_l2(acc[some], want) < 1e-4
    assert rel_l2(pot[some], want_pot) < 1e-4


@pytest.mark.parametrize("clump", [0.0, 0.5])
@pytest.mark.parametrize("n", [100, 3000, 9000])
def test_elongated_box_2d(oracle, n, clump):
    rng = np.random.default_rng(n)
    pos = rng.random((n, 2)) * np.array([1.0, 0.4])
    k = int(clump * n)
    pos[:k] = np.array([0.3, 0.12]) + 1e-3 * rng.normal(size=(k, 2))
    m = np.full(n, 1.0 / n)
    with fmmgpu.Context(dim=2, p=10, leaf_cap=16, direct_max=64, m2l_mode=fmmgpu.FMM_M2L_TC) as c:
        acc, pot = c.evaluate(pos, m, want_pot=True)
    want, want_pot = oracle.fmm(pos, m, 10, 16, direct_max=64, want_pot=True)
    assert rel_l2(acc[k:], want[k:]) < 1e-6
    assert rel_l2(acc, want) < 1e-6
    assert rel_l2(pot, want_pot) < 1e-6
