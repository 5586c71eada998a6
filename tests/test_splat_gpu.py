"""Splat pass on the device: integer grids bit-exact against the CPU
fixed-point deposit in both modes, and the resolve bit-exact against the FP32
replica, through the C ABI."""
import numpy as np
import pytest

import oracle_ffi as O

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    import gargantua_b200 as g

    c = g.Context()
    yield c
    c.close()


@pytest.fixture(scope="module")
def settled(ctx):
    """A small seeded disk after 200 substeps."""
    import gargantua_b200 as g

    ps = g.Particles(ctx, 60000, seed=1)
    ps.seed_particles()
    ps.step(100)
    return ps


@pytest.mark.parametrize("size", [8, 96])
@pytest.mark.parametrize("exact", [True, False])
def test_integer_grids_are_bit_exact(ctx, settled, size, exact):
    import gargantua_b200 as g

    vol = g.Volume(ctx, size)
    vol.bin(settled, exact=exact, frame=3)
    em, mo, ma = vol.read_sums()
    parts = settled.read()
    rem, rmo, rma = O.deposit32(parts, size, frame=3, exact=exact, seed=1)
    assert ma.sum() > 0
    assert np.array_equal(em, rem)
    assert np.array_equal(mo, rmo)
    assert np.array_equal(ma, rma)
    vol.close()


def test_edge_particles_deposit_like_the_reference(ctx):
    """Particles on the cube faces, just outside, at voxel centres and at the
    low/high clamps (splat.metal:52-70)."""
    import gargantua_b200 as g

    h = 30.0
    pts = np.array([[-h, -h, -h], [h - 1e-4, h - 1e-4, h - 1e-4], [h, 0, 0], [-h - 1e-3, 0, 0], [0, 0, 0],
                    [-h + 60 / 16 * 0.5, 0.1, -0.1], [29.9, -29.9, 0.0], [1.0, 2.0, 3.0]], np.float32)
    n = len(pts)
    parts = np.zeros((n, 8), np.float32)
    parts[:, :3] = pts
    parts[:, 3:6] = [[0.5, -0.25, 0.125]] * n
    parts[:, 6] = np.linspace(1000, 12000, n)
    ps = g.Particles(ctx, n, seed=9)
    ps.write(parts)
    vol = g.Volume(ctx, 16)
    for exact in (True, False):
        vol.clear()
        vol.bin(ps, exact=exact, frame=11)
        em, mo, ma = vol.read_sums()
        rem, rmo, rma = O.deposit32(parts, 16, frame=11, exact=exact, seed=9)
        assert np.array_equal(em, rem) and np.array_equal(mo, rmo) and np.array_equal(ma, rma)


@pytest.mark.parametrize("size", [32, 96, 30, 33])  # whole and partial 32 x 8 blocks
def test_resolve_is_bit_exact_and_clears_the_sums(ctx, settled, size):
    import gargantua_b200 as g

    vol = g.Volume(ctx, size)
    vol.bin(settled, exact=True, frame=0)
    em, mo, ma = vol.read_sums()
    vol.resolve()
    e, v = vol.read()
    bb = ctx.blackbody()[:, :3].copy()
    ref_bb = O.blackbody_table().astype(np.float16).astype(np.float32)
    assert np.array_equal(bb, ref_bb)
    re, rv = O.resolve32(em, mo, ma, size, bb)
    assert np.array_equal(e.view(np.uint16), re.astype(np.float16).view(np.uint16))
    assert np.array_equal(v.view(np.uint16), rv.astype(np.float16).view(np.uint16))
    em2, mo2, ma2 = vol.read_sums()
    assert not em2.any() and not mo2.any() and not ma2.any()


def test_splat_equals_bin_then_resolve_and_is_repeatable(ctx, settled):
    import gargantua_b200 as g

    a = g.Volume(ctx, 24)
    b = g.Volume(ctx, 24)
    a.splat(settled, exact=True)
    b.bin(settled, exact=True, frame=0)
    b.resolve()
    ea, va = a.read()
    eb, vb = b.read()
    assert np.array_equal(ea.view(np.uint16), eb.view(np.uint16))
    assert np.array_equal(va.view(np.uint16), vb.view(np.uint16))
    a.frame = 0
    a.splat(settled, exact=True)  # sums were cleared: same result again
    ea2, _ = a.read()
    assert np.array_equal(ea.view(np.uint16), ea2.view(np.uint16))


def test_size_mismatch_is_an_argument_error(ctx, settled):
    import ctypes as C

    import gargantua_b200 as g
    from gargantua_b200 import _lib

    vol = g.Volume(ctx, 8)
    u = g.splat_uniforms(16, settled.count, 1)
    status = _lib.lib().gg_splat(settled.handle, vol.handle, C.byref(u))
    assert status == 1


SHAPES = [(0, 0), (4, 1024), (8, 64), (8, 1000), (8, 2048), (16, 3), (16, 4096), (16, 100000)]


@pytest.mark.parametrize("shape", SHAPES, ids=[f"edge{e}-chunk{c}" for e, c in SHAPES])
@pytest.mark.parametrize("size", [100, 128])
@pytest.mark.parametrize("exact", [True, False])
def test_every_splat_shape_is_bit_exact(ctx, settled, shape, size, exact):
    """Direct atomics and the brick-privatised deposit (ragged last bricks at
    100^3, many work items per brick at chunk 64, a chunk that is not a power
    of two, and chunk 3: over 20,000 work items taken by the persistent
    deposit blocks) give the replica's grids."""
    import gargantua_b200 as g

    vol = g.Volume(ctx, size)
    vol.set_shape(exact, *shape)
    vol.bin(settled, exact=exact, frame=5)
    em, mo, ma = vol.read_sums()
    rem, rmo, rma = O.deposit32(settled.read(), size, frame=5, exact=exact, seed=1)
    assert ma.sum() > 0
    assert np.array_equal(em, rem) and np.array_equal(mo, rmo) and np.array_equal(ma, rma)
    vol.close()


@pytest.mark.parametrize("exact", [True, False])
def test_crowded_voxels_are_bit_exact(ctx, exact):
    """The max preset's contention case scaled down: 70 % of 400k particles
    seeded from a surface density rising as r^-3 toward the ISCO, settled,
    into 48^3, so hundreds of particles share each inner-disk voxel and the
    deposit's atomics collide on the same words."""
    import gargantua_b200 as g

    ps = g.Particles(ctx, 400_000, seed=7)
    ps.seed_profile(0.7, 3.0)
    ps.advance(50, seed_first=True)
    vol = g.Volume(ctx, 48)
    for edge, chunk in [(8, 4096), (16, 16384), (4, 1024)]:
        vol.set_shape(exact, edge, chunk)
        vol.bin(ps, exact=exact, frame=3)
        em, mo, ma = vol.read_sums()
        vol.clear()
        rem, rmo, rma = O.deposit32(ps.read(), 48, frame=3, exact=exact, seed=7)
        assert ma.max() > 256 * 100  # some voxel holds the mass of over a hundred particles
        assert np.array_equal(em, rem) and np.array_equal(mo, rmo) and np.array_equal(ma, rma), (edge, chunk)
    vol.close()
    ps.close()


@pytest.mark.parametrize("exact", [True, False])
def test_particles_all_outside_leave_the_grid_empty(ctx, exact):
    """No particle inside the cube: the count pass keys none, the scan lists
    no work item, and every brick shape leaves the sums at zero."""
    import gargantua_b200 as g

    n = 5000
    parts = np.zeros((n, 8), np.float32)
    rng = np.random.default_rng(3)
    parts[:, :3] = rng.uniform(31.0, 50.0, (n, 3)).astype(np.float32) * rng.choice([-1.0, 1.0], (n, 3))
    parts[:, 3] = 1.0
    ps = g.Particles(ctx, n, seed=1)
    ps.write(parts)
    vol = g.Volume(ctx, 64)
    for edge, chunk in [(0, 0), (4, 1024), (8, 64), (16, 4096)]:
        vol.set_shape(exact, edge, chunk)
        vol.bin(ps, exact=exact, frame=1)
        em, mo, ma = vol.read_sums()
        assert not em.any() and not mo.any() and not ma.any(), (edge, chunk)
    vol.close()
    ps.close()


def test_shapes_refused_outside_their_limits(ctx):
    import gargantua_b200 as g

    vol = g.Volume(ctx, 256)
    for edge, chunk in [(5, 1024), (8, 0), (4, 1024)]:  # 64^3 bricks of edge 4 exceed the histogram
        with pytest.raises(g.GargantuaError):
            vol.set_shape(True, edge, chunk)
    vol.set_shape(True, 16, 4096)
    vol.close()


def test_autotune_keeps_a_valid_shape_and_zeroed_sums(ctx, settled):
    import gargantua_b200 as g

    vol = g.Volume(ctx, 64)
    edge, chunk, ms = vol.autotune(settled, exact=True)
    assert edge in (0, 4, 8, 16) and ms > 0.0
    em, mo, ma = vol.read_sums()
    assert not em.any() and not mo.any() and not ma.any()
    vol.bin(settled, exact=True, frame=2)
    em, mo, ma = vol.read_sums()
    rem, rmo, rma = O.deposit32(settled.read(), 64, frame=2, exact=True, seed=1)
    assert np.array_equal(em, rem) and np.array_equal(mo, rmo) and np.array_equal(ma, rma)
    vol.close()


@pytest.mark.parametrize("size", [33, 40])
def test_resolve_clears_records_of_any_one_word(ctx, size):
    """A record is cleared whichever single word of it holds something."""
    import gargantua_b200 as g

    n3 = size ** 3
    em, mo, ma = np.zeros(2 * n3, np.uint32), np.zeros(3 * n3, np.int32), np.zeros(n3, np.uint32)
    voxels = np.random.default_rng(size).choice(n3, 60, replace=False)
    for k, v in enumerate(voxels):
        word = k % 6
        if word < 2:
            em[2 * v + word] = 1 + k
        elif word < 5:
            mo[3 * v + word - 2] = -1 - k
        else:
            ma[v] = 0x80000000
    vol = g.Volume(ctx, size)
    vol.write_sums(em, mo, ma)
    vol.resolve()
    assert not any(a.any() for a in vol.read_sums())
    vol.close()
