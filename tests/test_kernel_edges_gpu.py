"""Edges of the kernels' tiles and branches, against the oracle or the FP64
path: row counts around the tile sizes, every l count, orbital l of 0..3,
projection slices, bands and row blocks that fill no tile."""
import numpy as np
import pytest
import torch

from hack_wein2k_b200 import forces as FO
from hack_wein2k_b200 import lapw1gpu, synth
from oracle import oracle as O
from tests import force_ref as FR
from tests.helpers import rel_errors

TOL_FP64 = 1e-12
# the slice counts' bounds of tests/test_split_gpu.py
TOL_SPLIT = {4: 2e-7, 5: 2e-9, 6: 2e-11, 7: 1e-12}

pytestmark = pytest.mark.gpu


def _rows(p, nv):
    """The problem's first nv plane waves (no local orbitals)."""
    assert p.nlo == 0 and nv <= p.nv
    return p.copy(nv=nv, kzz=p.kzz[:nv], xk=p.xk[:nv], yk=p.yk[:nv], zk=p.zk[:nv], rk=p.rk[:nv])


def _plain(rkmax, k=(0.13, 0.27, 0.41), lmax=10, **kw):
    return synth.synth_problem(synth.cell_small_mixed(), rkmax, k, seed=11, lmax=lmax, **kw)


def _check(ctx, p, tol):
    hs, hsd = ctx.setup(p)
    err = rel_errors(hs, hsd, *O.setup(p))
    assert err["H"] <= tol and err["S"] <= tol, (p.n, err)


# 32- and 64-row tiles of k_spherical and k_tri_gemm; 1537 rows take the
# 64-wide product tiles (25 tile rows, 325 tiles: at least two per SM), 1472
# (23, 276) the 32-wide ones
@pytest.mark.parametrize("nv", [1, 31, 32, 33, 63, 64, 65, 97, 1472, 1537])
def test_fp64_row_counts(ctx, nv):
    ctx.set_precision(lapw1gpu.PREC_FP64)
    _check(ctx, _rows(_plain(6.0 if nv < 200 else 13.5), nv), TOL_FP64)


@pytest.mark.parametrize("lmax", [4, 9, 10, 12])
@pytest.mark.parametrize("lnsmax", [0, 2, 4])
def test_fp64_l_counts(ctx, lmax, lnsmax):
    """k_spherical with fewer and more l than its unrolled count, the HNS
    operand product with 2, 18 and 50 rows, LO rows on every atom."""
    ctx.set_precision(lapw1gpu.PREC_FP64)
    _check(ctx, _plain(5.0, lmax=lmax, lnsmax=lnsmax, lo_l=(0, 1, 2), rotate_local=True), TOL_FP64)


@pytest.mark.parametrize("slices", [4, 5, 6, 7])
@pytest.mark.parametrize("lmax", [4, 10, 12])
def test_split_row_counts(ctx, slices, lmax):
    """k_sph_tc at the edges of its 12- and 8-I and 128-J tiles: an element
    depends on its two rows only (scales are per row, the level sums exact), so
    the first nv rows alone give the bits they have in the whole problem,
    which is within the slices' bound of the oracle.  k along an axis puts many
    pairs on one line (the x P_(l-1) branch)."""
    full = _plain(6.0, k=(0.0, 0.0, 0.3), lmax=lmax)
    ctx.set_precision(lapw1gpu.PREC_SPLIT, slices)
    try:
        hs, hsd = ctx.setup(full, stages=1)
        err = rel_errors(hs, hsd, *O.setup(full, stages=1))
        assert err["H"] <= TOL_SPLIT[slices] and err["S"] <= TOL_SPLIT[slices], err
        for nv in (1, 7, 8, 9, 11, 12, 13, 127, 128, 129):
            h, d = ctx.setup(_rows(full, nv), stages=1)
            assert np.array_equal(h, hs[:nv, :nv]) and np.array_equal(d, hsd[:nv]), nv
    finally:
        ctx.set_precision(lapw1gpu.PREC_FP64)


@pytest.mark.parametrize("prec,tol", [(lapw1gpu.PREC_FP64, TOL_FP64), (lapw1gpu.PREC_SPLIT, TOL_SPLIT[7])])
@pytest.mark.parametrize("orb", [((1, (0,)),), ((1, (3, 1)), (2, (0, 2, 3)))])
def test_orbital_l(ctx, prec, tol, orb):
    ctx.set_precision(prec, 7)
    try:
        _check(ctx, _plain(5.0, lo_l=(0, 2), apw_l=(1,), rotate_local=True, orb=orb), tol)
    finally:
        ctx.set_precision(lapw1gpu.PREC_FP64)


@pytest.fixture(scope="module")
def many_lo():
    """17 equivalent atoms of one type and five one-atom types, local orbitals
    on all: k_lo and k_force_lo hold the Y_lm of eight atoms at a time."""
    return synth.synth_problem(synth.cell_many_equiv(), 2.2, (0.13, 0.27, 0.41), seed=7, lo_l=(0, 1), rotate_local=True)


@pytest.mark.parametrize("prec,tol", [(lapw1gpu.PREC_FP64, TOL_FP64), (lapw1gpu.PREC_SPLIT, TOL_SPLIT[7])])
@pytest.mark.parametrize("orb", [False, True])
def test_local_orbitals_of_many_equivalent_atoms(ctx, many_lo, prec, tol, orb):
    p = many_lo if not orb else synth.synth_problem(synth.cell_many_equiv(), 2.2, (0.13, 0.27, 0.41), seed=7,
                                                    lo_l=(0, 2), rotate_local=True, orb=((1, (2,)), (3, (0, 1))))
    ctx.set_precision(prec, 7)
    try:
        _check(ctx, p, tol)
    finally:
        ctx.set_precision(lapw1gpu.PREC_FP64)


def test_local_orbital_forces_of_many_equivalent_atoms(ctx, many_lo):
    """Atoms of the first, second and third eight of the type, and one of
    another type, against the oracle's Hellmann-Feynman sum."""
    p = many_lo
    w, _ = FR.eigh(p)
    nb, _ = FR.gapped_nb(w)
    atoms = (0, 9, 16, 21)
    ref = FR.hf_gradient(p, nb, atoms=atoms)
    occ = torch.ones(nb, dtype=torch.float64, device=torch.device("cuda", ctx.device))
    ctx.set_precision(lapw1gpu.PREC_FP64)
    _, eps, X, kp = FO.band_energy(ctx, p, occ)
    g = FO.gradient(ctx, kp, X, occ, eps).cpu().numpy()
    kp.free()
    assert np.abs(g - ref)[list(atoms)].max() <= 1e-8 * np.abs(ref).max()


# bands around a tile of 40 (32 at 7 and 8 slices), blocks whose last rows
# fill no K block of 64
@pytest.mark.parametrize("slices,nb,block,lmax", [(4, 40, 64, 10), (5, 1, 96, 8), (6, 41, 64, 12), (6, 39, 160, 10),
                                                  (7, 33, 64, 9), (8, 31, 128, 10)])
def test_projection_tiles(ctx, slices, nb, block, lmax):
    """The projections against the FP64 adjoint of the same vectors.  The
    slices leave (S+1) 2^(-7S) of the largest terms, whose sum over some
    hundred rows exceeds the result by less than 64; 1e-9 for pairs that the
    pair kernel takes as parallel."""
    p = _plain(7.0, lmax=lmax, lo_l=(0, 1), rotate_local=True)
    assert p.nv > 2 * block
    rng = np.random.default_rng(5)
    dev = torch.device("cuda", ctx.device)
    c = torch.from_numpy(rng.standard_normal((nb, p.n)) + 1j * rng.standard_normal((nb, p.n))).to(dev)
    eps = torch.from_numpy(np.sort(rng.uniform(-1.0, 1.0, nb))).to(dev)
    occ = torch.from_numpy(rng.uniform(0.0, 2.0, nb)).to(dev)
    kp = ctx.upload(p)
    out = []
    try:
        for prec in (lapw1gpu.PREC_FP64, lapw1gpu.PREC_SPLIT):
            ctx.set_precision(prec, 7)
            ctx.set_force_slices(8, 8)
            ctx.set_force_projection(slices, block)
            g = torch.empty((p.ndf, 3), dtype=torch.float64, device=dev)
            kp.forces(c.data_ptr(), p.n, nb, occ.data_ptr(), eps.data_ptr(), g.data_ptr())
            out.append(g.cpu().numpy())
    finally:
        kp.free()
        ctx.set_precision(lapw1gpu.PREC_FP64)
        ctx.set_force_slices(6, 6)
        ctx.set_force_projection(-1, 1024)
    assert np.abs(out[1] - out[0]).max() <= (64 * (slices + 1) * 2.0 ** (-7 * slices) + 1e-9) * np.abs(out[0]).max()


@pytest.mark.parametrize("slices,nb", [(6, 41), (7, 33)])
def test_projection_chunks_of_atoms(ctx, slices, nb):
    """Operands of a few atoms at a time: chunks of one atom, chunks that end
    inside the type of 17 atoms and span several types, and a budget of which
    less and less fits.  An atom's sums do not depend on its chunk, so the
    gradient is the single chunk's up to the order of the atomic sums.  What
    does not fit at all is an error that leaves the context usable."""
    p = synth.small_case("manyeq", rkmax=2.5)
    block, nband = 64, (40 if slices == 6 else 32)
    nblk = -(-p.nv // block)
    assert nblk > 2 and p.ndf == 22
    types = np.repeat(np.arange(p.nat), p.mult)
    kp_bytes = nblk * block  # one operand row
    type_bytes = slices * -(-p.ltop ** 2 // 16) * 128 * kp_bytes
    atom_bytes = slices * 2 * -(-nb // nband) * nband * kp_bytes
    rng = np.random.default_rng(5)
    dev = torch.device("cuda", ctx.device)
    c = torch.from_numpy(rng.standard_normal((nb, p.n)) + 1j * rng.standard_normal((nb, p.n))).to(dev)
    eps = torch.from_numpy(np.sort(rng.uniform(-1.0, 1.0, nb))).to(dev)
    occ = torch.from_numpy(rng.uniform(0.0, 2.0, nb)).to(dev)
    g = torch.empty((p.ndf, 3), dtype=torch.float64, device=dev)
    kp = ctx.upload(p)

    def gradient(budget, fit=0):
        ctx.test_projection_bytes(budget, fit)
        g.fill_(np.nan)
        torch.cuda.synchronize()
        kp.forces(c.data_ptr(), p.n, nb, occ.data_ptr(), eps.data_ptr(), g.data_ptr())
        return g.cpu().numpy(), ctx.last_launches()

    try:
        ctx.set_precision(lapw1gpu.PREC_SPLIT, 5)
        ctx.set_force_projection(slices, block)
        ref, launches = gradient(0)
        exps = 4 * 2 * -(-p.ltop ** 2 // 16) * 128 * nblk
        for budget in (1, type_bytes + 5 * atom_bytes, 2 * type_bytes + 8 * atom_bytes):
            n, a0, a1 = 0, 0, 0  # the chunks' count
            while a1 < p.ndf:
                n, a0, a1 = n + 1, a1, a1 + 1
                while a1 < p.ndf and (types[a1] - types[a0] + 1) * type_bytes + (a1 + 1 - a0) * atom_bytes <= budget:
                    a1 += 1
            # (twice: with no more room than the budget and the exponents of two types)
            for fit in (0, max(budget, type_bytes + atom_bytes) + exps):
                out, nl = gradient(budget, fit)
                assert np.abs(out - ref).max() <= 1e-12 * np.abs(ref).max(), budget
                assert n > 3 and nl == launches + 3 * (n - 1), (budget, n, nl - launches)
        out, nl = gradient(0, 2 * type_bytes + 8 * atom_bytes + exps)
        assert np.abs(out - ref).max() <= 1e-12 * np.abs(ref).max() and nl > launches
        with pytest.raises(lapw1gpu.Lapw1GpuError) as e:
            gradient(0, atom_bytes)
        assert e.value.code == 2  # LAPW1GPU_ERR_NOMEM
        out, nl = gradient(0)
        assert np.abs(out - ref).max() <= 1e-12 * np.abs(ref).max() and nl == launches
    finally:
        ctx.test_projection_bytes()
        ctx.set_force_projection(-1, 1024)
        ctx.set_precision(lapw1gpu.PREC_FP64)
        kp.free()


@pytest.mark.parametrize("pin", [False, True])
def test_upload_is_done_with_the_callers_arrays(ctx, pin):
    """Arrays of up to 256 KiB go through the context's staging buffer, longer
    ones (the T blocks of six types and of four, 540 and 360 KB) straight from
    the caller's memory, page-locked or not.  Once upload returns, the caller
    may overwrite either: the k-points still give what they held, also after
    another upload has used the staging buffer."""
    dev = torch.device("cuda", ctx.device)
    ctx.set_precision(lapw1gpu.PREC_FP64)
    four = synth.Cell("P", (12.0, 12.0, 12.0), (90.0, 90.0, 90.0),
                      [dict(pos=[[0.25 * q, 0.3 * q, 0.2 * q]], rmt=1.2) for q in range(4)])
    probs = [synth.small_case("manyeq", rkmax=2.5), synth.synth_problem(four, 2.6, (0.1, 0.2, 0.3), seed=4)]
    want = [ctx.setup(p) for p in probs]
    kps = []
    for p in probs:
        mine = {}
        for name in ("tns", "warp", "kzz", "xk", "p", "pos"):
            a = np.ascontiguousarray(getattr(p, name))
            t = torch.empty(a.nbytes, dtype=torch.uint8, pin_memory=pin)
            mine[name] = t.numpy().view(a.dtype).reshape(a.shape)
            mine[name][...] = a
        assert mine["tns"].nbytes > 256 << 10 > mine["xk"].nbytes
        kps.append(ctx.upload(p.copy(**mine)))
        for a in mine.values():
            a.view(np.uint8)[...] = 0xff  # NaN, or -1
    for p, kp, (hs, hd) in zip(probs, kps, want):
        d_hs = torch.empty((p.n, p.n), dtype=torch.complex128, device=dev)
        d_hd = torch.empty(p.n, dtype=torch.complex128, device=dev)
        kp.run(d_hs.data_ptr(), p.n, d_hd.data_ptr(), stats=True)
        assert np.array_equal(d_hs.cpu().numpy().T, hs) and np.array_equal(d_hd.cpu().numpy(), hd)
        kp.free()


@pytest.mark.parametrize("prec", [lapw1gpu.PREC_FP64, lapw1gpu.PREC_SPLIT])
@pytest.mark.parametrize("blk", [2, 5, 6, 7, 8])
@pytest.mark.parametrize("value", [np.nan, np.inf])
def test_nonfinite_t_entry_of_an_absent_l(ctx, prec, blk, value):
    """An entry of the local orbitals' T blocks at an l without local orbitals
    meets zero coefficients only, which make the sums NaN as they stand: the
    setup reports it."""
    p = _plain(5.0, lo_l=(0,))
    tns = np.array(p.tns, copy=True)
    tns[p.nat - 1, blk, 3, 7] = value  # l = 1, l' = 2
    ctx.set_precision(prec, 5)
    try:
        with pytest.raises(lapw1gpu.Lapw1GpuError) as ei:
            ctx.setup(p.copy(tns=tns))
        assert ei.value.code == 4
        ctx.setup(p)
    finally:
        ctx.set_precision(lapw1gpu.PREC_FP64)


# one writer of HS each: k_spherical, k_lo, the HNS product
@pytest.mark.parametrize("field,lo,stages", [("e", (), 1), ("alo", (0, 1), 1), ("tns", (), 3)])
@pytest.mark.parametrize("value", [np.nan, np.inf])
def test_fp64_writers_report_nonfinite(ctx, field, lo, stages, value):
    ctx.set_precision(lapw1gpu.PREC_FP64)
    p = _plain(5.0, lo_l=lo)
    a = np.array(getattr(p, field), copy=True)
    if field == "alo":  # every local orbital's coefficient
        a[...] = value
    else:
        a.flat[0] = value
    with pytest.raises(lapw1gpu.Lapw1GpuError) as ei:
        ctx.setup(p.copy(**{field: a}), stages=stages)
    assert ei.value.code == 4
    ctx.setup(p, stages=stages)
