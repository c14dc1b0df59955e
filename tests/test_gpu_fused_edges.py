"""The fused tensor-core kernel where its tiles, groups and stages end: odd and
even numbers of tile rows (a pair's second CTA without a tile), groups of eight
columns that straddle the diagonal or the last column, every way row entries
are stored (strides and bases that take 32-byte, 16-byte and no vectors), odd
numbers of 256-column blocks, rows without a valid site, identical rows.  Every
value must be the oracle's within the float parity rule of test_gpu_parity.py.
"""
import numpy as np
import pytest

from oracle import oracle
from rapidnj_b200 import synth

from test_gpu_parity import assert_matrix_parity

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


def alignment(typ, n, L, seed):
    s = (synth.tree_dna if typ == 0 else synth.tree_protein)(n, L, seed=seed)
    if n > 4:
        s[n // 2] = ord("-")          # no valid site with anything
        s[n - 1] = s[0]               # identical rows
        s[1] = (synth.iid_dna if typ == 0 else synth.iid_protein)(1, L, seed=seed)[0]  # saturated
    return s


CASES = [(0, "kim"), (0, "jc"), (1, "kim"), (1, "jc")]


@pytest.mark.parametrize("typ,model", CASES)
@pytest.mark.parametrize("n,L", [(7, 300), (120, 255), (136, 513), (255, 257), (257, 1025),
                                 (385, 90), (521, 770)])
@pytest.mark.parametrize("pad,shift", [(0, 0), (1, 0), (4, 0), (8, 0), (8, 1), (8, 4)])
def test_tile_and_store_edges(ctx, typ, model, n, L, pad, shift):
    if pad and n not in (136, 521):
        pytest.skip("one small and one large size for every store form")
    s = alignment(typ, n, L, seed=n + L)
    ld = (n + 7) // 8 * 8 + pad if pad else n
    buf = torch.full((n * ld + shift,), -7.0, dtype=torch.float32, device="cuda")
    out = buf[shift:].view(n, ld)
    aln = ctx.alignment(s, typ)
    mx = ctx.distance_into(aln, model, out, want_max=True)
    got = out[:, :n].cpu().numpy()
    ref, want = oracle.matrix(oracle.counts(s, typ), L, typ, 0 if model == "jc" else 1)
    assert_matrix_parity(got, ref)
    assert abs(mx - want) <= 1e-6 * max(1.0, want)
    if ld > n:  # nothing outside the matrix is written
        assert bool((out[:, n:] == -7.0).all()) and bool((buf[:shift] == -7.0).all())


@pytest.mark.parametrize("depth", [2, 3, 4, 5, 6])
def test_ring_depths(ctx, depth):
    from rapidnj_b200 import api
    s = synth.tree_dna(400, 1700, seed=depth)
    want = ctx.distance(ctx.alignment(s, 0), "kim").to_numpy()
    api.tune_set(400, 1700, "dna", tc_stages=depth)
    try:
        got = ctx.distance(ctx.alignment(s, 0), "kim").to_numpy()
    finally:
        api.tune_clear()
    assert np.array_equal(got.view(np.int32), want.view(np.int32))


def test_batch_of_every_variant(ctx):
    # DNA and protein, both models and the wrapping valid count in one batch: each
    # equals its plain call bit for bit.
    from rapidnj_b200 import api
    b = api.Batch(ctx, max_alignments=16, max_tiles=4096)
    want, slots = [], []
    for k, (n, L) in enumerate([(130, 400), (257, 128), (300, 640), (64, 256), (511, 900)]):
        for typ in (0, 1):
            s = alignment(typ, n, L, seed=31 * k + typ)
            model = "jc" if k % 2 else "kim"
            a = ctx.alignment(s, typ, compat_wrap=k == 1)
            want.append(ctx.distance(a, model).to_numpy())
            slots.append(b.add(a, model))
    b.run()
    b.synchronize()
    for w, slot in zip(want, slots):
        assert np.array_equal(b.take(slot).to_numpy().view(np.int32), w.view(np.int32))
    b.close()


@pytest.mark.parametrize("typ,model,wrap", [(0, "kim", False), (0, "jc", False), (1, "kim", False),
                                            (1, "jc", False), (1, "kim", True)])
@pytest.mark.parametrize("n", [2, 129, 897, 1025, 1409, 1700])
def test_column_slices(ctx, typ, model, wrap, n):
    """Plain calls around the sizes at which their tiles are split into column slices
    against the batch's whole tiles: bit for bit, the maximum too."""
    from rapidnj_b200 import api
    s = alignment(typ, n, 640, seed=n + typ)
    a = ctx.alignment(s, typ, compat_wrap=wrap)
    out = torch.full((n, n + 3), -7.0, dtype=torch.float32, device="cuda")
    mx = ctx.distance_into(a, model, out, want_max=True)
    with_batch = api.Batch(ctx, max_alignments=1, max_tiles=4096)
    slot = with_batch.add(a, model)
    with_batch.run()
    want = with_batch.take(slot).to_numpy()
    assert np.array_equal(out[:, :n].cpu().numpy().view(np.int32), want.view(np.int32))
    assert np.float32(mx) == np.float32(with_batch.max(slot))
    assert bool((out[:, n:] == -7.0).all())


@pytest.mark.parametrize("residues", [1, 2, 3, 4, 9])
@pytest.mark.parametrize("L", [100, 600])
@pytest.mark.parametrize("depth", [0, 3])
def test_fewer_and_more_stages_than_the_ring(ctx, residues, L, depth):
    """1 + residues feature blocks of one or two stages each, from half a ring to
    several rounds of it, with one and several items a pair of CTAs."""
    from rapidnj_b200 import api
    letters = np.frombuffer(b"ARNDCQEGH", np.uint8)[:residues]
    rng = np.random.default_rng(residues + L)
    for n in (5, 300, 2300):
        s = letters[rng.integers(0, residues, (n, L))]
        s[rng.random((n, L)) < 0.05] = ord("-")
        if depth:
            api.tune_set(n, L, "protein", tc_stages=depth)
        try:
            fused = ctx.distance(ctx.alignment(s, 1), "kim")
            got, mx = fused.to_numpy(), fused.max
        finally:
            api.tune_clear()
        planes = ctx.distance(ctx.alignment(s, 1, popcount=True), "kim")
        assert np.array_equal(got.view(np.int32), planes.to_numpy().view(np.int32))
        assert mx == planes.max
