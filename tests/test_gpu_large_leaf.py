"""Data at the leaf kernels' limits.  Rows that the trees cannot split below 8,192
points (all alike, one of NaNs): the build ends with the error that names the limit,
whatever an earlier build left in the workspace, and the next one is right.  Rows so
far out that their scores overflow: no list names what is no row.  Needs a B200."""
import numpy as np
import pytest

from drpt_b200 import DrptError, build_graph, build_graph_batched, synth

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def torch():
    import torch as _t
    if not _t.cuda.is_available():
        pytest.skip("no CUDA device")
    return _t


@pytest.mark.parametrize("kw", [dict(mode="mixed"), dict(mode="mixed", precision="fp8"),
                                dict(mode="fp32_gram")])
@pytest.mark.parametrize("nn", [10, 20])
@pytest.mark.parametrize("data", ["alike", "half alike", "nan"])
def test_leaf_beyond_the_limit(torch, kw, nn, data):
    big = torch.from_numpy(synth.clustered_f32(40_000, 64, n_clusters=40, seed=1)).cuda()
    want = build_graph(big, 3, nn, 5, leaf_size=512, **kw)[:2]  # ids up to 39,999 in the lists
    X = torch.from_numpy(synth.clustered_f32(12_000, 64, n_clusters=12, seed=2)).cuda()
    if data == "nan":
        X[7_000] = float("nan")  # in every projected column, so in every median
    else:
        X[:9_000 if data == "half alike" else 12_000] = X[0].clone()
    with pytest.raises(DrptError) as e:
        build_graph(X, 3, nn, 5, leaf_size=512, **kw)
    torch.cuda.synchronize()
    assert e.value.status == 8 and "8192" in str(e.value)
    if kw["mode"] == "mixed":
        with pytest.raises(DrptError) as e:
            build_graph_batched(torch.cat([big[:3_000], X]), np.array([0, 3_000, 15_000]), 3, nn,
                                5, leaf_size=512, precision=kw.get("precision", "bf16"))
        torch.cuda.synchronize()
        assert e.value.status == 8
    got = build_graph(big, 3, nn, 5, leaf_size=512, **kw)[:2]
    assert torch.equal(got[0], want[0]) and torch.equal(got[1], want[1])


@pytest.mark.parametrize("kw", [dict(mode="mixed"), dict(mode="mixed", precision="fp8"),
                                dict(mode="fp32_gram")])
@pytest.mark.parametrize("nn", [10, 20])
@pytest.mark.parametrize("d", [64, 104])
def test_rows_whose_products_overflow(torch, kw, nn, d):
    # two rows so far out that their products with the others are infinite: their
    # scores are -inf or NaN.  The other rows' lists are those without them.
    r = np.random.default_rng(d + nn)
    X = (r.standard_normal((3_002, d)) * 1e7).astype(np.float32)
    X[3_000:] = np.where(r.random((2, d)) < 0.5, -1e30, 1e30)
    X = torch.from_numpy(X).cuda()
    want = build_graph(X[:3_000].contiguous(), 2, nn, 5, leaf_size=4096, **kw)[:2]
    idx, dist = build_graph(X, 2, nn, 5, leaf_size=4096, **kw)[:2]
    assert torch.equal(idx[:3_000], want[0]) and torch.equal(dist[:3_000], want[1])
    assert ((idx[3_000:] >= -1) & (idx[3_000:] < 3_002)).all()
