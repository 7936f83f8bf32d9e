"""Data that the trees cannot split below the leaf kernels' limit of 8,192 points
(rows that are all alike, one of NaNs): the build ends with the error that
names the limit, whatever an earlier build left in the workspace, and the next one
is right.  Needs a B200."""
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
