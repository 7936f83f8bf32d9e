"""A captured batch replayed after another batch of the same context has run.
Needs a B200."""
import numpy as np
import pytest

from drpt_b200 import build_graph_batched, synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mode", ["mixed", "fp32_leaf"])
def test_replay_after_another_batch(mode):
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    X = torch.from_numpy(synth.clustered_f32(12_000, 48, n_clusters=12, seed=3)).cuda()
    out = (torch.empty((12_000, 10), dtype=torch.int32, device="cuda"),
           torch.empty((12_000, 10), device="cuda"))

    def captured():
        out[0].fill_(-9)
        out[1].fill_(-9.0)
        build_graph_batched(X, np.array([0, 3_000, 5_000, 12_000]), 4, 10, 7, mode=mode,
                            leaf_size=256, use_graph=True, out=out)
        return out[0].clone(), out[1].clone()

    want = captured()
    small = X[:6_000].contiguous()  # no larger than the captured one in anything
    for offs in ([0, 2_000, 4_500, 6_000], [0, 6_000]):
        got = captured()
        assert torch.equal(got[0], want[0]) and torch.equal(got[1], want[1])
        build_graph_batched(small, np.array(offs), 4, 10, 8, mode=mode, leaf_size=256)
    got = captured()
    assert torch.equal(got[0], want[0]) and torch.equal(got[1], want[1])
