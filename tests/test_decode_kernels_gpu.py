"""GPU: small batches, whose bricks several CTAs decode together, against the same requests one CTA each."""
import numpy as np
import pytest

from conftest import read_golden
from test_index_sidecar_gpu import patch_nsym

pytestmark = pytest.mark.gpu


def decode(codec, ds, bricks, lods, skew: int, alone: bool):
    """Labels and statuses; `alone`: at one CTA per SM, which keeps a request to its CTA."""
    import torch
    from csvb200 import DecodeConfig, requests, requests_tensor
    sizes = 8 ** lods.astype(np.uint64)
    dst = np.concatenate([[0], np.cumsum(sizes + np.uint64(skew))[:-1]]).astype(np.uint64) + np.uint64(skew)
    out = torch.full((int((sizes + np.uint64(skew)).sum()) + 1,), -7, dtype=torch.int64, device="cuda")
    st = torch.full((len(bricks),), -1, dtype=torch.int32, device="cuda")
    reqs = requests_tensor(requests(bricks, lods, dst))
    if alone:
        g = codec.decode_graph(ds, reqs, out, st, DecodeConfig(1, 1, 0, 0))
        g.launch()
    else:
        codec.decode_batch(ds, reqs, out, st)
    torch.cuda.synchronize()
    return out.cpu().numpy(), st.cpu().numpy()


def volume(codec, fill: str):
    import torch
    vol = torch.empty((192, 256, 320), dtype=torch.int64, device="cuda")
    if fill == "distinct":  # palettes past 65,535 entries: 32-bit node values
        vol = torch.arange(128 ** 3, dtype=torch.int64, device="cuda").reshape(128, 128, 128).contiguous()
    elif fill == "dense":  # several hundred labels a brick: 16-bit
        codec.synth_volume(vol, 1, 30, 1200, 0.5, 1.5, 0.0, 5)
    else:
        codec.synth_volume(vol, 1, 400, 60, 2.0, 12.0, 0.15, 5)
    return vol


# one request, a few (eight CTAs each), more (four, two) up to about as many as there are SMs; outputs on and off a
# 32-byte boundary; LODs on both sides of the coarsest that is shared
@pytest.mark.parametrize("fill,brick", [("neurite", 64), ("neurite", 32), ("dense", 64), ("dense", 16), ("distinct", 64)])
@pytest.mark.parametrize("n,skew", [(1, 0), (7, 1), (24, 0), (60, 3), (130, 4)])
def test_small_batches_equal_single_ctas(codec, fill, brick, n, skew):
    codec.encode_device(volume(codec, fill), brick)
    ds = codec.open_encoded()
    rng = np.random.default_rng(n)
    top = brick.bit_length() - 1
    bricks = rng.integers(0, ds.num_bricks, n)
    lods = np.where(rng.random(n) < 0.6, top, rng.integers(0, top + 1, n)).astype(np.uint32)
    a, sa = decode(codec, ds, bricks, lods, skew, alone=False)
    b, sb = decode(codec, ds, bricks, lods, skew, alone=True)
    assert sa.max() == 0 and np.array_equal(sa, sb) and np.array_equal(a, b)
    ds.close()


def test_small_batch_statuses(codec):
    """A truncated brick, a missing brick and a LOD that is too fine among good requests: each CTA's part of a status
    is in it, and the others' output is untouched by them."""
    img = read_golden("shipped_subset")
    ds = codec.open(patch_nsym(img, 1, 2000))
    ids = np.array([0, 1, 2, 10 ** 6, 3, 4, 0], np.uint32)
    lods = np.array([6, 6, 6, 6, 9, 5, 2], np.uint32)

    def run(alone):
        import torch
        from csvb200 import DecodeConfig, requests, requests_tensor
        dst = np.arange(len(ids), dtype=np.uint64) << np.uint64(18)
        out = torch.full((len(ids) << 18,), -7, dtype=torch.int64, device="cuda")
        st = torch.full((len(ids),), -1, dtype=torch.int32, device="cuda")
        reqs = requests_tensor(requests(ids, lods, dst))
        if alone:
            codec.decode_graph(ds, reqs, out, st, DecodeConfig(1, 1, 0, 0)).launch()
        else:
            codec.decode_batch(ds, reqs, out, st)
        torch.cuda.synchronize()
        return out.cpu().numpy().reshape(len(ids), -1), st.cpu().numpy()

    a, sa = run(False)
    b, sb = run(True)
    assert np.array_equal(sa, sb)
    good = sa == 0
    assert good.tolist() == [True, False, True, False, False, True, True] and np.array_equal(a[good], b[good])
    ds.close()
