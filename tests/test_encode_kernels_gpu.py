"""GPU: the encoder's kernels at the sizes where they can go wrong, against the oracle's bytes."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _volume(shape, seed, labels=40):
    """Blobs of a few labels with single voxels of others scattered in: every op, short and long palettes."""
    rng = np.random.default_rng(seed)
    c = [np.arange(n) // 5 for n in shape]
    ids = rng.integers(1, 2 ** 63, labels, dtype=np.uint64)
    vol = ids[(c[0][:, None, None] * 7 + c[1][None, :, None] * 3 + c[2][None, None, :]) % (labels // 3)]
    at = rng.random(shape) < 0.03
    vol[at] = ids[rng.integers(0, labels, int(at.sum()))]
    return vol


def _tables(common):
    """Frequencies with `common` in the places of ops that occur often: symbols that take one, two or three steps."""
    t = np.full((len(common), 16), 3, np.uint32)
    for k, f in enumerate(common):
        t[k, [1, 3, 6, 9]] = f
        t[k, 15] = 1
        t[k, 0] += 4096 - t[k].sum()
    return t


# bricks: one chain per block, four, eight (the last block not full), and whole 64^3 bricks
@pytest.mark.parametrize("shape,brick", [((8, 8, 8), 8), ((64, 64, 72), 8), ((80, 104, 104), 8), ((113, 128, 128), 8),
                                         ((64, 64, 70), 64)])
def test_rans_steps_and_checkpoints(codec, oracle, shape, brick):
    import torch
    from csvb200 import requests, requests_tensor
    vol = _volume(shape, sum(shape))
    d = torch.from_numpy(vol.view(np.int64)).cuda()
    tables = _tables([1, 2, 15, 16, 900])
    nb = int(np.prod([-(-n // brick) for n in shape]))
    sel = np.random.default_rng(nb).integers(0, len(tables), nb).astype(np.uint8) << 4
    n = codec.encode_device_sel(d, brick, tables, torch.from_numpy(sel).cuda())
    img = bytes(codec.encoded_image_tensor().cpu().numpy())
    assert len(img) == n and img == oracle.encode_sel(vol, brick, sel, tables)
    # the encoder's own seek index: every brick at full resolution
    ds, lod = codec.open_encoded(), brick.bit_length() - 1
    out = torch.zeros(nb * brick ** 3, dtype=torch.int64, device="cuda")
    st = torch.zeros(nb, dtype=torch.int32, device="cuda")
    dst = np.arange(nb, dtype=np.uint64) * brick ** 3
    codec.decode_batch(ds, requests_tensor(requests(np.arange(nb), np.full(nb, lod), dst)), out, st)
    assert int(st.abs().max()) == 0
    ref, _ = oracle.decode_image(oracle.encode(vol, brick), lod)
    assert np.array_equal(out.cpu().numpy().view(np.uint64), ref.ravel())
    ds.close()
