"""GPU: the seek index's serial chain pass on streams of every length and end, against the oracle's chain."""
import struct

import numpy as np
import pytest

from test_index_sidecar_gpu import SEED, decode_all, parse_sidecar

pytestmark = pytest.mark.gpu


def image(freq, brick: int, streams, nsyms) -> bytes:
    """A version-1 image of bricks with five palette entries around these streams."""
    cum = np.concatenate([[0], np.cumsum(freq)[:-1]])
    out = [struct.pack("<6I", 0x43534244, 1, len(streams), brick, 16, 4096), np.asarray(freq, np.uint32).tobytes(),
           cum.astype(np.uint32).tobytes()]
    for i, (s, n) in enumerate(zip(streams, nsyms)):
        out.append(struct.pack("<2I", i, 5) + np.arange(1, 6, dtype=np.uint64).tobytes() + struct.pack("<I", len(s)) + s
                   + struct.pack("<I", n))
    return b"".join(out)


# symbols of frequency 1 (two bytes at once), none below 16, and almost one symbol only; few bricks (a lane per warp,
# long streams), and enough that several share a warp
@pytest.mark.parametrize("nb,brick,longest", [(120, 64, 9000), (3700, 16, 600)])
@pytest.mark.parametrize("freq", [(4081,) + (1,) * 15, (256,) * 16, (2689, 347, 104, 651, 46, 201, 10, 31, 5, 1, 1, 1, 2, 3, 1, 3),
                                  (16,) * 13 + (3856, 16, 16)])
def test_chain_of_every_length(codec, oracle, freq, nb, brick, longest):
    assert sum(freq) == 4096
    rng = np.random.default_rng(nb + freq[0])
    cum = np.concatenate([[0], np.cumsum(freq)[:-1]]).astype(np.uint32)
    E = np.concatenate([4 + np.arange(90), rng.integers(4, 4 + longest // 3, nb - 90)])
    ns = np.concatenate([1 + np.arange(70), rng.integers(1, longest, nb - 70)])
    streams = [rng.integers(0, 256, e, dtype=np.uint8).tobytes() for e in E]
    for k in range(0, nb, 3):  # a third start below 2^23, the others as an encoder leaves them
        streams[k] = streams[k][:-1] + b"\0"
    img = image(freq, brick, streams, ns)
    ds = codec.open(img)
    sc = ds.index_sidecar()
    rows, states = parse_sidecar(sc)
    at = 0
    for i in range(nb):
        want = oracle.rans_states(np.asarray(freq, np.uint32), cum, streams[i], int(ns[i]), SEED)
        if rows[i, 2] == 0:  # the root's stop bit: no chain
            x = struct.unpack("<I", streams[i][-4:])[0]
            sym = int(np.searchsorted(cum, x & 4095, side="right")) - 1
            assert sym & 1
            continue
        got = states[at:at + rows[i, 2]]
        assert rows[i, 2] == -(-int(ns[i]) // SEED) and np.array_equal(got, want[:len(got)]), i
        at += rows[i, 2]
    # the symbols: the pieces of a sidecar's chain, stepped in the general form, index the same ops (labels of a brick
    # that reports an error are not defined: its missing ops differ from decode to decode)
    ds2 = codec.open(img, sidecar=sc)
    lod = brick.bit_length() - 1
    a, sa = decode_all(codec, ds, lod)
    b, sb = decode_all(codec, ds2, lod)
    assert np.array_equal(sa, sb) and np.array_equal(a[sa == 0], b[sa == 0])
    ds.close()
    ds2.close()


# chains that end while their ring is being filled (fewer symbols named than the stream holds; four pieces in every four
# groups of 32 symbols), many blocks one after the other on an SM
@pytest.mark.parametrize("nb,longest", [(40, 6000), (4000, 1600)])
def test_chains_that_end_with_copies_on_their_way(codec, oracle, nb, longest):
    freq, cum = (256,) * 16, 256 * np.arange(16, dtype=np.uint32)
    rng = np.random.default_rng(nb)
    ns = rng.integers(600, longest, nb)
    # no stop bit in the root (its symbol is even), a state of an encoder's range
    streams = [rng.integers(0, 256, longest, dtype=np.uint8).tobytes() +
               struct.pack("<I", (1 << 30) | int(rng.integers(0, 8)) << 9) for _ in range(nb)]
    ds = codec.open(image(freq, 16, streams, ns))
    rows, states = parse_sidecar(ds.index_sidecar())
    assert np.array_equal(rows[:, 2], -(-ns // SEED))
    at = 0
    for i in range(nb):
        want = oracle.rans_states(np.asarray(freq, np.uint32), cum, streams[i], int(ns[i]), SEED)
        assert want[-1, 1] > 512 and np.array_equal(states[at:at + rows[i, 2]], want), i
        at += rows[i, 2]
    ds.close()


# images of several tables: few chains of all of them, and so many that the bricks of model 0 too take the form without
# a ring; the states against the oracle's, the labels against the volume
@pytest.mark.parametrize("side,n_tables", [(40, 16), (120, 3), (184, 16)])
def test_chains_of_several_tables(codec, oracle, side, n_tables):
    import torch
    rng = np.random.default_rng(side)
    vol = rng.integers(1, 9, (side // 2,) * 3).repeat(2, 0).repeat(2, 1).repeat(2, 2)
    vol[rng.random(vol.shape) < 0.02] = 77
    d = torch.from_numpy(vol).cuda()
    tables = np.full((n_tables, 16), 16, np.uint32)
    tables[np.arange(n_tables), np.arange(n_tables)] += 4096 - 256
    nb = (side // 8) ** 3
    sel = rng.integers(0, n_tables, nb).astype(np.uint8) << 4
    codec.encode_device_sel(d, 8, tables, torch.from_numpy(sel).cuda())
    img = bytes(codec.encoded_image_tensor().cpu().numpy())
    ds = codec.open(img)
    rows, states = parse_sidecar(ds.index_sidecar())
    at, p = 0, 28 + 128 * n_tables
    for i in range(nb):
        _, s, P = struct.unpack_from("<3I", img, p)
        E, = struct.unpack_from("<I", img, p + 12 + 8 * P)
        stream, ns = img[p + 16 + 8 * P:p + 16 + 8 * P + E], struct.unpack_from("<I", img, p + 16 + 8 * P + E)[0]
        p += 20 + 8 * P + E
        f = tables[s >> 4]
        cum = (np.cumsum(f) - f).astype(np.uint32)
        if rows[i, 2]:
            want = oracle.rans_states(f, cum, stream, ns, SEED)
            assert np.array_equal(states[at:at + rows[i, 2]], want), i
        at += rows[i, 2]
    assert p == len(img)
    got, st = decode_all(codec, ds, 3)
    assert not st.any()
    ref, _ = oracle.decode_image(oracle.encode(vol.view(np.uint64), 8), 3)
    assert np.array_equal(np.asarray(got).reshape(-1).view(np.uint64), ref.reshape(-1).view(np.uint64))
    ds.close()
