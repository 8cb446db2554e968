"""GPU: the selector network's gradient step and the dense layer's tiles, against the oracle and the layer itself."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _rel(a, b):
    return float(np.linalg.norm(a - b) / max(np.linalg.norm(b), 1e-12))


# one row; a tile and its remainder; one partial bias sum and several; a large batch, then smaller ones in its buffers
@pytest.mark.parametrize("batches", [(1,), (128, 200), (256, 257), (2048,), (8300, 8192, 100)])
def test_gradients_by_batch(codec, oracle, batches):
    import torch
    from csvb200 import SelectorNet
    p = SelectorNet.init_params(len(batches))
    p[-32:-4] = np.linspace(-0.3, 0.3, 28)
    net = SelectorNet(codec, p)
    rng = np.random.default_rng(batches[0])
    for n in batches:
        f = rng.random((n, 32)).astype(np.float32)
        y = (rng.integers(0, 12, n) | rng.integers(0, 16, n) << 4).astype(np.uint8)
        loss = net.grad(torch.from_numpy(f).cuda(), torch.from_numpy(y).cuda())
        _, g = net.params(grads=True)
        ref_loss, ref = oracle.mlp_grad(p, f, y)
        assert abs(loss - ref_loss) <= 1e-3 * abs(ref_loss)
        o = 0
        for name, size in [("W1", 256 * 64), ("b1", 256), ("W2", 256 * 256), ("b2", 256), ("W3", 32 * 256), ("b3", 32)]:
            # bf16 rounding of weights, activations and their gradients: 2^-9 each, three layers deep
            assert _rel(g[o:o + size], ref[o:o + size]) < 2e-2, (n, name)
            o += size
        assert not g[:256 * 64].reshape(256, 64)[:, 32:].any()  # the input's padding has no gradient
    assert net.status() == 0
    net.close()


# column tiles of 64 and their remainders, K below, at and above what a CTA has in flight (three and four chunks of 64);
# outputs that start off a 16-byte boundary
@pytest.mark.parametrize("M,N,K", [(128, 80, 64), (256, 208, 320), (128, 64, 192), (128, 64, 256), (384, 112, 832)])
def test_dense_layer_tiles(codec, M, N, K):
    import torch
    rng = np.random.default_rng(M + N + K)
    A = torch.from_numpy(rng.standard_normal((M, K)).astype(np.float32)).to(torch.bfloat16).cuda()
    B = torch.from_numpy(rng.standard_normal((N, K)).astype(np.float32)).to(torch.bfloat16).cuda()
    ref = A.double().cpu() @ B.double().cpu().T
    # fp32 accumulation of K exact products: K roundings of the running sum at most
    tol = K * 2.0 ** -24 * (A.double().abs().cpu() @ B.double().abs().cpu().T) + 1e-6
    mask = torch.from_numpy(rng.standard_normal(M * N + 8).astype(np.float32)).to(torch.bfloat16).cuda()
    for off in (0, 1):
        C = torch.full((M * N + 8,), float("nan"), device="cuda")
        Cb = torch.zeros(M * N + 8, dtype=torch.bfloat16, device="cuda")
        codec.gemm_bf16(A, B, C=C[off:], Cb=Cb[off:], mask=mask[off:])
        got = C[off:off + M * N].view(M, N).cpu()
        want = ref * (mask[off:off + M * N].view(M, N).float().cpu() > 0)
        assert torch.all((got.double() - want).abs() <= tol)
        assert torch.equal(Cb[off:off + M * N].view(M, N).cpu(), got.to(torch.bfloat16))
        assert torch.isnan(C[off + M * N:]).all()


# a layer in place: the output over the rows it was computed from (all columns are one CTA's), more rows of CTAs than
# run at once, and over the other operand where one CTA reads all of it
@pytest.mark.parametrize("M,N,over", [(128, 64, "A"), (256, 256, "A"), (128 * 700, 256, "A"), (128 * 300, 192, "A"),
                                      (128, 256, "B")])
def test_dense_layer_in_place(codec, M, N, over):
    import torch
    K = N if over == "A" else 128
    g = torch.Generator(device="cuda")
    g.manual_seed(M + N)
    A = torch.randn((M, K), device="cuda", generator=g).to(torch.bfloat16)
    B = torch.randn((N, K), device="cuda", generator=g).to(torch.bfloat16)
    want = torch.empty((M, N), dtype=torch.bfloat16, device="cuda")
    codec.gemm_bf16(A, B, relu=True, Cb=want)
    # the sums' order does not depend on the tile: bit for bit the output beside the operands
    if over == "A":
        codec.gemm_bf16(A, B, relu=True, Cb=A)
        assert torch.equal(A, want)
    else:
        codec.gemm_bf16(A, B, relu=True, CbT=B.view(-1))
        assert torch.equal(B.view(-1).view(N, M), want.T)


# a warp per brick: its block not full, one table to all sixteen, and ties between equal tables and equal modes
@pytest.mark.parametrize("bricks", [1, 4, 9])
@pytest.mark.parametrize("n_tables", [1, 3, 16])
def test_exhaustive_choice(codec, oracle, bricks, n_tables):
    import torch
    rng = np.random.default_rng(bricks * 16 + n_tables)
    hist = rng.integers(0, 1 << 18, (bricks, 12, 16)).astype(np.uint32)
    hist[0, 5:] = hist[0, 5]
    hist[-1, :, 3:] = 0
    tables = np.full((n_tables, 16), 1, np.uint32)
    for t in range(n_tables):
        tables[t, rng.integers(0, 16)] += 4096 - 16
    d = torch.from_numpy(hist.view(np.int32)).cuda()
    sel = torch.zeros(bricks, dtype=torch.uint8, device="cuda")
    cost = torch.zeros(bricks * 12 * n_tables, dtype=torch.int64, device="cuda")
    codec.select_exhaustive(d, tables, sel, cost)
    want, want_cost = oracle.select_exhaustive(hist, tables)
    assert np.array_equal(sel.cpu().numpy(), want)
    assert np.array_equal(cost.cpu().numpy().view(np.uint64), np.asarray(want_cost).reshape(-1))
