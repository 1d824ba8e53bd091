"""The forms a GEMM can take (128-row tiles of 32, 64 and 128 columns, K split
over 2, 4 and 8 CTAs, two tiles per SM, persistent tiles, CTA pairs) and the
all-layer kernels of a training step, at their edges.

Tolerances: a sum of K products in FP32 (any order, rounding or truncating)
is within 2 K 2^-24 sum |a b| of the exact one; Adam is the same IEEE FP32
operations as numpy's, so bits. Predictions and gradients: an FP32 sum that
falls on the other side of a rounding boundary moves a stored BF16 value by one
unit, 2^-8 of it; with every value of every layer moved that is 2^-8 per layer
of the forward pass and again of the backward pass."""
import numpy as np
import pytest

import surrogate_oracle as so
from test_gpu_surrogate import rel

pytestmark = pytest.mark.gpu


# one 32-column tile; odd numbers of 64-element column blocks (576, 2624: the
# last pair is half zero fill); splits by 8, 4 and 2; 128-column tiles;
# several waves of two tiles per SM, of persistent tiles and of pairs
@pytest.mark.parametrize("M,N,K", [(128, 128, 64), (640, 128, 576), (128, 256, 2624), (128, 128, 8192),
                                   (128, 2048, 8192), (512, 384, 4096), (768, 1024, 8192), (1024, 2048, 4096),
                                   (2688, 1664, 192), (2432, 4096, 1536), (4096, 4096, 576), (384, 3712, 64)])
def test_gemm_forms(pkg, M, N, K):
    import torch
    g = torch.Generator(device="cuda").manual_seed(M + N + K)
    a = torch.randn(M, K, device="cuda", generator=g).to(torch.bfloat16)
    b = torch.randn(N, K, device="cuda", generator=g).to(torch.bfloat16)
    want = a.double() @ b.double().T
    bound = 2 * K * 2.0 ** -24 * (a.double().abs() @ b.double().abs().T)
    out = []
    for _ in range(2):
        c = torch.full((M, N), float("nan"), device="cuda")
        pkg.surrogate.gemm_bf16(a, b, c, torch.cuda.current_stream().cuda_stream)
        out.append(c)
    assert bool(((out[0].double() - want).abs() <= bound).all())
    assert torch.equal(out[0], out[1])


# smallest; odd multiples of 128 with rows to spare; weight gradients too
# large for one launch; the most layers
@pytest.mark.parametrize("freq,hidden,layers,out,batch,n", [
    (64, 128, 2, 128, 128, 1), (192, 384, 3, 640, 384, 300), (128, 1024, 2, 4096, 1024, 1024),
    (64, 256, 16, 128, 256, 256)])
def test_training_step_of_all_layers(pkg, freq, hidden, layers, out, batch, n):
    S = pkg.surrogate
    m = S.Mlp(n_in=10, n_freq=freq, hidden=hidden, n_layers=layers, n_out=out, batch=batch, seed=7, fourier_sigma=1.5)
    rng = np.random.default_rng(11)
    x = rng.uniform(0, 1, (n, 10)).astype(np.float32)
    y = (0.3 * rng.standard_normal((n, out))).astype(np.float32)
    p, f = m.params, np.float32
    W = m.weights()
    m.gradients(x, y)
    G = [(m.get(S.GRAD_WEIGHT, l), m.get(S.GRAD_BIAS, l)) for l in range(layers)]
    m.train_step(x, y)
    one, b1, b2 = f(1), f(p.beta1), f(p.beta2)
    c1, c2 = one - b1, one - b2  # first step: 1 - b^1
    for l in range(layers):
        for w, g, got in zip(W[l], G[l], m.weights()[l]):
            mm, vv = (one - b1) * g, (one - b2) * g * g
            want = w - f(p.lr) * (mm / c1) / (np.sqrt(vv / c2) + f(p.eps))
            assert np.array_equal(got, want), (l, np.abs(got - want).max())
    # the BF16 copies in both orientations, through the next passes
    W = m.weights()
    pred = m.predict(x)
    feat = m.get(S.FEATURES)
    assert not feat[n:].any()
    if layers <= 3:
        assert rel(pred, so.forward(feat[:n], W, bf16=True)[1]) < layers * 2.0 ** -8
        loss = m.gradients(x, y)
        want_loss, want = so.gradients(feat[:n], W, y, bf16=True)
        assert abs(loss - want_loss) / want_loss < 1e-5
        for l in range(layers):
            assert rel(m.get(S.GRAD_WEIGHT, l), want[l][0]) < 2 * layers * 2.0 ** -8
            assert rel(m.get(S.GRAD_BIAS, l), want[l][1]) < 2 * layers * 2.0 ** -8
    m.close()


def test_split_product_in_a_cuda_graph(pkg):
    """The cluster launch of a split product captured and replayed: the bits
    of the plain call."""
    import torch
    g = torch.Generator(device="cuda").manual_seed(2)
    a = torch.randn(128, 8192, device="cuda", generator=g).to(torch.bfloat16)
    b = torch.randn(128, 8192, device="cuda", generator=g).to(torch.bfloat16)
    c, want = torch.zeros(128, 128, device="cuda"), torch.zeros(128, 128, device="cuda")
    status = torch.zeros(1, dtype=torch.int32, device="cuda")
    pkg.surrogate.gemm_bf16(a, b, want, torch.cuda.current_stream().cuda_stream)
    graph, s = torch.cuda.CUDAGraph(), torch.cuda.Stream()
    with torch.cuda.stream(s):
        with torch.cuda.graph(graph, stream=s):
            pkg.surrogate.gemm_bf16_async(a, b, c, status, s.cuda_stream)
    graph.replay()
    torch.cuda.synchronize()
    assert int(status.item()) == 0 and torch.equal(c, want)


# grouped and single weight gradients; the chain of early launches against
# steps that end before the next begins: the same kernels, so the same bits
@pytest.mark.parametrize("hidden,out,batch", [(128, 128, 128), (512, 2048, 1024), (1024, 4096, 1024)])
def test_queued_steps_equal_single_steps(pkg, hidden, out, batch):
    import torch
    g = torch.Generator(device="cuda").manual_seed(1)
    x = torch.rand(3 * batch, 10, device="cuda", generator=g)
    y = 0.3 * torch.randn(3 * batch, out, device="cuda", generator=g)
    torch.cuda.synchronize()
    kept = []
    for queued in (True, True, False):
        m = pkg.surrogate.Mlp(n_in=10, n_freq=64, hidden=hidden, n_layers=4, n_out=out, batch=batch, seed=2)
        for k in range(24):
            at = k % 3 * batch
            m.train_step(x[at:at + batch], y[at:at + batch], want_loss=False)
            if not queued:
                m.sync()
        kept.append(m.weights())
        m.close()
    for other in kept[1:]:
        assert all(np.array_equal(a, b) for p, q in zip(kept[0], other) for a, b in zip(p, q))
