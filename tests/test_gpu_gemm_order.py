"""A product takes the same time whichever operand is the long one: the tiles in
flight share the panels of both, 16 row panels at a time. Tolerance of a sum of
K products in FP32, in any order: 2 K 2^-24 sum |a b|."""
import pytest

pytestmark = pytest.mark.gpu


def test_tall_product_as_fast_as_its_transpose(pkg):
    """10880x896x12288 against 896x10880x12288 (the same tiles, neither size a
    multiple of 256): as fast up to an eighth, timed in turn, best of several."""
    import torch
    g = torch.Generator(device="cuda").manual_seed(0)
    a = torch.randn(10880, 12288, device="cuda", generator=g).to(torch.bfloat16)
    b = torch.randn(896, 12288, device="cuda", generator=g).to(torch.bfloat16)
    c, ct = torch.empty(10880, 896, device="cuda"), torch.empty(896, 10880, device="cuda")
    status = torch.zeros(1, dtype=torch.int32, device="cuda")
    s = torch.cuda.current_stream().cuda_stream

    def ms(x, y, out):
        for _ in range(2):
            pkg.surrogate.gemm_bf16_async(x, y, out, status, s)
        e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        e0.record()
        for _ in range(5):
            pkg.surrogate.gemm_bf16_async(x, y, out, status, s)
        e1.record()
        e1.synchronize()
        return e0.elapsed_time(e1)

    tall, wide = zip(*[(ms(a, b, c), ms(b, a, ct)) for _ in range(6)])
    assert int(status.item()) == 0
    assert min(tall) < 1.125 * min(wide)


# tile forms with fewer, as many and more row panels than a group, a last group
# of one, several columns of tiles
@pytest.mark.parametrize("M,N,K", [(1920, 128, 128), (2048, 128, 128), (2176, 128, 192), (4224, 384, 64),
                                   (6272, 128, 2048)])
def test_row_panel_groups(pkg, M, N, K):
    import torch
    g = torch.Generator(device="cuda").manual_seed(M + N + K)
    a = torch.randn(M, K, device="cuda", generator=g).to(torch.bfloat16)
    b = torch.randn(N, K, device="cuda", generator=g).to(torch.bfloat16)
    c = torch.full((M, N), float("nan"), device="cuda")
    pkg.surrogate.gemm_bf16(a, b, c, torch.cuda.current_stream().cuda_stream)
    want = a.double() @ b.double().T
    bound = 2 * K * 2.0 ** -24 * (a.double().abs() @ b.double().abs().T)
    assert bool(((c.double() - want).abs() <= bound).all())
