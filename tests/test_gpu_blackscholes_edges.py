"""Black-Scholes kernels at the edges of their launch shapes: counts around a
CTA's 512 options, odd counts, every alignment class of both layouts, and the
arguments where the packed exp reads its table at the ends (d near 0, at the
zero cut-off, far beyond it, infinite and NaN). Bar: bit-exact against the
restated device kernel, nothing written outside the outputs.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _fields(n, seed):
    from hb_hammerbench_b200 import blackscholes as bs
    rec = bs.option_records(n, seed)
    k = min(n, 64)  # deep in / out of the money, at the money, tiny volatility and maturity
    rng = np.random.Generator(np.random.PCG64(seed + 1))
    rec[:k, 3] = rng.choice(np.float32([1e-3, 0.01, 0.05, 2.0]), k)
    rec[:k, 4] = rng.choice(np.float32([1e-4, 0.01, 1.0, 4.0]), k)
    if n > 3:
        rec[1, 3] = 0.0    # d = x / 0: infinite
        rec[2, 4] = -1.0   # square root of a negative: NaN
    return rec


def _same(got, want):
    return np.array_equal(got, want, equal_nan=True)


@pytest.mark.parametrize("n", [1, 2, 3, 511, 512, 513, 1023, 1025, 4097])
@pytest.mark.parametrize("offset", [0, 1, 2, 4])
def test_counts_and_alignments_bit_exact(oracle_mod, n, offset):
    import torch

    from hb_hammerbench_b200 import blackscholes as bs
    rec = _fields(n, n)
    want = oracle_mod.bs_device(rec)
    call, put = want[:, 5], want[:, 6]
    buf = torch.full((8 * n + 16,), -7.0, device="cuda")
    view = buf[offset:offset + 8 * n].view(n, 8)
    view.copy_(torch.from_numpy(rec))
    bs.price(view)
    out = view.cpu().numpy()
    assert _same(out[:, 5], call) and _same(out[:, 6], put)
    assert _same(out[:, :5], rec[:, :5]) and _same(out[:, 7], rec[:, 7])
    rest = torch.cat([buf[:offset], buf[offset + 8 * n:]]).cpu().numpy()
    assert (rest == -7.0).all()

    bufs = [torch.full((n + 8,), -7.0, device="cuda") for _ in range(7)]
    views = [b[offset:offset + n] for b in bufs]
    for i in range(5):
        views[i].copy_(torch.from_numpy(np.ascontiguousarray(rec[:, i])))
    bs.price_arrays(*views[:5], call=views[5], put=views[6])
    assert _same(views[5].cpu().numpy(), call) and _same(views[6].cpu().numpy(), put)
    for b in bufs:
        assert (torch.cat([b[:offset], b[offset + n:]]).cpu().numpy() == -7.0).all()
