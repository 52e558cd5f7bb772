"""Float32 products of short inner dimensions and many results: the bits that the same rows have one by one, and the product in 64 bits."""
from ctypes import c_int

import pytest
import torch

pytestmark = pytest.mark.gpu


def takes_whole_sums(m, n, kk):
    from gemmars_b200 import kernels
    return kernels._fn("gemm_ref", "gb_gemm_ref_short", [c_int] * 3)(m, n, kk) == 1


@pytest.mark.parametrize("m,n,kk", [(520, 1030, 1), (517, 1031, 16), (513, 1024, 31), (700, 770, 32), (1030, 1025, 33), (1025, 1050, 63), (1024, 1024, 64),
                                    (2050, 1027, 65), (2048, 1024, 96), (2050, 2049, 97), (2048, 2048, 128), (2049, 1025, 129), (2050, 1030, 160),
                                    (2048, 1025, 191), (2048, 1024, 192)])
@pytest.mark.parametrize("apart", [0, 3])
def test_the_bits_of_single_rows(m, n, kk, apart):
    from gemmars_b200 import kernels as k
    assert takes_whole_sums(m, n, kk) and not takes_whole_sums(40, n, kk)
    g = torch.Generator(device="cuda").manual_seed(m + kk)
    x = torch.randn(m, kk + apart, generator=g, device="cuda")[:, :kk]            # rows that start anywhere
    w, bias, scale = torch.randn(n, kk, generator=g, device="cuda"), torch.randn(n, generator=g, device="cuda"), torch.rand(n, generator=g, device="cuda")
    y, start = torch.empty(m, n, device="cuda"), torch.randn(m, n, generator=g, device="cuda")
    added = start.clone()
    k.gemm_ref(x, w, y, bias, act="gelu")
    k.gemm_ref(x, w, added, bias, accumulate=True, col_scale=scale)
    for rows in (slice(0, 40), slice(m // 2, m // 2 + 1), slice(m - 17, m)):
        part, sums = torch.empty_like(y[rows]), start[rows].clone()
        k.gemm_ref(x[rows], w, part, bias, act="gelu")
        k.gemm_ref(x[rows], w, sums, bias, accumulate=True, col_scale=scale)
        assert torch.equal(part, y[rows]) and torch.equal(sums, added[rows])
    plain = torch.empty_like(y)
    k.gemm_ref(x, w, plain)
    xd, wd = x.double(), w.double()
    bound = kk * 2.0 ** -24 * (xd.abs() @ wd.abs().T)        # half an ulp of the largest partial sum per addition
    assert ((plain.double() - xd @ wd.T).abs() <= bound).all()


def test_the_line():
    for m, n, kk, whole in ((512, 1024, 32, True), (511, 1024, 32, False), (512, 1024, 33, False), (1024, 1024, 64, True), (1024, 1024, 65, False),
                            (2048, 1024, 96, True), (2048, 1024, 97, False), (2048, 2048, 97, True), (2048, 1024, 129, True), (2048, 1024, 193, False),
                            (8192, 8192, 193, False), (1, 151936, 16, False)):
        assert takes_whole_sums(m, n, kk) is whole
