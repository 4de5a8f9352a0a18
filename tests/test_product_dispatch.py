"""Which kernel a gated product goes to: at both sides of every border of the rules, for a device of any number of SMs (no kernel runs here)."""
import pytest
import torch

from pylon_b200.kernels import ops


@pytest.fixture
def route(monkeypatch):
    taken = []
    monkeypatch.setattr(ops, "_need_cuda", lambda *tensors: None)
    for name, label in (("linear_gated_columns", "columns"), ("linear_stream", "stream"), ("linear_tcgen05", "tcgen05"), ("linear", "library"), ("swiglu", None)):
        monkeypatch.setattr(ops, name, lambda *args, label=label, **options: label and taken.append(label))

    def of(sms, m, n, k, row=None):
        monkeypatch.setattr(ops, "_multiprocessors", lambda device: sms)
        del taken[:]
        x = torch.empty_strided((m, k), (k if row is None else row, 1), dtype=torch.bfloat16, device="meta")
        ops.linear_swiglu(x, torch.empty(n, k, dtype=torch.bfloat16, device="meta"))
        assert len(taken) == 1
        return taken[0]

    return of


@pytest.mark.parametrize("sms", [132, 148, 160])
def test_gated_products_of_9_to_32_rows(route, sms):
    past, most = 192 * sms + 64, 256 * sms   # a second round of the streaming kernel's blocks; one round of two wide blocks an SM
    for n in (past, most):
        for m, k in ((16, 2_560), (17, 1_536), (32, 8_192)):
            assert route(sms, m, n, k) == "columns"
        for m, k in ((8, 2_560), (9, 2_552), (16, 2_552), (17, 1_528), (32, 64)):
            assert route(sms, m, n, k) == "stream"
    for n in (16, past - 64, most + 16, 3 * most):
        assert route(sms, 16, n, 4_096) == "stream"


@pytest.mark.parametrize("sms", [132, 148, 160])
def test_gated_products_of_33_to_127_rows(route, sms):
    for n in (192 * sms, 256 * sms, 384 * sms, 512 * sms):   # whole rounds of tiles
        assert route(sms, 33, n, 2_048) == route(sms, 65, n, 64) == route(sms, 127, n, 8_192) == "tcgen05"
        assert route(sms, 33, n, 2_040) == route(sms, 64, n, 64) == "library"
    for m in (33, 64, 65, 72):
        assert route(sms, m, 192 * sms - 16, 4_096) == "library"
        assert route(sms, m, 256 * sms + 16, 4_096) == "library"   # a second round of tiles for hardly more rows
    assert route(sms, 73, 128 * sms, 64) == route(sms, 127, 128 * sms, 8_192) == "tcgen05"
    assert route(sms, 73, 128 * sms - 16, 64) == "library"
    assert route(sms, 100, 256 * sms + 16, 4_096) == "library" and route(sms, 100, 256 * sms + 16, 4_088) == "tcgen05"


def test_gated_products_that_only_the_library_takes(route):
    assert route(148, 80, 37_888, 2_048, row=2_040) == route(148, 80, 37_888, 2_048, row=0) == route(148, 80, 37_888, 0) == "library"   # rows that share memory; no k
    assert route(148, 128, 1_024, 64) == route(148, 4_096, 19_456, 2_560) == "tcgen05"
