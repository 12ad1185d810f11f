"""The decode step's linear layers (weights streamed once for one to eight rows) against FP64, at the edges of the 16-row
units, the 512-column stages and the ring, with fewer and more units than SMs; sizes it does not take are refused."""

import ctypes

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"
PLAIN, ADD, SILU_MUL, FLOAT = range(4)


def _call(x, norm, weight, out, n, mode):
    from reskv_b200._extension import _stream, bound_library, check

    lib = bound_library(x.device)
    check(lib.reskv_skinny_linear(x.data_ptr(), None if norm is None else norm.data_ptr(), 1e-5, weight.data_ptr(), out.data_ptr(),
                                  x.shape[0], n, x.shape[1], mode, _stream(x.device)))
    status = ctypes.c_uint32(7)
    check(lib.reskv_skinny_linear_status(ctypes.byref(status), _stream(x.device)))
    assert status.value == 0


@pytest.mark.parametrize("mode", [PLAIN, ADD, SILU_MUL, FLOAT])
@pytest.mark.parametrize("norm", [False, True])
@pytest.mark.parametrize("rows,n,k", [(1, 16, 512), (8, 48, 1024), (3, 2368, 512), (5, 2384, 1536), (7, 4752, 2560), (2, 160, 14336)])
def test_against_fp64(rows, n, k, norm, mode):
    g = torch.Generator(device=DEV).manual_seed(rows + n)
    wide = 2 * n if mode == SILU_MUL else n
    weight = (torch.randn(wide, k, generator=g, device=DEV) * k**-0.5).half()
    x = torch.randn(rows, k, generator=g, device=DEV).half()
    gain = (1 + 0.1 * torch.randn(k, generator=g, device=DEV)).half() if norm else None
    residual = torch.randn(rows, n, generator=g, device=DEV).half()
    guard = 64
    buf = torch.full((rows * n + guard,), 7.0, device=DEV, dtype=torch.float32 if mode == FLOAT else torch.float16)
    out = buf[: rows * n].view(rows, n)
    if mode == ADD:
        out.copy_(residual)
    _call(x, gain, weight, out, n, mode)
    assert (buf[rows * n:] == 7.0).all()

    a = x.double()
    slack = 0.0
    if norm:
        a = a * torch.rsqrt((a * a).mean(-1, keepdim=True) + 1e-5) * gain.double()
        slack = 2.0**-10  # x is rounded to FP16 after the norm
    y = a @ weight.double().t()
    # FP32 sums of k products, x's own rounding, one rounding of the result to FP16
    sums = (k * 2.0**-24 + slack) * (a.abs() @ weight.double().abs().t())
    if mode == SILU_MUL:
        gate, up = y[:, :n], y[:, n:]
        want = torch.nn.functional.silu(gate) * up
        # |silu'| < 1.1; gate, up and silu(gate) are rounded to FP16 before the product
        bound = 1.1 * (sums[:, :n] + 2.0**-11 * gate.abs()) * up.abs() + want.abs() * 2.0**-9 + sums[:, n:] * gate.abs() + 1e-6
    else:
        want = y + residual.double() if mode == ADD else y
        bound = sums + want.abs() * 2.0**-10 + 1e-6
    assert ((out.double() - want).abs() <= bound).all()


@pytest.mark.parametrize("rows,n,k,mode", [(9, 16, 512, 0), (0, 16, 512, 0), (1, 24, 512, 0), (1, 16, 768, 0), (1, 4, 512, 2), (8, 4096, 14336, 1), (1, 16, 512, 4)])
def test_other_sizes_are_refused(rows, n, k, mode):
    from reskv_b200._extension import _stream, bound_library

    lib = bound_library(torch.device(DEV))
    assert not lib.reskv_skinny_linear_fits(rows, n, k, mode)
    t = torch.zeros(16, dtype=torch.float16, device=DEV)
    assert lib.reskv_skinny_linear(t.data_ptr(), None, 1e-5, t.data_ptr(), t.data_ptr(), rows, n, k, mode, _stream(t.device)) != 0


@pytest.mark.parametrize("batch", [1, 3, 9])  # nine rows: the library's products
def test_graph_step_of_a_model_of_fitting_width(batch):
    from reskv_b200 import ResKVKernelConfig
    from reskv_b200.models import LlamaShape, ResKVLlama

    cfg = ResKVKernelConfig(num_clusters=4, max_clusters=8, group_size=16, recent_size=8, kmeans_iterations=2)
    model = ResKVLlama(LlamaShape(hidden=512, layers=2, heads=4, kv_heads=1, ffn=1024, vocab=336), cfg, seed=3)
    ids = torch.randint(0, 336, (batch, 90), generator=torch.Generator().manual_seed(2)).cuda()
    eager = [model.prefill(ids[:, :60], reserve=40)] + [model.decode(ids[:, 60 + i]) for i in range(20)]
    model.prefill(ids[:, :60], reserve=40)
    model.begin_graph_decode(batch)
    for i in range(20):
        torch.testing.assert_close(model.decode_graph(ids[:, 60 + i]), eager[i + 1], atol=2e-2, rtol=2e-2)
