"""Weights that a caller has assigned to a model: the captured step reads a weight by its address only where that is the whole
truth about it (dense row-major FP16, aligned), and gives the logits of the eager step for every other one as well."""

import ctypes

import pytest
import torch


def _half(*shape):
    return torch.arange(torch.Size(shape).numel(), dtype=torch.float32).half().reshape(shape)


def _misaligned(x):
    buf = torch.zeros(x.numel() + 1, dtype=x.dtype, device=x.device)
    buf[1:] = x.flatten()
    return buf[1:].view(x.shape)


# the same values, laid out another way
LAYOUTS = {
    "transposed": lambda w: w.t().contiguous().t(),
    "column slice": lambda w: torch.cat((w + 1, w), 1)[:, w.shape[1]:],
    "every other row": lambda w: torch.stack((w, w + 1), 1).flatten(0, 1)[::2],
    "misaligned": _misaligned,
}


def test_only_dense_aligned_fp16_is_read_by_address():
    from reskv_b200.models.llama import _dense_half

    w, cpu = _half(32, 64), torch.device("cpu")
    assert _dense_half(w, (32, 64), cpu) and _dense_half(torch.nn.Parameter(w), (32, 64), cpu) and _dense_half(w[8:16], (8, 64), cpu)
    for other in (*(how(w) for how in LAYOUTS.values()), w[:1].expand(32, 64), w.float(), w.bfloat16(), w.to_sparse(), w[:31],
                  w.flatten(), torch.Tensor._make_subclass(type("Own", (torch.Tensor,), {}), w), w.to("meta"), torch._neg_view(w)):
        assert not _dense_half(other, (32, 64), cpu)


def _step_logits(change, batch):
    """Logits of some eager and captured steps of a model that ``change`` has been let loose on."""
    from reskv_b200 import ResKVKernelConfig
    from reskv_b200.models import LlamaShape, ResKVLlama

    cfg = ResKVKernelConfig(num_clusters=4, max_clusters=8, group_size=16, recent_size=8, kmeans_iterations=2)
    model = ResKVLlama(LlamaShape(hidden=512, layers=2, heads=4, kv_heads=1, ffn=1024, vocab=336), cfg, seed=3)
    change(model)
    ids = torch.randint(0, 336, (batch, 90), generator=torch.Generator().manual_seed(2)).cuda()
    model.prefill(ids[:, :60], reserve=40)
    eager = [model.decode(ids[:, 60 + i]) for i in range(3)]
    model.prefill(ids[:, :60], reserve=40)
    model.begin_graph_decode(batch)
    return eager, [model.decode_graph(ids[:, 60 + i]).clone() for i in range(3)]


@pytest.mark.gpu
@pytest.mark.parametrize("batch", [2, 9])  # nine rows: not streamed, the norms still are kernels
@pytest.mark.parametrize("name", ["wqkv", "wo", "w_gate_up", "w_down", "lm_head"])
@pytest.mark.parametrize("how", LAYOUTS)
def test_captured_step_with_another_layout(how, name, batch):
    def change(model):
        if name == "lm_head":
            model.lm_head = LAYOUTS[how](model.lm_head)
        else:
            for layer in model.layers:
                layer[name] = LAYOUTS[how](layer[name])

    for got, want in zip(*reversed(_step_logits(change, batch))):
        torch.testing.assert_close(got, want, atol=2e-2, rtol=2e-2)  # as for dense weights


@pytest.mark.gpu
@pytest.mark.parametrize("batch", [2, 9])
@pytest.mark.parametrize("how", ["strided", "float", "misaligned", "one element"])
def test_captured_step_with_other_norm_weights(how, batch):
    def other(w):
        w = (1 + 0.25 * torch.cos(torch.arange(w.numel(), device=w.device))).half()
        if how == "one element":
            return w[3:4]
        return {"strided": torch.stack((w, -w), 1)[:, 0], "float": w.float(), "misaligned": _misaligned(w)}[how]

    def change(model):
        model.final_norm = other(model.final_norm)
        for layer in model.layers:
            layer["norm1"], layer["norm2"] = other(layer["norm1"]), other(layer["norm2"])

    for got, want in zip(*reversed(_step_logits(change, batch))):
        torch.testing.assert_close(got, want, atol=2e-2, rtol=2e-2)


@pytest.mark.gpu
def test_captured_step_with_an_expanded_head():
    def change(model):
        model.lm_head = model.lm_head[:1].expand(336, 512)  # one row of storage

    for got, want in zip(*reversed(_step_logits(change, 2))):
        torch.testing.assert_close(got, want, atol=2e-2, rtol=2e-2)


@pytest.mark.gpu
@pytest.mark.parametrize("which", ["linear", "attention"])
def test_a_step_whose_wait_ran_out_raises(which, monkeypatch):
    """With RESKV_CHECK_STATUS=1; the status words are set by the host, no wait runs out here."""
    from reskv_b200 import ResKVKernelConfig
    from reskv_b200.models import LlamaShape, ResKVLlama

    cfg = ResKVKernelConfig(num_clusters=4, max_clusters=8, group_size=16, recent_size=8, kmeans_iterations=2)
    model = ResKVLlama(LlamaShape(hidden=512, layers=1, heads=4, kv_heads=1, ffn=1024, vocab=336), cfg, seed=3)
    monkeypatch.setattr(ResKVLlama, "_check_status", True)
    ids = torch.randint(0, 336, (2, 62), generator=torch.Generator().manual_seed(2)).cuda()
    model.prefill(ids[:, :60], reserve=40)
    model.begin_graph_decode(2)
    model.decode_graph(ids[:, 60])
    if which == "attention":
        model._workspace[0] = 1
    else:
        library = model._native()

        class Ran:
            def __getattr__(self, name):
                return getattr(library, name)

            def reskv_skinny_linear_status(self, status, stream):
                ctypes.c_uint32.from_address(status).value = 1
                return 0

        model._lib = Ran()
    with pytest.raises(RuntimeError, match="device status"):
        model.decode_graph(ids[:, 61])


def test_rows_that_leave_room_for_the_stream():
    """A ring of at least four stages beside the rows of x: any of the eight at 4096 columns, five at 14336."""
    from reskv_b200._extension import library

    for columns, most in ((512, 8), (4096, 8), (8192, 8), (14336, 5)):
        for rows in range(1, 9):
            assert bool(library().reskv_skinny_linear_fits(rows, 4096, columns, 1)) == (rows <= most), (rows, columns)
