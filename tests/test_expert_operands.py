"""Operands of the routed experts that the kernels would misread - they get addresses and sizes only - are refused by both entry points."""
import pytest
import torch

E, F, H, T, TOP = 4, 16, 24, 5, 2


def operands(dev):
    z = lambda *s, dtype=torch.bfloat16: torch.zeros(s, dtype=dtype, device=dev)      # noqa: E731
    return dict(h=z(T, H), gate_up=z(E, 2, F, H), down=z(E, H, F), idx=z(T, TOP, dtype=torch.int32), wts=z(T, TOP, dtype=torch.float32),
                extra=z(T, H, dtype=torch.float32), extra_gate=z(T, dtype=torch.float32))


def faults(dev):
    f = operands(dev)
    return {"float32 weights": dict(gate_up=f["gate_up"].float()), "float32 down": dict(down=f["down"].float()),
            "experts in another order of axes": dict(gate_up=torch.zeros((2, E, F, H), dtype=torch.bfloat16, device=dev).transpose(0, 1)),
            "down of another width": dict(down=f["down"][:, :, :8].contiguous()), "transposed down": dict(down=f["down"].transpose(1, 2)),
            "half of the experts' down": dict(down=f["down"][:2]), "numbers of 64 bits": dict(idx=f["idx"].long()), "weights of 16 bits": dict(wts=f["wts"].bfloat16()),
            "choices of fewer tokens": dict(idx=f["idx"][:3]), "strided choices": dict(idx=f["idx"].t().contiguous().t()),
            "extra of another width": dict(extra=f["extra"][:, :8].contiguous()), "extra of 16 bits": dict(extra=f["extra"].bfloat16()),
            "gates of fewer tokens": dict(extra_gate=f["extra_gate"][:3])}


def test_the_checks(monkeypatch):
    from mini_sglang_b200 import ops
    monkeypatch.setattr(ops, "_need_cuda", lambda *t: None)
    good = operands("cpu")
    order = ("h", "gate_up", "down", "idx", "wts", "extra", "extra_gate")
    for more in ({}, dict(idx=torch.cat((good["idx"], good["idx"]))), dict(wts=good["wts"].view(-1))):
        idx, wts = ops._expert_operands(*[dict(good, **more)[k] for k in order])
        assert idx.shape == wts.shape == (T, TOP)
    for what, bad in faults("cpu").items():
        with pytest.raises((AssertionError, RuntimeError, ValueError)):
            ops._expert_operands(*[dict(good, **bad)[k] for k in order])
            raise KeyError(what)


@pytest.mark.gpu
@pytest.mark.parametrize("call", ["experts_few", "experts_many"])
def test_both_entry_points_refuse(call):
    from mini_sglang_b200 import ops
    good = operands("cuda")
    getattr(ops, call)(**good)
    for what, bad in faults("cuda").items():
        with pytest.raises((AssertionError, RuntimeError, ValueError)):
            getattr(ops, call)(**dict(good, **bad))
            raise KeyError(what)
    ops.check_kernel_status()


@pytest.mark.gpu
def test_without_tensor_maps_nothing_is_ordered_in_vain(monkeypatch):
    from mini_sglang_b200 import ops
    good = operands("cuda")
    monkeypatch.setattr(ops, "EXPERT_ROWS_MIN_WEIGHTS", 0)
    want = ops.experts_few(**good)
    monkeypatch.setattr(ops, "_tensor_maps", False)
    assert torch.equal(ops.experts_few(**good), want)
    before = ops.LAUNCHES
    assert ops.experts_many(**good) is None and ops.LAUNCHES == before        # nothing was ordered for a product that cannot run
    assert ops._gemm_rows(good["h"], good["gate_up"].view(-1, H), None, 1, torch.bfloat16) is None
