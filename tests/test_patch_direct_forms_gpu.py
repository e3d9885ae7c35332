"""Inference of a model on fields, settings and weights in every form that training takes them: what the patch layers on the image itself do
not take goes to the copies.

Bound: the two builds round the sum with the input once or twice (2^-9): 2 % of the norm for a whole model."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _model(build=None, **more):
    from terra_b200.models.hierarchical_swin import SequentialHierarchicalSwin

    torch.manual_seed(4)
    return (build or SequentialHierarchicalSwin)(2, num_channels=10, patch_size=4, window_size=4, height=64, width=96, embedding_dim=64, num_heads=2,
                                                 num_layers=2, **more).cuda()


def _field(offset=0):
    flat = torch.randn(64 * 96 * 10 + 8, generator=torch.Generator(device="cuda").manual_seed(1), device="cuda").to(torch.bfloat16)
    return flat[offset:offset + 64 * 96 * 10].view(1, 64, 96, 10)


def _unaligned(x):
    """``x`` at an address that the copies take"""
    flat = torch.empty(x.numel() + 8, device="cuda", dtype=x.dtype)
    return flat[1:1 + x.numel()].view(x.shape).copy_(x)


def _close(a, b):
    return ((a.double() - b.double()).norm() <= 2e-2 * b.double().norm()).item()


@pytest.mark.parametrize("offset", [0, 1, 2, 4, 8])
def test_a_field_at_any_address(offset):
    from terra_b200.ops.gemm import check_status
    from terra_b200.ops.patch import direct_patches_apply

    m, x = _model(), _field(offset)
    assert x.is_contiguous() and x.data_ptr() % 16 == 2 * offset % 16
    kept = m(x)
    with torch.no_grad():
        assert direct_patches_apply(x, 4, 0, 0, 64) == (offset % 8 == 0)
        free = m(x)
    check_status("cuda")
    assert _close(free, kept)


def _marks(monkeypatch, m, x, grad):
    from terra_b200.models import hierarchical_swin

    seen = []
    monkeypatch.setattr(hierarchical_swin, "mark_memory_timeline", lambda phase, label="", **more: seen.append((phase, label)))
    with torch.set_grad_enabled(grad):
        y = m(x)
    return y, seen


@pytest.mark.parametrize("modes", [{}, dict(checkpoint_down_mode="D0", checkpoint_up_mode="U1"), dict(checkpoint_down_mode="D1", checkpoint_up_mode="U0")])
@pytest.mark.parametrize("mode", ["none", "torch", "boundary_offload"])
def test_checkpoint_modes_and_their_marks(monkeypatch, modes, mode):
    m = _model(recompute_config=dict(enabled=True, mode=mode, **modes))
    kept, marks = _marks(monkeypatch, m, _field(), True)
    free, same = _marks(monkeypatch, m, _field(), False)
    assert same == marks and len(marks) >= 4 and _close(free, kept)


@pytest.mark.parametrize("key", ["checkpoint_down_mode", "checkpoint_up_mode"])
def test_an_unknown_checkpoint_mode_is_refused(key):
    m = _model(recompute_config=dict(enabled=True, **{key: "X9"}))
    with torch.no_grad(), pytest.raises(ValueError):
        m(_field())


@pytest.mark.parametrize("name", ["_core", "_run_patch_embed_down", "_run_up_patch_recovery", "_patch_embed", "_patch_recovery"])
@pytest.mark.parametrize("bound", [False, True])
def test_pieces_put_in_place_of_the_model_s_own(name, bound):
    from terra_b200.models.hierarchical_swin import SequentialHierarchicalSwin

    called = []

    def piece(self, *args):
        called.append([type(a) for a in args if a is not None])
        return getattr(super(Mine, self), name)(*args)

    Mine = type("Mine", (SequentialHierarchicalSwin,), {} if bound else {name: piece})
    m = _model(Mine)
    if bound:
        setattr(m, name, lambda *args: piece(m, *args))
    with torch.no_grad():
        y = m(_field())
    assert called and all(t is torch.Tensor for types in called for t in types)
    assert _close(y, _model()(_field()))


def _linears(model):
    return model._embed_linear(), model._recovery_linear()


def test_weights_changed_in_the_working_copy():
    from terra_b200.models.hierarchical_swin import SequentialSwinReference

    m, x = _model(SequentialSwinReference), _field()
    with torch.no_grad():
        m(x)
        for lin in _linears(m):
            for p in lin.parameters():
                p.bf16.mul_(-0.5)
        assert _close(m(x), m(_unaligned(x)))


def test_a_captured_call_reads_the_weights_of_its_replay():
    from terra_b200.models.hierarchical_swin import SequentialSwinReference

    m, x = _model(SequentialSwinReference), _field()
    with torch.no_grad():
        stream = torch.cuda.Stream()
        with torch.cuda.stream(stream):
            m(x)
        torch.cuda.synchronize()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            y = m(x)
        for lin in _linears(m):
            for p in lin.parameters():
                p.bf16.mul_(-0.5)
        graph.replay()
        assert _close(y, m(_unaligned(x)))


@pytest.mark.parametrize("where", ["w", "bias"])
def test_operands_on_another_device_are_refused(where):
    from terra_b200 import _ext
    from terra_b200.ops.gemm import status_word

    x, tokens = _field(), torch.zeros(1, 16, 24, 64, device="cuda", dtype=torch.bfloat16)
    ops = dict(w=torch.zeros(64, 4 * 64, device="cuda", dtype=torch.bfloat16), bias=torch.zeros(64, device="cuda", dtype=torch.bfloat16))
    back = dict(w=torch.zeros(4 * 64, 64, device="cuda", dtype=torch.bfloat16), bias=torch.zeros(4 * 64, device="cuda", dtype=torch.bfloat16))
    ops[where], back[where] = ops[where].cpu(), back[where].cpu()
    with pytest.raises(RuntimeError):
        _ext.load().embed_image(x, ops["w"], ops["bias"], tokens, 4, 0, 0, status_word("cuda"))
    with pytest.raises(RuntimeError):
        _ext.load().recover_image(tokens, back["w"], back["bias"], x, torch.empty_like(x), 4, 0, 0, status_word("cuda"))
