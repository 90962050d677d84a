"""The bf16 copies of a step's weights, made in one launch: what a conversion of each gives, and the same step with and without."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = torch.device("cuda")


def test_copies_are_those_of_torch():
    from tagseq2tagseq_b200.lm_fused import cast_weights
    g = torch.Generator(device=DEV).manual_seed(1)
    shapes = [(1, 1), (3, 5), (8, 1024), (1, 8191), (1, 8192), (1, 8193), (257, 768), (50, 1)] + [(7, 3)] * 140  # more than one launch takes
    ws = [torch.randn(s, device=DEV, generator=g) * 10.0 ** (i % 9 - 4) for i, s in enumerate(shapes)]
    ws.append(torch.empty(33 * 7 + 1, device=DEV).uniform_(-1, 1)[1:].view(33, 7))                              # not at a 16-byte boundary
    ws.append(torch.tensor([[0.0, -0.0, float("inf"), -float("inf"), 1e-40, 3.4e38, 1.00390625, 1.01171875]], device=DEV))  # ends, ties to even
    got = cast_weights(ws)
    assert all(torch.equal(a, w.bfloat16()) and a.shape == w.shape for a, w in zip(got, ws))
    nan = torch.full((2, 9), float("nan"), device=DEV)
    assert cast_weights([nan])[0].isnan().all() and cast_weights([]) == []
    with pytest.raises(ValueError):
        cast_weights([ws[0], ws[2].t()])


def test_a_step_with_copies_is_the_step_without():
    """A hook that does nothing makes every layer convert its own weight: same loss, same gradients, bit for bit (two documents of one tile: attention's
    dq adds nothing up in the order of arrival)."""
    from tagseq2tagseq_b200 import MaskSpec
    from tagseq2tagseq_b200.train_step import DecoderLM, LMConfig
    torch.manual_seed(3)
    vocab = 4096
    with torch.device(DEV):
        model = DecoderLM(LMConfig(2, 128, 2, 64, 256, vocab))
    tokens = torch.randint(0, vocab, (1, 129), device=DEV)
    spec = MaskSpec((torch.arange(128, device=DEV, dtype=torch.int32) // 70)[None], None)

    def run():
        model.zero_grad()
        with torch.autocast("cuda", dtype=torch.bfloat16):
            loss = model(tokens, spec)
        loss.backward()
        return [loss.detach().clone()] + [p.grad.clone() for p in model.parameters()]

    with torch.autocast("cuda", dtype=torch.bfloat16):
        assert len(model._weight_copies()) == 9
    want = run()
    handle = model.blocks[1].proj.register_forward_pre_hook(lambda m, a: None)
    with torch.autocast("cuda", dtype=torch.bfloat16):
        assert model._weight_copies() is None
    for a, b in zip(run(), want):
        assert torch.equal(a, b)
    handle.remove()
    with torch.no_grad(), torch.autocast("cuda", dtype=torch.bfloat16):
        assert model._weight_copies() is None and torch.equal(model(tokens, spec), want[0])


def _small(vocab=4096):
    from tagseq2tagseq_b200 import MaskSpec
    from tagseq2tagseq_b200.train_step import DecoderLM, LMConfig
    torch.manual_seed(3)
    with torch.device(DEV):
        model = DecoderLM(LMConfig(2, 128, 2, 64, 256, vocab))
    tokens = torch.randint(0, vocab, (1, 129), device=DEV)
    spec = MaskSpec((torch.arange(128, device=DEV, dtype=torch.int32) // 70)[None], None)

    def run():
        model.zero_grad()
        with torch.autocast("cuda", dtype=torch.bfloat16):
            loss = model(tokens, spec)
        loss.backward()
        return [loss.detach().clone()] + [p.grad.clone() for p in model.parameters()]
    return model, run


@pytest.mark.parametrize("which", ["Linear", "Block"])
def test_a_forward_replaced_on_the_class_gets_the_arguments_it_always_got(which, monkeypatch):
    from tagseq2tagseq_b200 import train_step
    model, run = _small()
    want = run()
    cls, calls = getattr(train_step, which), []
    own = cls.forward

    def linear(self, x):
        calls.append(self)
        return own(self, x)

    def block(self, x, a, mask, cos, sin):
        calls.append(self)
        return own(self, x, a, mask, cos, sin)

    monkeypatch.setattr(cls, "forward", linear if which == "Linear" else block)
    for a, b in zip(run(), want):
        assert torch.equal(a, b)
    assert len(calls) == (8 if which == "Linear" else 2)


def test_no_copies_ahead_where_something_of_the_callers_is_called_on_the_way():
    """Saved tensors that go to the host as they are saved, and modes that see every operator: each layer converts its own weight when it is its turn."""
    from torch.overrides import TorchFunctionMode
    from torch.utils._python_dispatch import TorchDispatchMode
    from tagseq2tagseq_b200 import MaskSpec
    from tagseq2tagseq_b200.train_step import DecoderLM, LMConfig

    class Function(TorchFunctionMode):
        def __torch_function__(self, f, types, args=(), kwargs=None):
            return f(*args, **(kwargs or {}))

    class Dispatch(TorchDispatchMode):
        def __torch_dispatch__(self, f, types, args=(), kwargs=None):
            return f(*args, **(kwargs or {}))

    small, _ = _small()
    with torch.autocast("cuda", dtype=torch.bfloat16):
        for mode in (Function(), Dispatch(), torch.autograd.graph.save_on_cpu()):
            with mode:
                assert small._weight_copies() is None
        assert len(small._weight_copies()) == 9

    with torch.device(DEV):
        model = DecoderLM(LMConfig(6, 512, 8, 64, 2048, 8192))         # 25 M + 4 M weights
    tokens = torch.randint(0, 8192, (1, 129), device=DEV)
    spec = MaskSpec(torch.zeros((1, 128), device=DEV, dtype=torch.int32), None)

    def peak():
        torch.cuda.synchronize()
        before = torch.cuda.memory_allocated()
        torch.cuda.reset_peak_memory_stats()
        with torch.autocast("cuda", dtype=torch.bfloat16), torch.autograd.graph.save_on_cpu():
            model(tokens, spec)
        return torch.cuda.max_memory_allocated() - before
    peak()                                                            # the plan, the rotation tables
    got = peak()
    model.blocks[0].proj.register_forward_pre_hook(lambda m, a: None)  # with a hook no copies are made ahead
    assert got <= peak() + (1 << 20)


@pytest.mark.parametrize("frozen", ["all", "embedding and first layers"])
def test_copies_that_no_backward_keeps_are_not_held(frozen):
    from tagseq2tagseq_b200 import MaskSpec
    from tagseq2tagseq_b200.train_step import DecoderLM, LMConfig
    with torch.device(DEV):
        model = DecoderLM(LMConfig(6, 512, 8, 64, 2048, 8192))
    for name, p in model.named_parameters():
        p.requires_grad_(frozen != "all" and name.startswith(("blocks.5", "norm", "head")))
    tokens = torch.randint(0, 8192, (1, 129), device=DEV)
    spec = MaskSpec(torch.zeros((1, 128), device=DEV, dtype=torch.int32), None)

    def peak():
        torch.cuda.synchronize()
        before = torch.cuda.memory_allocated()
        torch.cuda.reset_peak_memory_stats()
        with torch.autocast("cuda", dtype=torch.bfloat16):
            model(tokens, spec)
        return torch.cuda.max_memory_allocated() - before
    peak()                                                            # the plan, the rotation tables
    got = peak()
    model.blocks[0].proj.register_forward_pre_hook(lambda m, a: None)  # with a hook no copies are made ahead
    assert got <= peak() + (1 << 20)
    for p in (model.embed.weight, model.blocks[0].qkv.weight):        # either makes every layer keep its own
        model.blocks[0].proj._forward_pre_hooks.clear()
        model.requires_grad_(False)
        p.requires_grad_(True)
        with torch.autocast("cuda", dtype=torch.bfloat16):
            assert len(model._weight_copies()) == 25


def test_a_copy_is_bf16_of_the_weights_size_and_without_a_gradient():
    from tagseq2tagseq_b200.lm_fused import Linear, cast_weights, head_loss
    with torch.device(DEV):
        layer, x, target = Linear(64, 128), torch.randn(9, 64).bfloat16(), torch.randint(0, 128, (9,))
    good, = cast_weights([layer.weight])
    with torch.autocast("cuda", dtype=torch.bfloat16):
        want = layer(x), head_loss(x, layer.weight, target)
        assert torch.equal(layer(x, good), want[0]) and torch.equal(head_loss(x, layer.weight, target, good), want[1])
        for bad in (good.float(), good[:64], good.clone().requires_grad_(), layer.weight.to(torch.bfloat16)):
            with pytest.raises(ValueError):
                layer(x, bad)
            with pytest.raises(ValueError):
                head_loss(x, layer.weight, target, bad)
    head_loss(x, layer.weight, target, good).backward()
    assert layer.weight.grad is not None and good.grad is None


@pytest.mark.parametrize("vocab", [4096, 110592, 110600])
def test_a_head_whose_loss_takes_no_copy_gets_none(vocab):
    """The head's loss in two kernels (rows that do not fit shared memory) converts the weight itself."""
    model, run = _small(vocab)
    with torch.autocast("cuda", dtype=torch.bfloat16):
        copies = model._weight_copies()
    assert len(copies) == 9 and [len(c) for c in copies] == [1] * 8 + [int(vocab <= 110592)]
    want = run()
    model.blocks[1].proj.register_forward_pre_hook(lambda m, a: None)
    for a, b in zip(run(), want):
        assert torch.equal(a, b)
