"""CPU tests of what the kernel wrappers decide before a launch: devices they refuse, and which calls take which route.
The library is replaced by a recorder, so nothing is launched."""
import pytest
import torch

from hetu_dit_b200 import _C, kernels
from tests import cpu_stand_ins


class Recorder:
    """Stands in for the loaded library: records the entry points that are called and reports success."""

    def __init__(self):
        self.calls = []

    def __getattr__(self, name):
        def entry(*args):
            self.calls.append((name, args))
            return 0
        return entry


@pytest.fixture
def lib(monkeypatch):
    rec = Recorder()
    monkeypatch.setattr(_C, "lib", lambda: rec)
    monkeypatch.setattr(torch.cuda, "current_device", lambda: 0)
    monkeypatch.setattr(torch._C, "_cuda_getCurrentRawStream", lambda index: 1000 + index)
    return rec


class OnGpu(torch.Tensor):
    """A host tensor that says it is on the GPU."""
    is_cuda = property(lambda self: True)


def gpu_like(*shape, dtype=torch.bfloat16):
    return torch.randn(*shape).to(dtype).as_subclass(OnGpu)


BOX = (16, 32, 1, 0, 0, 1, 0, 0, 8)


def test_host_tensors_never_reach_a_kernel(lib):
    """A wrapper without an is_cuda check of its own still refuses a host tensor: a kernel on a host address would fault."""
    t = torch.zeros(1, 8, 2, 64, dtype=torch.bfloat16)
    calls = (lambda: kernels.copy_pieces([BOX], torch.device("cpu")),
             lambda: kernels.copy_2d(torch.empty(4, 8), torch.zeros(4, 8)),
             lambda: kernels.kv_scatter(torch.zeros(1, 8, 256), t.view(1, 8, 128).float(), t.view(1, 8, 128).float(), 0),
             lambda: kernels.qk_norm_rope([(t, None, 1, False)]))
    for call in calls:
        with pytest.raises(ValueError, match="cuda"):
            call()
    assert lib.calls == []


def test_ln_modulate_pair_refuses_a_host_tensor_beside_a_gpu_tensor(lib, monkeypatch):
    x, mod = gpu_like(1, 8, 256), gpu_like(1, 256)
    x_dev = type("OnGpu0", (OnGpu,), {"device": property(lambda self: torch.device("cuda", 0))})
    monkeypatch.setattr(torch, "empty", lambda shape, **kw: torch.zeros(shape, dtype=kw["dtype"]))
    with pytest.raises(RuntimeError, match="CUDA"):
        kernels.ln_modulate_pair(x.as_subclass(x_dev), mod, mod, torch.zeros(1, 4, 256, dtype=torch.bfloat16), mod, mod)
    assert "hdit_ln_modulate_items" not in [name for name, _ in lib.calls]


@pytest.mark.parametrize("device", ["cuda:0", "cuda", 0, -1, None, torch.device("cuda"), torch.device("cuda", 0)])
def test_devices_are_named_as_torch_names_them(lib, device):
    kernels.copy_pieces([BOX], device)
    (name, args), = lib.calls
    assert name == "hdit_copy_pieces" and args[1:] == (1, 1000)
    with pytest.raises(ValueError):
        kernels.copy_pieces([BOX], "cpu")
    assert len(lib.calls) == 1


@pytest.fixture
def fused(monkeypatch):
    """Calls of the fused linear kernels, by name; the kernels after a library GEMM are torch stand-ins."""
    calls = []

    def record(name, result):
        def call(*args, **kw):
            calls.append(name)
            return result(*args, **kw)
        return call

    monkeypatch.setattr(kernels, "linear_fused", record("linear_fused", lambda x, w, *a, **kw: x.new_zeros(*x.shape[:2], w.shape[0])))
    monkeypatch.setattr(kernels, "linear_group", record("linear_group", lambda items, *a, **kw: [
        it.x.new_zeros(*it.x.shape[:2], it.weight.shape[0]) for it in items]))
    for name in ("gelu_tanh", "gate_residual", "qk_norm_rope"):
        monkeypatch.setattr(kernels, name, getattr(cpu_stand_ins, name))
    monkeypatch.setattr(kernels, "_group_pays", lambda shapes, k: True)
    return calls


class Doubled(torch.nn.Linear):
    """A layer of its own with a weight, as an adapter or a quantised layer has."""

    def forward(self, x):
        return 2 * super().forward(x)


def _hook(linear):
    linear.register_forward_hook(lambda m, args, y: 2 * y)


def _pre_hook(linear):
    linear.register_forward_pre_hook(lambda m, args: (2 * args[0],))


def _own_forward(linear):
    linear.forward = lambda x: 2 * torch.nn.functional.linear(x, linear.weight, linear.bias)


def _other_module(linear):
    linear.__class__ = Doubled


def _other_weight(linear):
    class Packed(OnGpu):
        pass
    linear.weight = torch.nn.Parameter((2 * linear.weight.detach()).as_subclass(Packed))


def _everywhere(linear):
    return torch.nn.modules.module.register_module_forward_hook(lambda m, args, y: 2 * y if m is linear else None)


@pytest.mark.parametrize("rows", [64, 4608])
@pytest.mark.parametrize("epilogue", ["gelu_tanh", "gate_residual"])
@pytest.mark.parametrize("change", [_hook, _pre_hook, _own_forward, _other_module, _other_weight, _everywhere])
def test_a_layer_with_a_call_of_its_own_is_called(fused, change, epilogue, rows):
    """Whatever a program puts in the way of a linear layer's call changes the result, with fusion on."""
    linear = torch.nn.Linear(32, 64, bias=False, dtype=torch.bfloat16)
    x = gpu_like(1, rows, 32)
    rest = (gpu_like(1, rows, 64), gpu_like(1, 64)) if epilogue == "gate_residual" else ()
    with torch.no_grad():
        y = 2 * linear(x)
        want = cpu_stand_ins.gelu_tanh(y) if epilogue == "gelu_tanh" else cpu_stand_ins.gate_residual(rest[0], rest[1], y)
        handle = change(linear)
        try:
            one = kernels.linear_tail(linear, x, epilogue, *rest)
            plain = torch.nn.Linear(32, 64, dtype=torch.bfloat16)
            two = kernels.linear_tails([(linear, x, epilogue, *rest), (plain, x, epilogue, *rest)])[0]
        finally:
            if handle is not None:
                handle.remove()
    assert torch.equal(one, want) and torch.equal(two, want)


@pytest.mark.parametrize("epilogue", ["gelu_tanh", "gate_residual"])
def test_a_plain_layer_is_fused(fused, epilogue):
    linear, x = torch.nn.Linear(32, 64, dtype=torch.bfloat16), gpu_like(1, 64, 32)
    rest = (gpu_like(1, 64, 64), gpu_like(1, 64)) if epilogue == "gate_residual" else ()
    with torch.no_grad():
        kernels.linear_tail(linear, x, epilogue, *rest)
        kernels.linear_tails([(linear, x, epilogue, *rest)] * 2)
    assert fused == ["linear_fused", "linear_group"]


def _layer(n=64, k=32, bias=True):
    return torch.nn.Linear(k, n, bias=bias, dtype=torch.bfloat16)


def _odd_weight():
    linear = _layer()
    linear.weight = torch.nn.Parameter(torch.randn(64 * 32 + 1).to(torch.bfloat16)[1:].view(64, 32))
    return linear


def _odd_bias():
    linear = _layer()
    linear.bias = torch.nn.Parameter(torch.randn(65).to(torch.bfloat16)[1:])
    return linear


def _expanded_weight():
    linear = _layer()
    linear.weight = torch.nn.Parameter(torch.randn(1, 32).to(torch.bfloat16).expand(64, 32))
    return linear


# what the library GEMM takes and the fused kernel does not: (linear layer, input, out or None)
LAYOUTS = {
    "inner size not a multiple of 8": lambda: (_layer(k=36), gpu_like(1, 40, 36), None),
    "input not 16-byte aligned": lambda: (_layer(), gpu_like(1, 40, 40)[..., 1:33], None),
    "input row stride not a multiple of 8": lambda: (_layer(), gpu_like(1, 40, 36)[..., :32], None),
    "input rows expanded": lambda: (_layer(), gpu_like(1, 1, 32).expand(1, 40, 32), None),
    "weight rows expanded": lambda: (_expanded_weight(), gpu_like(1, 40, 32), None),
    "input columns strided": lambda: (_layer(), gpu_like(1, 40, 64)[..., ::2], None),
    "weight not 16-byte aligned": lambda: (_odd_weight(), gpu_like(1, 40, 32), None),
    "bias not 16-byte aligned": lambda: (_odd_bias(), gpu_like(1, 40, 32), None),
    "result not 16-byte aligned": lambda: (_layer(), gpu_like(1, 40, 32), gpu_like(1, 40, 72)[..., 1:65]),
    "result row stride not a multiple of 8": lambda: (_layer(), gpu_like(1, 40, 32), gpu_like(1, 40, 68)[..., :64]),
}


@pytest.mark.parametrize("epilogue", ["gelu_tanh", "gate_residual"])
@pytest.mark.parametrize("layout", LAYOUTS)
def test_layouts_of_the_library_gemm_stay_with_it(fused, layout, epilogue):
    linear, x, out = LAYOUTS[layout]()
    rest = (gpu_like(1, 40, 64), gpu_like(1, 64)) if epilogue == "gate_residual" else ()
    with torch.no_grad():
        y = linear(x)
        want = cpu_stand_ins.gelu_tanh(y) if epilogue == "gelu_tanh" else cpu_stand_ins.gate_residual(*rest, y)
        got = kernels.linear_tail(linear, x, epilogue, *rest, out=out)
    assert fused == [] and torch.equal(got, want)


# residuals and gates that gate_residual() takes or refuses by itself, and the fused kernel would not take or would misread
TAILS = {
    "residual in 32 bits": lambda: (gpu_like(2, 40, 64, dtype=torch.float32), gpu_like(2, 64)),
    "gate in 32 bits": lambda: (gpu_like(2, 40, 64), gpu_like(2, 64, dtype=torch.float32)),
    "residual not 16-byte aligned": lambda: (gpu_like(2, 40, 72)[..., 1:65], gpu_like(2, 64)),
    "gate with a row between": lambda: (gpu_like(2, 40, 64), gpu_like(2, 1, 64)),
    "residual rows expanded": lambda: (gpu_like(1, 1, 64).expand(2, 40, 64), gpu_like(2, 64)),
    "gate of one row for two": lambda: (gpu_like(2, 40, 64), gpu_like(1, 64)),
    "residual of another shape": lambda: (gpu_like(1, 80, 64), gpu_like(2, 64)),
    "residual on the host": lambda: (torch.zeros(2, 40, 64, dtype=torch.bfloat16), gpu_like(2, 64)),
}


@pytest.mark.parametrize("tail", TAILS)
def test_tails_of_the_separate_kernel_stay_with_it(fused, monkeypatch, tail):
    """Residuals and gates that the separate kernel takes, or refuses, go there and not to the fused kernel."""
    res, gate = TAILS[tail]()
    if tail == "residual on the host":
        monkeypatch.setattr(OnGpu, "device", property(lambda self: torch.device("cuda", 0)))
        monkeypatch.setattr(torch.nn.Parameter, "device", property(lambda self: torch.device("cuda", 0)), raising=False)
    seen = []
    monkeypatch.setattr(kernels, "gate_residual", lambda r, g, y, out=None: seen.append((r, g)) or y)
    linear, x = _layer(), gpu_like(2, 40, 32)
    with torch.no_grad():
        kernels.linear_tail(linear, x, "gate_residual", res, gate)
        kernels.linear_tails([(linear, x, "gate_residual", res, gate)] * 2)
    assert fused == [] and len(seen) == 3 and all(r is res and g is gate for r, g in seen)


@pytest.mark.parametrize("wrong", ["residual", "gate", "out"])
def test_fused_kernel_refuses_other_types_than_its_own(lib, wrong):
    """The kernel reads and writes 16-bit elements: a 32-bit residual, gate or result would be misread."""
    x = gpu_like(1, 40, 32)
    x = x.as_subclass(type("OnGpu0", (OnGpu,), {"device": property(lambda self: torch.device("cuda", 0))}))
    kw = {"residual": gpu_like(1, 40, 64), "gate": gpu_like(1, 64), "out": gpu_like(1, 40, 64)}
    kw[wrong] = kw[wrong].float()
    with pytest.raises(ValueError, match="dtype"):
        kernels.linear_fused(x, gpu_like(64, 32), None, "gate_residual", **kw)
    assert lib.calls == []


def _linear_group(items, cos=None, sin=None, **kw):
    """linear_group() as its documentation has it, in torch."""
    for it in items:
        y = torch.nn.functional.linear(it.x, it.weight, it.bias)
        if it.epilogue == "norm_rope":
            kind, w, b, eps = it.norm or (0, None, None, 1e-6)
            start, row0 = it.rope or (0, 0)
            cpu_stand_ins.qk_norm_rope([(y.view(*y.shape[:2], -1, it.head_dim), w, kind, it.rope is not None, b)], eps=eps,
                                       cos=cos, sin=sin, rope_seq_start=start, rope_row0=row0)
        it.out = y if it.out is None else it.out.copy_(y)
    return [it.out for it in items]


def _attention(kind, head_dim, **norms):
    from hetu_dit_b200.model_executor.models.shaped_dit import Attention, DiTShape
    shape = DiTShape("tiny", 1, 1, 256, 256 // head_dim, head_dim, 64, 128, 96, True, None, False, qk_norm_kind=kind)
    attn = Attention(shape, joint=False).to(torch.bfloat16)
    gen = torch.Generator().manual_seed(head_dim)
    for p in attn.parameters():
        p.data.copy_(torch.randn(p.shape, generator=gen) * (0.1 if p.dim() == 2 else 0.3) + (1 if p.dim() == 1 else 0))
    return attn


def _tables(rows, head_dim):
    ang = torch.randn(rows, head_dim // 2).repeat_interleave(2, -1)
    return torch.cos(ang), torch.sin(ang)


def _both_routes(monkeypatch, attn, ranges, rope, B=1, S=50):
    """[q, k, v] by the grouped launch where it is taken and by the separate kernels, and whether it was taken."""
    from hetu_dit_b200.model_executor.layers import attention_processor as ap
    taken = []
    monkeypatch.setattr(kernels, "linear_group", lambda *a, **kw: taken.append(1) or _linear_group(*a, **kw))
    stream = [(gpu_like(B, S, 256), (attn.to_q, attn.to_k, attn.to_v), (attn.norm_q, attn.norm_k), ranges)]
    with torch.no_grad():
        (got,) = ap._qkv(attn, stream, rope)
        monkeypatch.setattr(kernels, "FUSED_LINEAR", False)
        (want,) = ap._qkv(attn, stream, rope)
    return got, want, bool(taken)


def _break_nothing(attn, rope):
    return rope


def _fp32_weight(attn, rope):
    attn.norm_k.weight.data = attn.norm_k.weight.data.float()
    return rope


def _odd_norm_weight(attn, rope):
    attn.norm_q.weight.data = torch.ones(attn.head_dim + 1, dtype=torch.bfloat16)[1:]
    return rope


def _longer_sines(attn, rope):
    return rope[0], torch.cat([rope[1], rope[1]])


@pytest.mark.parametrize("kind,head_dim,change,grouped", [
    ("rms", 64, _break_nothing, True), ("rms", 128, _break_nothing, True), ("layer", 64, _break_nothing, True),
    ("layer", 128, _break_nothing, False), ("rms", 64, _fp32_weight, False), ("layer", 64, _odd_norm_weight, False),
    ("rms", 128, _longer_sines, False)])
@pytest.mark.parametrize("ranges", [[(0, 50, True, 0, 0)], [(0, 50, True, 3, 17)], [(0, 9, False, 0, 0), (9, 50, True, 5, 0)]])
def test_qkv_takes_the_grouped_launch_only_where_its_epilogue_can(fused, monkeypatch, kind, head_dim, change, grouped, ranges):
    """LayerNorm of 128-wide heads, norm weights and tables that the epilogue does not take: the separate kernels, as for
    all other layers that are not grouped. Where it is grouped the result is the same."""
    attn = _attention(kind, head_dim)
    got, want, taken = _both_routes(monkeypatch, attn, ranges, change(attn, _tables(60, head_dim)))
    assert taken is grouped
    for g, w in zip(got, want):
        assert torch.equal(g, w)


@pytest.mark.parametrize("norms", ["own eps", "K only", "Q only"])
@pytest.mark.parametrize("rotate", [False, True])
def test_qkv_normalises_the_same_on_both_routes(fused, monkeypatch, norms, rotate):
    """One eps, Q's, serves both; K alone is normalised only beside a rotation."""
    attn = _attention("rms", 64)
    attn.norm_q.eps, attn.norm_k.eps = 0.5, 2.0
    if norms == "K only":
        attn.norm_q = None
    if norms == "Q only":
        attn.norm_k = None
    got, want, taken = _both_routes(monkeypatch, attn, [(0, 50, rotate, 0, 0)], _tables(50, 64) if rotate else None)
    assert taken
    for g, w in zip(got, want):
        assert torch.equal(g, w)


@pytest.fixture
def block_of(fused, monkeypatch):
    """Builds a block whose kernels are torch stand-ins and runs it on tensors that say they are on the GPU."""
    from hetu_dit_b200.core.distributed import parallel_state as ps
    from hetu_dit_b200.core.resource_manager.cache_manager import reset_cache_manager
    from hetu_dit_b200.model_executor.models.shaped_dit import CogVideoXBlock, DiTShape, JointBlock
    ps.destroy_model_parallel()
    reset_cache_manager()
    for name in ("attn_fwd", "ln_modulate"):
        monkeypatch.setattr(kernels, name, getattr(cpu_stand_ins, name))
    monkeypatch.setattr(kernels, "ln_modulate_pair", lambda x, xs, xc, c, cs, cc, eps=1e-6, x_out=None, c_out=None: (
        kernels.ln_modulate(x, xs, xc, eps, x_out), kernels.ln_modulate(c, cs, cc, eps, c_out)))
    monkeypatch.setattr(kernels, "linear_group", _tails_group)
    monkeypatch.setattr(kernels, "linear_fused", lambda x, w, b, epilogue, **kw: _tails_group([_item(x, w, b, epilogue, **kw)])[0])

    def build(kind):
        torch.manual_seed(5)
        shape = DiTShape("tiny", 1, 0, 128, 2, 64, 64, 128, 96, True, None, False, block_kind=kind, temb_dim=128)
        block = (JointBlock if kind == "mmdit" else CogVideoXBlock)(shape).to(torch.bfloat16)
        x, c, temb = gpu_like(1, 40, 128), gpu_like(1, 33, 128), gpu_like(1, 128)

        def run():
            with torch.no_grad():
                return block(x, c, temb, None)
        return block, run
    return build


def _item(x, weight, bias, epilogue, residual=None, gate=None, out=None):
    linear = torch.nn.Linear(8, 8)
    linear.weight, linear.bias = weight, bias
    return kernels.Lin(x, linear, epilogue, residual, gate, out)


def _tails_group(items, cos=None, sin=None, **kw):
    outs = _linear_group(items, cos, sin)
    for i, it in enumerate(items):
        if it.epilogue == "gelu_tanh":
            outs[i] = cpu_stand_ins.gelu_tanh(outs[i], out=it.out)
        if it.epilogue == "gate_residual":
            outs[i] = cpu_stand_ins.gate_residual(it.residual, it.gate, outs[i])
    return outs


def _named(block, path):
    return block.get_submodule(path) if path else block


@pytest.mark.parametrize("kind", ["mmdit", "cogvideox"])
@pytest.mark.parametrize("path", ["ff", "ff.module", "ff.module.net.0", "ff.module.net.1", "ff.module.net.2"])
@pytest.mark.parametrize("how", ["hook", "class", "object"])
def test_an_mlp_of_its_own_is_called(block_of, kind, path, how):
    block, run = block_of(kind)
    plain, called = run(), []
    module = _named(block, path)
    if how == "hook":
        module.register_forward_hook(lambda *a: called.append(1))
    else:
        forward = module.forward

        def own(*args, **kw):
            called.append(1)
            return forward(*args, **kw)
        if how == "object":
            module.forward = own
        else:
            module.__class__ = type("Own", (type(module),), {"forward": lambda self, *args, **kw: own(*args, **kw)})
    for a, b in zip(run(), plain):
        assert torch.allclose(a.float(), b.float(), atol=0.05, rtol=0.05)
    assert called == [1]


@pytest.mark.parametrize("path", ["attn", "attn.module"])
def test_a_hook_on_attention_sees_the_projected_attention(block_of, monkeypatch, path):
    """The residual is added outside the attention module, whatever the kernels fuse: a hook sees and changes the projected
    attention output alone."""
    block, run = block_of("mmdit")
    plain = run()
    seen = []
    _named(block, path).register_forward_hook(lambda m, args, y: seen.append(y) or tuple(2 * t for t in y))
    got = run()
    monkeypatch.setattr(kernels, "FUSED_LINEAR", False)
    want = run()
    for a, b in zip(seen[0], seen[1]):
        assert torch.equal(a, b)
    for a, b, p in zip(got, want, plain):
        assert torch.equal(a, b) and not torch.equal(a, p)


def test_a_processor_of_its_own_need_not_know_the_residual(block_of, monkeypatch):
    from hetu_dit_b200.model_executor.layers.attention_processor import JointAttnProcessor

    class Own(JointAttnProcessor):
        def __call__(self, attn, x, tails=None, **kw):
            return tuple(2 * t for t in super().__call__(attn, x, **kw))

    block, run = block_of("mmdit")
    block.attn.module.processor = Own()
    got = run()
    monkeypatch.setattr(kernels, "FUSED_LINEAR", False)
    for a, b in zip(got, run()):
        assert torch.equal(a, b)


def test_switches_hold_for_grouped_layers_too(fused, monkeypatch):
    """The row limits count an input's rows once, however many layers read it; a tail that is not named is not fused."""
    attn = _attention("rms", 64)
    for name, value in (("FUSED_LINEAR_MIN_ROWS", 51), ("FUSED_LINEAR_MAX_ROWS", 49), ("FUSED_LINEAR_TAILS", {"gelu_tanh"}),
                        ("FUSED_LINEAR_TAILS", {"bias", "gelu_tanh", "gate_residual"})):
        with monkeypatch.context() as m:
            m.setattr(kernels, name, value)
            assert not _both_routes(m, attn, [(0, 50, True, 0, 0)], _tables(50, 64))[2], (name, value)
    monkeypatch.setattr(kernels, "FUSED_LINEAR_MIN_ROWS", 50)
    monkeypatch.setattr(kernels, "FUSED_LINEAR_MAX_ROWS", 50)
    with torch.no_grad():
        kernels.linear_tails([(_layer(), gpu_like(1, n, 32), "gate_residual", gpu_like(1, n, 64), gpu_like(1, 64))
                              for n in (17, 33)])
        with pytest.raises(ValueError):
            kernels.linear_tail(_layer(), gpu_like(1, 50, 32), "bias")  # a name of the switch, not a tail
    assert fused == ["linear_group"]
    assert _both_routes(monkeypatch, attn, [(0, 9, False, 0, 0), (9, 50, True, 0, 0)], _tables(50, 64))[2]
