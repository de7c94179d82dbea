"""Growing the key / value cache (host logic, on CPU tensors): rows are added in place only while nobody else holds the
cache, and caches of different steps never share memory."""
import types

import pytest
import torch

from plaquant_b200 import build, forward_pass


@pytest.fixture(scope="module")
def front_end():
    build.build_library()
    build.build_torch_front_end()


@pytest.fixture
def model(front_end):
    m = object.__new__(forward_pass.ResQForwardB200)
    m.kv_quant, m.kv_heads, m.device, m.layers = False, 2, torch.device("cpu"), [types.SimpleNamespace()]
    m.kv, m._kv_room, m.embed = [None], [], torch.empty(0)
    return m


def _append(m, b, t, pos0, value):
    k, v, n, cap = m._cache_room(0, b, t, pos0)
    assert n == pos0 and cap >= n + t and k.shape == v.shape == (b, n + t, 2, 128)
    k[:, n:], v[:, n:] = value, -value


def _check(cache, values):
    for x, sign in zip(cache, (1, -1)):
        assert x.shape[1] == len(values) and bool((x == sign * torch.tensor(values, dtype=x.dtype)[None, :, None, None]).all())


HOLD = {"entry": lambda m: m.kv[0], "list": lambda m: list(m.kv), "tensor": lambda m: m.kv[0][1], "slice": lambda m: m.kv[0][0][:, :1],
        "transposed": lambda m: m.kv[0][0].transpose(1, 2), "storage": lambda m: m.kv[0][1].untyped_storage(),
        "numpy": lambda m: m.kv[0][0].view(torch.int16).numpy()}


@pytest.mark.parametrize("mode", [torch.no_grad, torch.inference_mode, torch.enable_grad])
@pytest.mark.parametrize("b", [1, 3])
def test_steps_append_in_place_while_nobody_holds_the_cache(model, b, mode):
    with mode():
        _append(model, b, 5, 0, 1.0)
        _append(model, b, 1, 5, 2.0)                      # behind a prompt: copied once
        at = [x.data_ptr() for x in model.kv[0]]
        values = [1.0] * 5 + [2.0]
        for i in range(31):
            _append(model, b, 1, 6 + i, 3.0 + i)
            values.append(3.0 + i)
            assert [x.data_ptr() for x in model.kv[0]] == at
        _check(model.kv[0], values)
        _append(model, b, 2, 37, 50.0)                    # past the spare rows
        assert [x.data_ptr() for x in model.kv[0]] != at
        _check(model.kv[0], values + [50.0] * 2)


@pytest.mark.parametrize("mode", [torch.no_grad, torch.inference_mode])
@pytest.mark.parametrize("how", sorted(HOLD))
def test_a_held_cache_shares_no_memory_with_later_steps(model, how, mode):
    with mode():
        _append(model, 2, 3, 0, 1.0)
        _append(model, 2, 1, 3, 2.0)
        held = HOLD[how](model)
        at = [x.data_ptr() for x in model.kv[0]]
        _append(model, 2, 1, 4, 3.0)
        moved = [x.data_ptr() for x in model.kv[0]]
        assert not set(at) & set(moved)
        _check(model.kv[0], [1.0] * 3 + [2.0, 3.0])
        del held
        _append(model, 2, 1, 5, 4.0)                      # nobody holds this one
        assert [x.data_ptr() for x in model.kv[0]] == moved


def test_editing_a_held_cache_changes_no_other(model):
    _append(model, 2, 3, 0, 1.0)
    _append(model, 2, 1, 3, 2.0)
    first = list(model.kv)
    _append(model, 2, 1, 4, 3.0)
    second = list(model.kv)
    first[0][0][:, 0] = 9.0                               # an older step's
    _check(second[0], [1.0] * 3 + [2.0, 3.0])
    second[0][1][:, 1] = 7.0                              # the live one: the next step continues from the edit
    _append(model, 2, 1, 5, 4.0)
    third = [x.clone() for x in model.kv[0]]
    second[0][1].zero_()
    assert all(torch.equal(x, y) for x, y in zip(third, model.kv[0])) and float(third[1][0, 1, 0, 0]) == 7.0
    model.kv = first                                      # put back, edits included
    _append(model, 2, 1, 4, 5.0)
    assert float(model.kv[0][0][0, 0, 0, 0]) == 9.0 and float(first[0][0][1, 0, 0, 0]) == 9.0
    assert first[0][0].shape[1] == 5                      # the caller's list follows the model


def test_objects_pickled_by_an_earlier_version_still_work(model, monkeypatch):
    """Their state has no native object, no cache room and no RoPE tables."""
    from plaquant_b200 import ops, quantize
    lin = object.__new__(quantize.QuantizedLinear)
    lin.__dict__.update(_gemm_w="packed")
    monkeypatch.setattr(ops, "native_linear", lambda w: ("native", w))
    assert lin.native() == ("native", "packed") and lin.__getstate__()["_native"] is None
    del model._kv_room
    model.cfg = forward_pass.LlamaConfig()
    _append(model, 2, 3, 0, 1.0)
    _append(model, 2, 1, 3, 2.0)
    _check(model.kv[0], [1.0] * 3 + [2.0])
    want = model._rope_angles(torch.arange(5, 8, dtype=torch.float32))
    assert all(torch.equal(x, y) for x, y in zip(model._rope_rows(5, 3), want))
    assert len(object.__new__(forward_pass.ResQForwardB200)._kv_room) == 0


def test_rope_rows_follow_the_configuration(model):
    model.cfg = forward_pass.LlamaConfig()
    model._make_rope_tables()
    for theta in (model.cfg.rope_theta, 10000.0):
        model.cfg.rope_theta = theta
        for pos0, t in ((0, 4), (5, 1), (32767, 1), (32766, 3)):
            want = model._rope_angles(torch.arange(pos0, pos0 + t, dtype=torch.float32))
            # one angle, two calls of cos: vector body and tail may differ by a few units of 2^-24
            assert all(torch.allclose(x, y, rtol=0, atol=1e-6) for x, y in zip(model._rope_rows(pos0, t), want))


def test_a_cache_that_does_not_belong_to_the_model_is_refused(model):
    _append(model, 2, 3, 0, 1.0)
    good = model.kv[0]
    for bad in ([x.to("meta") for x in good], [x.float() for x in good], [x[:, :, :1] for x in good], [good[0], good[1][:, :2]], [x[:1] for x in good]):
        model.kv = [tuple(bad)]
        with pytest.raises(RuntimeError):
            model._cache_room(0, 2, 1, 3)


def test_a_step_that_fails_leaves_the_cache(model, monkeypatch):
    _append(model, 2, 3, 0, 1.0)
    _append(model, 2, 1, 3, 2.0)
    held = model.kv[0]

    def no_memory(*a, **kw):
        raise RuntimeError("out of memory")
    monkeypatch.setattr(forward_pass.torch, "empty", no_memory)
    with pytest.raises(RuntimeError):
        model._cache_room(0, 2, 1, 4)
    monkeypatch.undo()
    _check(model.kv[0], [1.0] * 3 + [2.0])
    _append(model, 2, 1, 4, 3.0)
    _check(model.kv[0], [1.0] * 3 + [2.0, 3.0])
    _check(held, [1.0] * 3 + [2.0])
    with pytest.raises(RuntimeError):
        model._cache_room(0, 3, 1, 5)                     # another batch size
    _check(model.kv[0], [1.0] * 3 + [2.0, 3.0])


def test_a_gate_up_switched_to_another_product_is_refused(model):
    """The activation in the product's epilogue takes the same linears as the call it replaces."""
    from plaquant_b200 import quantize
    lin = object.__new__(quantize.QuantizedLinear)
    lin.__dict__.update(gemm_impl="pytorch", _gemm_w=types.SimpleNamespace(rows=256))
    model.ffn, model.k_hi_ffn = 128, 0
    with pytest.raises(ValueError):
        model._gate_up(types.SimpleNamespace(gate_up=lin), None, like=100)


@pytest.mark.parametrize("mask_elements", [1 << 27, 0])
@pytest.mark.parametrize("b,t,ctx,heads", [(2, 1, 7, 4), (2, 5, 5, 2), (1, 2, 3, 4), (3, 5, 12, 2), (1, 64, 200, 2)])
def test_a_chunk_sees_every_position_before_it(model, monkeypatch, b, t, ctx, heads, mask_elements):
    """Query i of a chunk is position ctx - t + i: attention over that many positions and itself, in float64."""
    monkeypatch.setattr(forward_pass, "CHUNK_MASK_ELEMENTS", mask_elements)
    model.heads, model.cfg = heads, forward_pass.LlamaConfig()
    g = torch.Generator().manual_seed(t)
    q, kk, vv = (torch.randn(b, n, h, 128, generator=g).to(torch.bfloat16) for n, h in ((t, heads), (ctx + 3, 2), (ctx + 3, 2)))
    got = model._attend(q, kk, vv, ctx, None).view(b, t, heads, 128)
    qd, kd, vd = q.double(), kk[:, :ctx].double().repeat_interleave(heads // 2, 2), vv[:, :ctx].double().repeat_interleave(heads // 2, 2)
    w = torch.einsum("bthd,bshd->bhts", qd, kd) / 128 ** 0.5
    w = w.masked_fill(torch.arange(ctx)[None] > torch.arange(ctx - t, ctx)[:, None], float("-inf")).softmax(-1)
    want = torch.einsum("bhts,bshd->bthd", w, vd)
    # bf16 probabilities and results: two roundings of 2^-9 each, probabilities summed over values up to 5
    assert (got.double() - want).abs().max() <= 2.0 ** -9 * (want.abs().max() + vd.abs().max())
