"""The native calls that take a whole linear or a decoder layer: the same kernels on the same operands as the
operator-by-operator path, so every result is compared bit for bit with that path."""
import copy
import pickle

import pytest
import torch

from tests._util import synth_activation, synth_weight

pytestmark = pytest.mark.gpu
plq = pytest.importorskip("plaquant_b200")


# rows: one, the last of the decode kernel, the first of the GEMM, past one tile; k: scales padded (14336) or not
@pytest.mark.parametrize("k,n,k_hi_fraction", [(4096, 384, 1 / 32), (14336, 256, 1 / 32), (1024, 264, 0.0)])
@pytest.mark.parametrize("rows", [1, 16, 17, 130])
def test_linear_call_equals_pack_and_product(rows, k, n, k_hi_fraction):
    from plaquant_b200.quantize import QuantizedLinear
    lin = QuantizedLinear.from_weight(synth_weight(n, k, seed=k + n).cuda(), high_fraction=k_hi_fraction)
    x = synth_activation(rows, k, seed=rows).cuda()
    gamma = (torch.rand(k, generator=torch.Generator().manual_seed(1)) + 0.5).to(torch.bfloat16).cuda()
    for g in (None, gamma):
        want = lin(lin.quantize_input(x, g))
        got = lin(x, norm_weight=g)
        assert torch.equal(got, want)
    wide = torch.full((rows, n + 64), 7.0, dtype=torch.bfloat16, device="cuda")
    lin(x, out=wide[:, 32:32 + n])
    plain = lin(x)
    assert torch.equal(wide[:, 32:32 + n], plain) and bool((wide[:, :32] == 7).all()) and bool((wide[:, 32 + n:] == 7).all())
    strided = torch.zeros(rows, 2 * k, dtype=torch.bfloat16, device="cuda")[:, ::2]
    strided.copy_(x)
    assert torch.equal(lin(strided), plain) and torch.equal(lin(x.view(1, rows, 1, k)).view(rows, n), plain)
    for other in (copy.deepcopy(lin), pickle.loads(pickle.dumps(lin))):
        assert torch.equal(other(x), plain) and other.native() is not lin.native()
    with pytest.raises(TypeError):
        lin(x.float())
    with pytest.raises(TypeError):
        lin(x, norm_weight=gamma[:-1])
    with pytest.raises((ValueError, plq.PlqError)):
        lin(x[:, :-128].contiguous())
    with pytest.raises(plq.PlqError):
        lin(x[:0])
    plq.check_device_status()


@pytest.mark.parametrize("head_dim,heads,kv_heads,kv_quant", [(128, 4, 2, False), (128, 4, 1, True), (128, 4, 4, "fake"),
                                                              (64, 4, 2, False), (128, 18, 2, False)])
def test_layer_calls_equal_the_operator_path(monkeypatch, head_dim, heads, kv_heads, kv_quant):
    """Prompt, a chunk behind it, single steps, graph decode; also 9 query heads per key head."""
    from plaquant_b200 import forward_pass
    cfg = forward_pass.LlamaConfig(hidden_size=heads * head_dim, intermediate_size=1024, num_layers=2, num_heads=heads,
                                   num_kv_heads=kv_heads, head_dim=head_dim, vocab_size=400)
    ids = torch.randint(0, 400, (3, 40), generator=torch.Generator().manual_seed(7)).cuda()
    m = forward_pass.ResQForwardB200(cfg, "cuda", seed=3, kv_quant=kv_quant)

    def everything():
        out = [m.forward(ids[:, :21]), m.forward(ids[:, 21:24], pos0=21)]
        out += [m.forward(ids[:, i:i + 1], pos0=i) for i in range(24, 28)]
        out += [x.clone() for layer in m.kv for x in layer]
        m._decode_states.clear()
        return out + [m.generate(ids[:, :9], 5), m.forward(ids[:, :9], all_positions=True), m.forward(ids[:, :1])]
    got = everything()
    monkeypatch.setattr(forward_pass, "NATIVE_LAYER_ROWS", 0)
    want = everything()
    plq.check_device_status()
    assert all(torch.equal(a, b) for a, b in zip(got, want)) and len(got) == len(want)


def test_rope_rows_behind_the_table_equal_the_direct_form(monkeypatch):
    from plaquant_b200 import forward_pass
    cfg = forward_pass.LlamaConfig(hidden_size=256, intermediate_size=256, num_layers=1, num_heads=2, num_kv_heads=1,
                                   head_dim=128, vocab_size=100)
    m = forward_pass.ResQForwardB200(cfg, "cuda", seed=1)
    for pos0, t in ((0, 1), (5, 7), (32767, 1), (32767, 2), (40000, 3)):
        got = m._rope_rows(pos0, t)
        want = m._rope_angles(torch.arange(pos0, pos0 + t, device="cuda", dtype=torch.float32))
        assert all(a.shape == b.shape and torch.equal(a, b) for a, b in zip(got, want))


@pytest.mark.parametrize("rows_limit", [0, 4096])
@pytest.mark.parametrize("b,t,kv_quant", [(1, 17, False), (3, 40, False), (20, 3, True), (4, 4, False)])
def test_last_position_logits_equal_those_of_every_position(monkeypatch, rows_limit, b, t, kv_quant):
    """The layer behind the last attention runs for the last positions alone: logits and cache as of the whole pass."""
    from plaquant_b200 import forward_pass
    monkeypatch.setattr(forward_pass, "NATIVE_LAYER_ROWS", rows_limit)
    cfg = forward_pass.LlamaConfig(hidden_size=512, intermediate_size=1024, num_layers=2, num_heads=4, num_kv_heads=2,
                                   head_dim=128, vocab_size=400)
    ids = torch.randint(0, 400, (b, t), generator=torch.Generator().manual_seed(t)).cuda()
    m = forward_pass.ResQForwardB200(cfg, "cuda", seed=3, kv_quant=kv_quant)
    last = m.forward(ids)
    kv = [x for layer in m.kv for x in layer]
    full = m.forward(ids, all_positions=True)
    # the head's library GEMM may take another kernel for b rows than for b t: one bf16 step of a logit
    assert (last - full[:, -1]).abs().max() <= 2.0 ** -7 * full[:, -1].abs().max()
    assert all(torch.equal(x, y) for x, y in zip(kv, (x for layer in m.kv for x in layer)))
    h = torch.nn.functional.embedding(ids, m.embed)
    whole = m._run_layers(h, 0, m._rope_rows(0, t))
    short = m._run_layers(h, 0, m._rope_rows(0, t), last_only=True)
    assert all(torch.equal(x[:, -1], y[:, -1]) for x, y in zip(whole, short))
    assert short[0].shape[1] == (1 if b * t > 16 else t)
    plq.check_device_status()


@pytest.mark.parametrize("rows", [1, 16, 17])
def test_linear_refuses_an_output_that_does_not_fit(rows):
    """Every route to the product - a tensor, a packed operand in either layout - looks at `out` before it launches."""
    from plaquant_b200 import ops
    from plaquant_b200.quantize import QuantizedLinear
    lin = QuantizedLinear.from_weight(synth_weight(256, 1024, seed=1).cuda())
    x = synth_activation(rows, 1024, seed=2).cuda()
    forms = [x, x.view(1, rows, 1024), lin.quantize_input(x)]
    if rows <= 8:
        forms.append(ops.pack(x, lin.high_bits_length, hadamard=True, sf_layout="rowmajor"))
    for form in forms:
        want = lin(form)
        for shape, dtype in (((rows, 320), torch.bfloat16), ((rows + 1, 256), torch.bfloat16), ((rows, 256), torch.float16), ((rows * 256,), torch.bfloat16)):
            bad = torch.full(shape, 7, dtype=dtype, device="cuda")
            with pytest.raises((RuntimeError, TypeError)):
                lin(form, out=bad)
            assert bool((bad == 7).all())
        with pytest.raises(RuntimeError):
            lin(form, out=torch.empty(rows, 256, dtype=torch.bfloat16))
        for ok in (torch.empty(rows, 256, dtype=torch.bfloat16, device="cuda"), torch.empty(rows, 1, 256, dtype=torch.bfloat16, device="cuda")):
            got = lin(form, out=ok)
            assert torch.equal(got, want) and got.data_ptr() == ok.data_ptr()
    plq.check_device_status()


@pytest.mark.parametrize("mask_elements", [1 << 27, 0])
@pytest.mark.parametrize("head_dim,heads,kv_heads,kv_quant", [(128, 4, 2, False), (128, 4, 2, True), (128, 4, 2, "fake"), (64, 4, 4, False)])
def test_a_prompt_in_chunks_attends_like_the_whole_prompt(monkeypatch, head_dim, heads, kv_heads, kv_quant, mask_elements):
    """One layer, so that no later layer's 4-bit inputs amplify a rounding: the attention of a chunk behind a prompt against
    those rows of the whole prompt's attention, on the same projections."""
    from plaquant_b200 import forward_pass
    monkeypatch.setattr(forward_pass, "CHUNK_MASK_ELEMENTS", mask_elements)
    cfg = forward_pass.LlamaConfig(hidden_size=heads * head_dim, intermediate_size=256, num_layers=1, num_heads=heads,
                                   num_kv_heads=kv_heads, head_dim=head_dim, vocab_size=100)
    m = forward_pass.ResQForwardB200(cfg, "cuda", seed=3, kv_quant=kv_quant)
    qkv = torch.randn(2, 300, (heads + 2 * kv_heads) * head_dim, generator=torch.Generator().manual_seed(5)).to(torch.bfloat16).cuda()
    m.kv = [None]
    whole = m._attention(0, qkv, 0, m._rope_rows(0, 300), None)
    m.kv = [None]
    parts = [m._attention(0, qkv[:, a:b].contiguous(), a, m._rope_rows(a, b - a), None) for a, b in ((0, 100), (100, 102), (102, 299), (299, 300))]
    got = torch.cat(parts, 1)
    # bf16 results of float32 sums in another order: one step, 2^-8 of the largest
    assert (got.float() - whole.float()).abs().max() <= 2.0 ** -8 * whole.float().abs().max()
    assert m.kv[0][0].shape[1] == 300
    ids = torch.randint(0, 100, (2, 40), generator=torch.Generator().manual_seed(6)).cuda()
    m.forward(ids[:, :20])
    assert torch.isfinite(m.forward(ids[:, 20:], pos0=20, all_positions=True)).all()
    plq.check_device_status()


def test_a_subclass_quantises_its_own_way():
    from plaquant_b200.quantize import QuantizedLinear

    class Halved(QuantizedLinear):
        def quantize_input(self, x, norm_weight=None, eps=1e-6):
            return super().quantize_input(x * 0.5, norm_weight, eps)
    w, x = synth_weight(256, 1024, seed=1).cuda(), synth_activation(5, 1024, seed=2).cuda()
    assert torch.equal(Halved.from_weight(w)(x), QuantizedLinear.from_weight(w)(x * 0.5))
