"""Appending to the decoder's key / value cache: the packed-cache kernels against the kernels they replace, byte for
byte, and the in-place growth against caches that were handed out before."""
import pytest
import torch

from tests.test_gpu_7_rope import _tables

pytestmark = pytest.mark.gpu
plq = pytest.importorskip("plaquant_b200")


@pytest.mark.parametrize("b,t,heads,kv,pos0,t_max", [(1, 1, 1, 1, 0, 1), (2, 5, 4, 2, 0, 5), (3, 1, 8, 1, 7, 16),
                                                    (1, 33, 6, 2, 100, 160), (16, 1, 64, 8, 2048, 2176)])
def test_packed_append_and_unpack_byte_for_byte(b, t, heads, kv, pos0, t_max):
    from plaquant_b200 import kv_cache, ops
    g = torch.Generator().manual_seed(b * 100 + t)
    qkv = torch.randn(b, t, (heads + 2 * kv) * 128, generator=g) * 2
    qkv[..., ::37] = -0.0                                              # signed zeros, a zero block, large and tiny blocks
    qkv[..., -128:-112] = 0
    qkv[:, :1, -256:-192] *= 1e4
    qkv[:, :1, -64:] *= 1e-6
    qkv = qkv.to(torch.bfloat16).cuda()
    cos, sin = (x.cuda() for x in _tables(pos0, t))
    kb, vb = (torch.empty(b, t, kv, 128, dtype=torch.bfloat16, device="cuda") for _ in range(2))
    q_want = ops.rope_kv_append(qkv, cos, sin, heads, kv, kb, vb, 0)
    want = kv_cache.pack_head_rows(kb, hadamard=True), kv_cache.pack_head_rows(vb, hadamard=False)
    for pos in (pos0, torch.tensor([pos0], device="cuda")):
        rows = [torch.full((b, t_max, kv, 72), 7, dtype=torch.uint8, device="cuda") for _ in range(2)]
        q = ops.rope_kv_append(qkv, cos, sin, heads, kv, *rows, pos)
        plq.check_device_status()
        assert torch.equal(q, q_want)
        for got, w in zip(rows, want):
            assert torch.equal(got[:, pos0:pos0 + t], w)
            assert bool((got[:, :pos0] == 7).all()) and bool((got[:, pos0 + t:] == 7).all())
    for ctx in {1, pos0 + t, t_max}:
        rows[0].random_(0, 0x7F, generator=torch.Generator("cuda").manual_seed(1))       # any code, any finite scale
        got = ops.unpack_head_rows(*rows, ctx)
        for x, r in zip(got, rows):
            assert torch.equal(x.view(torch.int16), kv_cache.unpack_head_rows(r[:, :ctx]).view(torch.int16))


def test_packed_append_behind_the_cache_is_reported():
    from plaquant_b200 import ops
    qkv = torch.randn(2, 1, 4 * 128).to(torch.bfloat16).cuda()
    cos, sin = (x.cuda() for x in _tables(4, 1))
    rows = [torch.full((2, 4, 1, 72), 7, dtype=torch.uint8, device="cuda") for _ in range(2)]
    ops.rope_kv_append(qkv, cos, sin, 2, 1, *rows, torch.tensor([4], device="cuda"))
    with pytest.raises(plq.PlqError):
        plq.check_device_status()
    assert all(bool((r == 7).all()) for r in rows)
    with pytest.raises(plq.PlqError):
        ops.rope_kv_append(qkv, cos, sin, 2, 1, *rows, 4)


@pytest.mark.parametrize("kv_quant", [False, True])
def test_decoder_steps_leave_earlier_caches_alone(kv_quant):
    """A cache taken from the model before a step keeps its contents; put back, it continues from there; the appended
    cache equals the one of concatenated copies."""
    from plaquant_b200.forward_pass import LlamaConfig, ResQForwardB200
    cfg = LlamaConfig(hidden_size=512, intermediate_size=1024, num_layers=2, num_heads=4, num_kv_heads=2, head_dim=128,
                      vocab_size=300)
    ids = torch.randint(0, 300, (2, 60), generator=torch.Generator().manual_seed(3)).cuda()
    m = ResQForwardB200(cfg, "cuda", seed=4, kv_quant=kv_quant)
    m.forward(ids[:, :20])
    prompt = list(m.kv)
    m.forward(ids[:, 20:21], pos0=20)
    saved = list(m.kv)
    copies = [x.clone() for layer in prompt + saved for x in layer]
    a = m.forward(ids[:, 21:22], pos0=21)
    m.forward(ids[:, 22:23], pos0=22)
    m.kv = list(saved)
    m.forward(ids[:, 30:31], pos0=21)                                  # another continuation
    m.kv = list(saved)
    assert torch.equal(m.forward(ids[:, 21:22], pos0=21), a)
    m.forward(ids[:, 22:25], pos0=22)                                  # a chunk behind the prompt
    assert all(torch.equal(x, y) for x, y in zip(copies, (x for layer in prompt + saved for x in layer)))
    for i in range(25, 60):                                            # past the room that an append makes
        before = [x.clone() for x in m.kv[1]]
        step = m.forward(ids[:, i:i + 1], pos0=i)
        assert all(torch.equal(x[:, :i], y) for x, y in zip(m.kv[1], before))
    assert m.kv[0][0].shape[1] == 60 and torch.isfinite(step).all()
    m.kv = [tuple(x[:1] for x in layer) for layer in m.kv]
    with pytest.raises(RuntimeError):
        m.forward(ids[:, :1], pos0=60)                                 # a cache of another batch size
    plq.check_device_status()


@pytest.mark.parametrize("b,t,heads,kv,pos,ctx,t_max", [(2, 1, 4, 2, 9, 10, 10), (3, 1, 8, 1, 0, 1, 16), (2, 5, 4, 2, 0, 5, 5),
                                                       (1, 4, 6, 2, 30, 34, 60), (16, 1, 32, 8, 511, 512, 640), (2, 1, 2, 1, 5, 12, 12)])
def test_append_with_values_equals_append_then_unpack(b, t, heads, kv, pos, ctx, t_max):
    from plaquant_b200 import _lib, ops
    g = torch.Generator().manual_seed(pos)
    qkv = (torch.randn(b, t, (heads + 2 * kv) * 128, generator=g) * 2).to(torch.bfloat16).cuda()
    cos, sin = (x.cuda() for x in _tables(pos, t))
    rows = [torch.randint(0, 0x7F, (b, t_max, kv, 72), dtype=torch.uint8, generator=g).cuda() for _ in range(2)]
    want_rows = [r.clone() for r in rows]
    want_q = ops.rope_kv_append(qkv, cos, sin, heads, kv, *want_rows, pos)
    want = ops.unpack_head_rows(*want_rows, ctx)
    for at in (pos, torch.tensor([pos], device="cuda")):
        if not isinstance(at, torch.Tensor) and pos + t > ctx:
            continue
        got_rows = [r.clone() for r in rows]
        q = torch.empty(b, t, heads, 128, device="cuda")
        vals = [torch.full((b, ctx, kv, 128), 7.0, dtype=torch.bfloat16, device="cuda") for _ in range(2)]
        on_device = isinstance(at, torch.Tensor)
        _lib.check(_lib.lib().plq_rope_kv_append_nvfp4_values(
            qkv.data_ptr(), qkv.shape[-1], cos.data_ptr(), sin.data_ptr(), b, t, heads, kv, 128, q.data_ptr(), got_rows[0].data_ptr(),
            got_rows[1].data_ptr(), t_max, at.data_ptr() if on_device else None, 0 if on_device else at, ctx, vals[0].data_ptr(),
            vals[1].data_ptr(), ops.status_word("cuda").data_ptr(), torch.cuda.current_stream().cuda_stream))
        plq.check_device_status()
        assert torch.equal(q, want_q.float())
        assert all(torch.equal(x, y) for x, y in zip(got_rows, want_rows))
        assert all(torch.equal(x.view(torch.int16), y.view(torch.int16)) for x, y in zip(vals, want))
