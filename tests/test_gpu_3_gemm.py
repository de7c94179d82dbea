"""Fused mixed GEMM (tcgen05, through the C ABI) against the CPU oracle's
dequantise-then-float32-matmul.  Tolerance: rel-L2 <= 1e-3 measured in the output dtype (the
oracle's float32 product is rounded to bf16 before comparing; bf16 rounding alone is 1.6e-3
against an unrounded float32 product)."""
import os

import numpy as np
import pytest
import torch

from oracle import formats as F
from tests._util import bits_of, f32_of, from_bits, packed_to_numpy, rel_l2, synth_activation, synth_weight

pytestmark = pytest.mark.gpu
plq = pytest.importorskip("plaquant_b200")

TOL = 1e-3
VARIANTS = ["128x128", "128x256", "pair256x256"]


def _to_device(pd: dict, layout: str):
    """oracle dict -> PackedMatrix on the GPU (used to feed hand-made codes to the kernel)."""
    rows, k_lo, k_hi = pd["rows"], pd["k_lo"], pd["k_hi"]
    lay = 1 if layout == "tiled" else 0
    def sf(a, n):
        if n == 0:
            return torch.zeros(0, dtype=torch.uint8, device="cuda")
        return torch.from_numpy(F.tile_sf(a) if lay else np.ascontiguousarray(a)).cuda()
    return plq.PackedMatrix(rows, k_lo, k_hi, torch.from_numpy(pd["lo_codes"]).cuda().contiguous(),
                            sf(pd["lo_sf"], k_lo // 16), torch.from_numpy(pd["hi_codes"]).cuda().contiguous(),
                            sf(pd["hi_sf"], k_hi // 32), lay)


def _oracle_bf16(pa: dict, pb: dict) -> np.ndarray:
    return F.round_to_bf16(F.linear(pa, pb))


def _run(pa_dev, pb_dev, variant):
    y = plq.mixed_gemm(pa_dev, pb_dev, variant=variant)
    plq.check_device_status()
    return f32_of(y)


@pytest.mark.parametrize("variant", VARIANTS)
def test_known_answer_all_ones(variant):
    """Codes 1.0, scales 1.0: every output equals K.  Catches descriptor / pipeline errors."""
    m, n, k_lo, k_hi = 128, 256, 512, 128
    pa = {"rows": m, "k_lo": k_lo, "k_hi": k_hi, "lo_codes": np.full((m, k_lo // 2), 0x22, np.uint8),
          "lo_sf": np.full((m, k_lo // 16), 0x38, np.uint8), "hi_codes": np.full((m, k_hi), 0x38, np.uint8),
          "hi_sf": np.full((m, k_hi // 32), 127, np.uint8)}
    pb = {**pa, "rows": n, "lo_codes": np.full((n, k_lo // 2), 0x22, np.uint8),
          "lo_sf": np.full((n, k_lo // 16), 0x38, np.uint8), "hi_codes": np.full((n, k_hi), 0x38, np.uint8),
          "hi_sf": np.full((n, k_hi // 32), 127, np.uint8)}
    y = _run(_to_device(pa, "tiled"), _to_device(pb, "tiled"), variant)
    assert np.array_equal(y, np.full((m, n), float(k_lo + k_hi), np.float32))


@pytest.mark.parametrize("variant", VARIANTS)
def test_known_answer_layout_probes(variant):
    """Row-, column-, K- and scale-dependent patterns with exactly representable results, so any
    permutation of rows, columns, K blocks, nibbles or scale bytes shows up as a wrong integer."""
    rng = np.random.default_rng(5)
    m, n, k_lo, k_hi = 256, 512, 768, 256
    def mk(rows):
        lo = rng.integers(0, 16, (rows, k_lo), dtype=np.uint8)
        hi_mag = rng.integers(0x30, 0x48, (rows, k_hi), dtype=np.uint8)      # 0.5 .. 3.75
        hi = hi_mag | (rng.integers(0, 2, (rows, k_hi), dtype=np.uint8) << 7)
        return {"rows": rows, "k_lo": k_lo, "k_hi": k_hi, "lo_codes": F.pack_nibbles(lo),
                "lo_sf": rng.integers(0x30, 0x41, (rows, k_lo // 16), dtype=np.uint8),   # 0.5 .. 2.0
                "hi_codes": hi, "hi_sf": rng.integers(124, 131, (rows, k_hi // 32), dtype=np.uint8)}
    pa, pb = mk(m), mk(n)
    want = F.linear(pa, pb)
    y = _run(_to_device(pa, "tiled"), _to_device(pb, "tiled"), variant)
    assert rel_l2(y, F.round_to_bf16(want)) <= TOL


@pytest.mark.parametrize("m,n,k,k_hi", [
    (128, 128, 256, 0), (128, 256, 256, 128), (7, 136, 192, 64), (129, 8, 128, 64), (300, 392, 1024, 448),
    (64, 264, 128, 128), (16, 4096, 4096, 128), (130, 640, 14336, 448),
])
@pytest.mark.parametrize("variant", VARIANTS)
def test_random_shapes_against_oracle(m, n, k, k_hi, variant):
    x = synth_activation(m, k, seed=m + k)
    w = synth_weight(n, k, seed=n + k + 1)
    had = k % 128 == 0
    pa = plq.pack(x.cuda(), k_hi, hadamard=had, sf_layout="tiled")
    pb = plq.pack(w.cuda(), k_hi, hadamard=had, sf_layout="tiled")
    y = _run(pa, pb, variant)
    want = _oracle_bf16(packed_to_numpy(pa), packed_to_numpy(pb))
    r = rel_l2(y, want)
    assert r <= TOL, r


def test_config0_single_linear_against_reference_fixture(golden_dir):
    """X [16,4096] x W [4096,4096], block-Hadamard 128 on both, K = 3968 NVFP4 + 128 MXFP8;
    compared with the reference's own fake-quant product (float32 matmul, rounded to bf16)."""
    g = np.load(os.path.join(golden_dir, "linear_cfg0.npz"))
    w = synth_weight(4096, 4096, seed=1)
    assert int(bits_of(w).astype(np.uint64).sum()) == int(g["w_checksum"])
    pa = plq.pack(from_bits(g["x"]), 128, hadamard=True, sf_layout="tiled")
    pb = plq.pack(w.cuda(), 128, hadamard=True, sf_layout="tiled")
    y = f32_of(plq.mixed_gemm(pa, pb))
    plq.check_device_status()
    ref = F.round_to_bf16(g["y_f32"])
    r = rel_l2(y, ref)
    # the rotation's float32 summation order differs from torch's (a bf16 ulp on a small share of the rotated
    # inputs), which could move a code.  The measured value and the number of codes that moved against the
    # reference's own rotated activations are printed (measured on B200: 3.1e-4 and 0 of 65536).
    ref_codes = F.pack_mixed(F.bf16_bits_to_f32(g["xr"]), 128)
    mine = packed_to_numpy(pa)
    moved = int((F.unpack_nibbles(mine["lo_codes"]) != F.unpack_nibbles(ref_codes["lo_codes"])).sum()) + \
        int((mine["hi_codes"] != ref_codes["hi_codes"]).sum())
    print(f"config 0 end to end: rel-L2 {r:.3e} against the reference's product; {moved} of {16 * 4096} activation "
          f"codes differ from those of the reference's rotated input")
    assert r <= TOL, r
    # with the reference's own rotated activations the input-side slack disappears
    pa2 = plq.pack(from_bits(g["xr"]), 128, hadamard=False, sf_layout="tiled")
    want = _oracle_bf16(packed_to_numpy(pa2), packed_to_numpy(pb))
    assert rel_l2(f32_of(plq.mixed_gemm(pa2, pb)), want) <= TOL


@pytest.mark.parametrize("m", [512, 2048, 8192])
@pytest.mark.parametrize("n,k", [(6144, 4096), (4096, 4096), (28672, 4096), (4096, 14336)])
def test_prefill_full_size_properties(n, k, m):
    """M = 512, 2048, 8192 on the four Llama-3-8B shapes, tile shape chosen by the library (the down projection
    at M = 8192 runs the banded tile order): sampled rows against the oracle, identical rows whatever the M they
    are computed in (tiles are independent), determinism, clean status."""
    k_hi = k // 32
    x = synth_activation(m, k, seed=3000)
    w = synth_weight(n, k, seed=3001)
    pa = plq.pack(x.cuda(), k_hi, hadamard=True, sf_layout="tiled")
    pb = plq.pack(w.cuda(), k_hi, hadamard=True, sf_layout="tiled")
    y1 = plq.mixed_gemm(pa, pb, variant=None)
    y2 = plq.mixed_gemm(pa, pb, variant=None)
    plq.check_device_status()
    assert torch.equal(y1, y2)
    sel = np.sort(np.random.default_rng(1).choice(m, 12, replace=False))
    na, nb = packed_to_numpy(pa), packed_to_numpy(pb)
    sub = {**na, "rows": len(sel), **{key: na[key][sel] for key in ("lo_codes", "lo_sf", "hi_codes", "hi_sf")}}
    want = _oracle_bf16(sub, nb)
    assert rel_l2(f32_of(y1)[sel], want) <= TOL
    ps = plq.pack(x[:256].cuda(), k_hi, hadamard=True, sf_layout="tiled")
    assert torch.equal(plq.mixed_gemm(ps, pb), y1[:256])


@pytest.mark.parametrize("n,k", [(4096, 4096), (4096, 14336)])
def test_full_size_chain_from_bf16_against_oracle(n, k):
    """The whole chain at full K: bf16 X and W -> QuantizedLinear (rotation, quantiser, packed GEMM) -> y, against
    the oracle computed from the same bf16 tensors (its own rotation and quantiser, float32 product): sampled
    token rows x sampled output rows, prefill (M = 2048, GEMM) and decode (M = 8, tensor-core GEMV)."""
    from plaquant_b200.quantize import QuantizedLinear
    k_hi = k // 32
    x = synth_activation(2048, k, seed=4100 + k)
    w = synth_weight(n, k, seed=4200 + n)
    lin = QuantizedLinear.from_weight(w.cuda(), 1.0 / 32, rotate=True, online_had=True)
    rows = np.sort(np.random.default_rng(3).choice(2048, 10, replace=False))
    cols = np.sort(np.random.default_rng(4).choice(n, 96, replace=False))
    want_x = F.prepare_activation(f32_of(x)[rows], k_hi, hadamard=True)
    want_w = F.prepare_activation(f32_of(w)[cols], k_hi, hadamard=True)
    want = F.round_to_bf16(F.linear(want_x, want_w))
    y = f32_of(lin(x.cuda()))
    plq.check_device_status()
    r = rel_l2(y[np.ix_(rows, cols)], want)
    assert r <= TOL, r
    y8 = f32_of(lin(x[rows[:8]].cuda()))
    plq.check_device_status()
    r8 = rel_l2(y8[:, cols], want[:8])
    assert r8 <= TOL, r8


def test_argument_errors():
    x = synth_activation(16, 256, seed=1).cuda()
    pa = plq.pack(x, 64, sf_layout="tiled")
    pb = plq.pack(x, 64, sf_layout="rowmajor")
    with pytest.raises(ValueError):
        plq.mixed_gemm(pa, pb)                      # weights in the wrong scale layout
    pb = plq.pack(x[:12], 64, sf_layout="tiled")     # N = 12 is not a multiple of 8
    with pytest.raises(plq.PlqError) as e:
        plq.mixed_gemm(pa, pb)
    assert e.value.status == -2


# A last wave of at most half the pairs is worked on in half tiles: a lone tile (all of it halved; n that ends in its first
# half, at its edge, in its second half), rows past one CTA, whole waves with a few tiles left (74 pairs on 148 SMs: 76,
# 150 and 224 tiles); k: ragged last stages of both formats, one format only, more stages than the ring
@pytest.mark.parametrize("m,n,k,k_hi", [(1, 8, 128, 64), (77, 128, 1024, 64), (129, 136, 192, 64), (256, 256, 512, 128),
                                        (300, 640, 384, 384), (333, 392, 14336, 448), (100, 19456, 256, 64), (300, 19208, 448, 0),
                                        (333, 28672, 1024, 64)])
def test_half_tiles_of_the_last_wave_equal_other_tile_shapes(m, n, k, k_hi):
    x, w = synth_activation(m, k, seed=m + k).cuda(), synth_weight(n, k, seed=n + k + 1).cuda()
    had = k % 128 == 0
    pa, pb = (plq.pack(t, k_hi, hadamard=had, sf_layout="tiled") for t in (x, w))
    y = _run(pa, pb, "pair256x256")
    assert np.array_equal(y, _run(pa, pb, "128x128"))              # the same K order: the same bits
    assert np.array_equal(y, _run(pa, pb, None))
    if n < 1000:
        assert rel_l2(y, _oracle_bf16(packed_to_numpy(pa), packed_to_numpy(pb))) <= TOL


# m: one row, past a CTA, past a pair, several row tiles, one wave and more; n: one tile and several; k: ragged last stages
# of both formats, one format only, more stages than the ring
@pytest.mark.parametrize("m,n,k,k_hi", [(1, 128, 128, 64), (17, 256, 1024, 64), (129, 128, 192, 64), (300, 384, 384, 384),
                                        (333, 512, 14336, 448), (1000, 256, 448, 0), (77, 14336, 512, 64), (600, 9728, 256, 64)])
def test_silu_mul_in_the_epilogue_equals_gemm_and_silu_prologue(m, n, k, k_hi):
    x, w = synth_activation(m, k, seed=m + k).cuda(), synth_weight(2 * n, k, seed=n + k).cuda() * 4
    x[0, :2] = 1e4                                                     # some gates far out on both sides
    had = k % 128 == 0
    pa, pb = (plq.pack(t, k_hi, hadamard=had, sf_layout="tiled") for t in (x, w))
    from plaquant_b200 import ops
    got = ops.mixed_gemm_silu_mul(pa, pb)
    plq.check_device_status()
    gu = f32_of(plq.mixed_gemm(pa, pb))
    want = F.silu_mul_bf16(gu[:, :n], gu[:, n:])
    assert np.array_equal(f32_of(got), want)
    with pytest.raises(plq.PlqError):                                  # up rows inside a 128-row group of scales
        ops.mixed_gemm_silu_mul(pa, plq.pack(w[:208], k_hi, hadamard=had, sf_layout="tiled"))
