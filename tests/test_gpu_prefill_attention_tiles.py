"""The two prefill attention kernels by themselves, with their sums before the rounding to bf16: the tensor-core kernel
against 64 bits and against the fp32 row kernel at the edges of its tiles (16 rows per warp, 64 rows per CTA, 64 keys per
tile), behind keys of earlier pieces, and with infinities and NaN in queries, keys and values."""
import ctypes
import math

import numpy as np
import pytest

import native_build

pytestmark = pytest.mark.gpu

HEADS = [(64, 4, 2), (64, 2, 2), (128, 4, 1), (128, 2, 2)]


@pytest.fixture(scope="module")
def attention(qmm_lib):
    import torch
    lib = native_build.load("attn_prefill", device_code=True)
    fn = lib.attn_prefill_f32
    fn.argtypes = [ctypes.c_int, ctypes.c_void_p] + [ctypes.c_int] * 5 + [ctypes.c_void_p] * 3 + [ctypes.c_int, ctypes.c_void_p]

    def run(rows_kernel, qkv, keys, values, heads, pos0):
        m, (n_kv, max_seq, hd) = qkv.shape[0], keys.shape
        ctx = torch.full((m + 1, heads * hd), 7.0, device="cuda")
        assert fn(hd, qkv.data_ptr(), m, pos0, heads, n_kv, max_seq, keys.data_ptr(), values.data_ptr(), ctx.data_ptr(),
                  m if rows_kernel else 0, torch.cuda.current_stream().cuda_stream) == 0
        torch.cuda.synchronize()
        assert bool((ctx[m] == 7.0).all())
        return ctx[:m]
    return run


def inputs(m, pos0, head_dim, heads, kv_heads, spread, seed):
    import torch
    gen = torch.Generator(device="cuda")
    gen.manual_seed(seed)
    max_seq = pos0 + m + 5
    qkv = torch.randn(m, (heads + 2 * kv_heads) * head_dim, device="cuda", generator=gen) * spread
    keys, values = (torch.randn(kv_heads, max_seq, head_dim, device="cuda", generator=gen).half() for _ in range(2))
    keys[:, pos0 + m:] = float("nan")    # what lies behind the last position is nobody's business
    values[:, pos0 + m:] = float("nan")
    return qkv, keys, values


def in_64_bits(qkv, keys, values, heads, pos0):
    import torch
    m, (kv_heads, _, hd) = qkv.shape[0], keys.shape
    n = pos0 + m
    hidden = torch.arange(n, device="cuda")[None] > pos0 + torch.arange(m, device="cuda")[:, None]
    out = torch.empty(m, heads, hd, dtype=torch.float64, device="cuda")
    for h in range(heads):
        kv = h // (heads // kv_heads)
        s = qkv[:, h * hd:(h + 1) * hd].double() @ keys[kv, :n].double().T / math.sqrt(hd)
        out[:, h] = torch.softmax(s.masked_fill(hidden, -math.inf), -1) @ values[kv, :n].double()
    return out.view(m, heads * hd)


def rel(got, want):
    return float((got.double() - want).norm() / want.norm())


# spread: scores of about one, and of about sixteen, where an error of a score shows sixteen times as much
@pytest.mark.parametrize("spread", [1.0, 16.0])
@pytest.mark.parametrize("head_dim,heads,kv_heads", HEADS)
@pytest.mark.parametrize("m,pos0", [(1, 0), (15, 1), (16, 63), (17, 64), (63, 0), (64, 65), (65, 0), (129, 62), (200, 157)])
def test_tiles_match_64_bits(attention, m, pos0, head_dim, heads, kv_heads, spread):
    qkv, keys, values = inputs(m, pos0, head_dim, heads, kv_heads, spread, seed=m + pos0)
    got = attention(False, qkv, keys, values, heads, pos0)
    # a score carries some 2^-24 of its size (up to five times the spread), exp two units more; half of a query's bits
    # lost would show as 2^-12 of the score
    assert rel(got, in_64_bits(qkv, keys, values, heads, pos0)) <= 2.0 ** -24 * (8.0 + 5.0 * spread)


@pytest.mark.parametrize("spread", [0.25, 1.0, 4.0, 16.0])
@pytest.mark.parametrize("head_dim", [64, 128])
@pytest.mark.parametrize("m,pos0", [(300, 0), (257, 700), (1999, 0)])
def test_tiles_lose_nothing_against_fp32_rows(attention, m, pos0, head_dim, spread):
    qkv, keys, values = inputs(m, pos0, head_dim, 4, 4, spread, seed=3)
    want = in_64_bits(qkv, keys, values, 4, pos0)
    tiles, rows = (rel(attention(r, qkv, keys, values, 4, pos0), want) for r in (False, True))
    assert tiles <= rows, (tiles, rows)


@pytest.mark.parametrize("head_dim,heads,kv_heads", HEADS)
@pytest.mark.parametrize("what,value", [("v", math.inf), ("v", math.nan), ("k", -math.inf), ("k", math.inf), ("k", math.nan),
                                        ("q", math.inf), ("q", math.nan), ("q", 3e38)])
def test_infinities_reach_the_rows_that_see_them(attention, what, value, head_dim, heads, kv_heads):
    """Row by row what the fp32 row kernel gives: a key or value hides from the rows before it, a key of -inf weighs
    nothing."""
    m, pos0, at = 150, 70, 40
    qkv, keys, values = inputs(m, pos0, head_dim, heads, kv_heads, 1.0, seed=11)
    if what == "q":
        qkv[at, 5] = value
    elif what == "k":
        qkv[:, 7:heads * head_dim:head_dim] = qkv[:, 7:heads * head_dim:head_dim].abs() + 0.1  # the same sign in every row
        keys[0, pos0 + at, 7] = value
    else:
        values[0, pos0 + at, 7] = value
    tiles, rows = (attention(r, qkv, keys, values, heads, pos0).cpu().numpy() for r in (False, True))
    assert np.array_equal(np.isnan(tiles), np.isnan(rows)) and np.array_equal(np.isinf(tiles), np.isinf(rows))
    ok = np.isfinite(rows)
    assert ok[:at].all()
    assert np.abs(tiles[ok] - rows[ok]).max() <= 1e-5 * np.abs(rows[ok]).max()
