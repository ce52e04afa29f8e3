"""Which prompts the tcgen05 attention kernel takes: the library's own answer, a host function that follows no pointer."""
import ctypes as C

import pytest

from tensorsharp_b200.ops import kernels as K
from tensorsharp_b200.ops import native

pytestmark = pytest.mark.skipif(not native.available(), reason="the kernel library is not built here")


def takes(cache_rows=4096, max_q=1000, **kw):
    a = K.AttnArgs()
    plain = dict(q=1 << 20, k_cache=2 << 20, v_cache=3 << 20, out=4 << 20, block_table=5 << 20, kv_lens=6 << 20, cu_q=7 << 20, scale=0.1, B=2, Hq=8,
                 Hkv=2, Dh=128, Dv=128, page_size=64, max_pages=40, splits=1)
    for k, v in {**plain, **kw}.items():
        setattr(a, k, v)
    return bool(K._lib().tsb_attn_prefill_tc_takes(C.byref(a), C.c_int(max_q), C.c_long(cache_rows)))


@pytest.mark.parametrize("Dh", [64, 128, 256])
def test_plain_forms(Dh):
    assert takes(Dh=Dh, Dv=Dh) and takes(Dh=Dh, Dv=0, page_size=256, window=100, sinks=1 << 22, softcap=30.0) and takes(Dh=Dh, Dv=Dh, gate=1 << 22, gate_tok=8)


@pytest.mark.parametrize("name", ["q", "k_cache", "v_cache", "out"])
@pytest.mark.parametrize("off", [2, 4, 8])
def test_every_pointer_on_sixteen_bytes(name, off):
    assert not takes(**{name: (1 << 20) + off}) and takes(**{name: (1 << 20) + 16})


@pytest.mark.parametrize("kw", [dict(Dh=512, Dv=512), dict(Dh=96, Dv=96), dict(Dv=64), dict(page_size=16), dict(page_size=96), dict(cache_rows=32), dict(k_ld=2048),
                                dict(v_ld=2048), dict(q_pos0=64), dict(lse_out=64), dict(keep_first=4), dict(slopes=64), dict(gate=64, gate_cols=1),
                                dict(kv_scale=256), dict(log_r1=64), dict(sig_bias=64)])
def test_what_stays_with_the_other_kernels(kw):
    assert not takes(**kw)


def test_smallest_prompts_and_small_capped_grids():
    """The lines of the rule: 64 slots, 256 heads of all prompts together, 72 CTAs (at two heads a tile 64 tokens each)."""
    tiny = dict(Dh=64, Dv=64, max_pages=1, max_q=40)
    assert not takes(**tiny) and takes(**{**tiny, "max_pages": 2}) and takes(**{**tiny, "B": 32}) and not takes(**{**tiny, "B": 31})
    assert not takes(**{**tiny, "B": 32, "Hkv": 8}) and takes(**{**tiny, "Dh": 128, "Dv": 128}) and takes(**{**tiny, "Dh": 256, "Dv": 256})
    cap = dict(Dh=64, Dv=64, softcap=30.0, Hq=4, Hkv=2, B=1)
    assert not takes(max_q=35 * 64, **cap) and takes(max_q=35 * 64 + 1, **cap) and takes(max_q=64, **{**cap, "softcap": 0.0})
    assert not takes(Dh=128, softcap=30.0, max_pages=1) and takes(Dh=128, softcap=30.0, max_pages=2)


def test_single_heads_of_64_on_two_pages():
    """One head per row tile: 65 to 128 tokens up to 74 CTAs, at most 64 tokens beyond 296, both up to 128 slots."""
    one = dict(Dh=64, Dv=64, Hq=10, Hkv=2, max_pages=2)
    assert not takes(max_q=65, **one, B=7) and takes(max_q=64, **one, B=7) and takes(max_q=65, **one, B=8) and takes(max_q=65, **{**one, "max_pages": 3}, B=7)
    assert not takes(max_q=64, **one, B=30) and takes(max_q=64, **one, B=29) and takes(max_q=65, **one, B=30) and takes(max_q=64, **{**one, "max_pages": 3}, B=30)
    assert takes(max_q=65, **{**one, "Hq": 8}, B=7) and takes(max_q=65, **{**one, "Dh": 128, "Dv": 128}, B=7)


def test_a_whole_library_without_the_kernel_is_refused(monkeypatch):
    """An old build is an error, not the slower kernel; a library of selected sources may lack it."""
    class Old:
        pass
    old = Old()
    monkeypatch.setattr(K, "_configured", False)
    monkeypatch.setattr(K, "_prefill_tc", True)
    monkeypatch.setattr(native, "lib", lambda: old)
    old._name = str(native.LIB_PATH)
    with pytest.raises(native.NativeLibraryError, match="build it again"):
        K._lib()
    old._name = str(native.OUT_DIR / "libtsb200-part-0.so")
    assert K._lib() is old and K._prefill_tc is False
