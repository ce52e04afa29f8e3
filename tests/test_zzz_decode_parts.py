"""How decode attention cuts the sequences of a merged step (csrc/attn_args.cuh): the plan on the host (csrc/tests/parts_check.cu), and who asks for it."""
import subprocess
from types import SimpleNamespace

import pytest

from tensorsharp_b200.ops import functional as F
from tensorsharp_b200.ops import native


def test_the_plan_covers_and_fits():
    exe = str({p.name: p for p in native.build_tests()}["parts_check"])
    p = subprocess.run([exe], capture_output=True, text=True, timeout=120)
    assert p.returncode == 0 and p.stdout.startswith("OK"), p.stdout


@pytest.mark.parametrize("B,Hkv,longest,window,cut", [(1, 8, 32000, 0, None), (16, 8, 2048, 0, (85, 3)), (32, 8, 4096, 0, (101, 2)), (64, 8, 1024, 0, (101, 1)),
                                                      (64, 8, 1024, 128, None), (2, 1, 129, 0, (424, 64)), (3, 64, 128, 0, None), (4, 500, 4000, 1024, (5, 1))])
def test_parts_go_by_the_number_of_sequences(B, Hkv, longest, window, cut):
    assert F.decode_parts(SimpleNamespace(B=B, max_kv_len=longest), Hkv, window) == cut
    assert cut is None or F.decode_parts(SimpleNamespace(B=B, max_kv_len=8 * longest), Hkv, window) == cut
