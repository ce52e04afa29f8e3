"""Where MXFP4 experts go: to the tensor cores, or to the kernels that took them before, whichever is the faster one for their number and size."""
from types import SimpleNamespace

import pytest

from tensorsharp_b200.ops import functional as F

PAIRS = (8, 16, 24, 32, 48, 64, 128, 512, 1024)
# (experts, width, width of an expert) -> us of a layer by so many pairs: the GEMV of a pair each up to 64, tiles of eight and sixteen above; tensor cores
MEASURED = {
    (32, 2880, 2880): [(70, 84), (121, 120), (172, 143), (222, 149), (326, 180), (425, 167), (232, 210), (390, 233), (622, 268)],
    (8, 4096, 4096): [(103, 96), (192, 129), (278, 132), (363, 132), (537, 136), (712, 136), (241, 140), (696, 276), (1266, 457)],
    (128, 2048, 768): [(32, 45), (47, 52), (61, 60), (74, 68), (103, 85), (131, 96), (135, 125), (198, 184), (224, 205)],
    (64, 1024, 512): [(24, 34), (32, 35), (38, 37), (44, 37), (58, 39), (71, 48), (47, 53), (68, 66), (90, 78)],
    (16, 512, 256): [(19, 29), (23, 29), (27, 29), (30, 30), (37, 31), (43, 31), (31, 33), (40, 46), (51, 57)],
}


@pytest.mark.parametrize("E,D,width", list(MEASURED))
def test_no_slower_than_the_other_kernels(E, D, width):
    gate_up, down = SimpleNamespace(N=2 * width, K=D, experts=E), SimpleNamespace(N=D, K=width, experts=E)
    for pairs, (others, tensor) in zip(PAIRS, MEASURED[E, D, width]):
        took = tensor if F.expert_blocks(pairs, gate_up, down) else others
        assert took <= others and took <= 1.08 * min(others, tensor), pairs
