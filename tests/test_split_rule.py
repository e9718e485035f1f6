"""How many blocks share a tile of the 32-bit product in parts, on devices of every size (the rule alone, on the host)."""
import pytest

from burn_transformers_b200 import kernels


@pytest.mark.parametrize("sms", list(range(1, 65)) + [78, 108, 132, 148, 160])
def test_blocks_a_tile(sms):
    blocks = kernels.library().bt_linear_split_blocks
    for m in (1, 128, 129, 804, 16384):
        for n, k in ((256, 768), (768, 3072), (2048, 2048)):
            tiles, k_blocks = -(-m // 128) * -(-n // 64), -(-k // 64)
            costs = {}
            for s, places in ((1, sms), (2, sms // 2), (4, sms // 4 - 5), (8, sms // 8 - 4)):
                if places >= 1:
                    rounds = -(-tiles // places)
                    costs[s] = 2500 + (1500 if s > 1 else 0) + rounds * (-(-k_blocks // s) * 1350 + (3000 if s > 1 and rounds > 1 else 0))
            assert blocks(m, n, k, sms) == min(costs, key=lambda s: (costs[s], s))
