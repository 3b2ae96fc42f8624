"""The fixed rules that choose a product's kernel from its counts (host functions of libcqb200.so, no GPU)."""
import pytest

import cq_b200

TILES, BLOCKS = 0, 1

# (pairs, useful flops, tensor flops the tiles issue, blocks of range rb) of two-part split products and the kernel that is
# faster on them (us blocks / tiles on B200)
MEASURED = {
    "c512_dzp_26_16": (33.93e6, 149.3e9, 3764e9, 63664, BLOCKS),        # 4004 / 4897
    "c512_dzp_20_20": (38.49e6, 169.2e9, 4161e9, 124000, TILES),        # 5439 / 5040
    "c1000_dzp_26_16": (66.27e6, 291.3e9, 6827e9, 124350, TILES),       # 9267 / 8615
    "c1000_dzp_26_16_t2": (66.28e6, 291.3e9, 8244e9, 124350, BLOCKS),   # 8683 / 10494
    "c1728_dzp_26_16": (114.5e6, 503.7e9, 11714e9, 214900, TILES),      # 16655 / 14643
    "c4096_dzp_26_16": (271.5e6, 1193e9, 31580e9, 509000, TILES),       # 40200 / 39500
    "k1500_dzp_22_16_t2": (33.3e6, 146.4e9, 3960e9, 141400, BLOCKS),    # 3931 / 4581
    "c216_dzp_26_16": (14.31e6, 62.9e9, 1497e9, 26830, BLOCKS),         # 1549 / 2162
    "k300_dzp_16": (1.786e6, 7.85e9, 181e9, 22140, BLOCKS),             # 236 / 270
    "k300_dzp_20": (5.681e6, 24.97e9, 446e9, 39766, TILES),             # 594 / 499
    "k300_dzp_32": (21.75e6, 95.5e9, 1030e9, 80442, TILES),             # 2387 / 1252
    "k300_mix_32": (21.75e6, 15.1e9, 302e9, 80442, TILES),              # 2318 / 470
    "k150_u16_32_t2": (3.379e6, 27.6e9, 187e9, 22510, TILES),           # 461 / 345
    "k100_dzp_20": (0.683e6, 3.0e9, 34.9e9, 8190, TILES),               # 91 / 79
    "k100_dzp_16": (0.310e6, 1.36e9, 24.3e9, 5394, BLOCKS),             # 55 / 66
    "k50_dzp_20": (0.121e6, 0.532e9, 5.7e9, 2462, BLOCKS),              # 31 / 49
    "c512_sz_26_16": (33.9e6, 4.34e9, 300e9, 63664, BLOCKS),            # fraction 0.04: below the bound of 0.11
}


@pytest.mark.parametrize("name", sorted(MEASURED))
def test_split_kernel_rule_takes_the_faster_kernel(name):
    pairs, flops, issued, b_blocks, kernel = MEASURED[name]
    assert cq_b200.split_kernel_rule(pairs, flops, issued, b_blocks) == kernel


def test_split_kernel_rule_edges():
    ok = dict(n_pairs=300000, flops=int(2e9), issued_flops=2e9, b_blocks=1000)
    assert cq_b200.split_kernel_rule(**ok) == TILES           # 40 + 2.6 us against 18 + 33.6
    assert cq_b200.split_kernel_rule(**{**ok, "n_pairs": 299999}) == BLOCKS             # no estimate is made of fewer pairs
    assert cq_b200.split_kernel_rule(**{**ok, "flops": int(1e12), "issued_flops": 10e9}) == BLOCKS   # 40 + 12.8 us
    assert cq_b200.split_kernel_rule(**{**ok, "issued_flops": 0.0}) == BLOCKS           # nothing known of the tiles
    assert cq_b200.split_kernel_rule(**{**ok, "flops": int(0.109 * 2e9 / 3)}) == BLOCKS
    assert cq_b200.split_kernel_rule(**{**ok, "flops": int(0.111 * 2e9 / 3)}) == TILES
    with pytest.raises(cq_b200.CQError):
        cq_b200.split_kernel_rule(-1, 0, 0.0, 0)
