"""Which form of the causal attention forward a launch takes: a team per item, or items shared by the two teams of a CTA."""
import pytest

from torchmpi_b200._lib import has_symbol, lib

pytestmark = pytest.mark.skipif(not has_symbol("tmpi_attention_fwd_shares"), reason="built without the CUDA kernels")
SMS = 148                                                  # of the chip, and what the library assumes without one


def _busiest(per_block, q_blocks, units, shared):
    """Time of the busiest team or CTA, in twentieths of a key block, item by item in the order in which the kernel deals them."""
    loads, t = [0] * units, 0
    for t in range(per_block * q_blocks):
        r, i = divmod(t, units)
        blocks = q_blocks - t // per_block
        loads[units - 1 - i if r & 1 else i] += (blocks + 1) // 2 * 20 + (40 if blocks > 1 else 20) if shared else 18 * blocks + 40
    return max(loads)


@pytest.mark.parametrize("q_blocks", [1, 2, 3, 4, 5, 7, 8, 13, 16, 20, 32])
def test_form_follows_the_busiest_unit(q_blocks):
    for per_block in [*range(1, 60), 64, 74, 96, 128, 148, 149, 192, 300]:
        items = per_block * q_blocks
        grid = min(items, SMS)
        want = q_blocks > 1 and items <= 4 * grid and _busiest(per_block, q_blocks, grid, True) < _busiest(per_block, q_blocks, 2 * grid, False)
        assert bool(lib.tmpi_attention_fwd_shares(per_block, 128 * q_blocks, 1)) == want, (per_block, q_blocks)


# heads x batch, key blocks: both forms measured, the faster one
@pytest.mark.parametrize("per_block,q_blocks,shares", [(64, 3, False), (52, 4, False), (27, 13, False), (20, 20, False), (16, 24, False),
                                                       (32, 10, False), (48, 5, False), (12, 32, False), (74, 1, False), (128, 8, False), (1, 2, True), (74, 2, True),
                                                       (16, 16, True), (12, 20, True), (37, 8, True), (24, 12, True), (1, 32, True)])
def test_form_at_measured_sizes(per_block, q_blocks, shares):
    assert bool(lib.tmpi_attention_fwd_shares(per_block, 128 * q_blocks, 1)) == shares


def test_form_of_many_items_is_a_team_each():
    assert not lib.tmpi_attention_fwd_shares(1 << 20, 1024, 16)
    assert not lib.tmpi_attention_fwd_shares(1 << 15, 1 << 17, 1024)
    assert not lib.tmpi_attention_fwd_shares(0, 1024, 16)
