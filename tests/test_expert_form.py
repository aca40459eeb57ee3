"""Which form of the decode experts a block of rows takes where activations stay f16 (no GPU needed)."""
from types import SimpleNamespace

import pytest

from titanic_flash_41_b200.config import EngineConfig, reference_1017_config
from titanic_flash_41_b200.models.engine import Engine


@pytest.mark.parametrize("T,over,ranks,on,want", [
    (1, {}, 1, True, True), (24, {}, 1, True, True), (32, {}, 1, True, True), (33, {}, 1, True, False),
    (24, {}, 1, False, False),                                       # not wanted
    (32, dict(n_experts=96), 1, True, True), (32, dict(n_experts=95), 1, True, False),      # two rows an expert on average
    (24, dict(moe_inter=2200), 1, True, False),                      # not in whole 256 inputs
    (1, dict(hidden=512, moe_inter=256), 1, True, False),            # little to stream
    (1, dict(topk=3), 1, True, True), (1, dict(topk=2), 1, True, False),                    # 53 and 35 MB
    (1, {}, 2, True, True), (1, {}, 4, True, False),                 # half and a quarter of 106 MB a rank
])
def test_rule_of_the_split_form(T, over, ranks, on, want):
    cfg = reference_1017_config(**over)
    eng = SimpleNamespace(cfg=cfg, ecfg=EngineConfig(moe_block_scaled=on), SMALL_M=Engine.SMALL_M, El=cfg.n_experts // ranks, world=ranks)
    assert Engine._moe_split_ok(eng, T) == want
