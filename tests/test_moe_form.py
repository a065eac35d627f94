"""Which kernel a mixture-of-experts stage runs on: a pure host function."""

import pytest

from flydsl_b200 import _lib

TWO_TILES, ONE_CTA, PAIRS = 1, 2, 3


@pytest.mark.parametrize(
    "tokens,topk,experts,model,inter,tile_m,forms",
    [  # forms of the gate-up and of the down stage; both measured, us (one CTA / pairs)
        (4096, 2, 8, 4096, 2048, 128, (PAIRS, PAIRS)),  # 128 / 122, 74 / 67
        (800, 4, 32, 3072, 1536, 64, (PAIRS, PAIRS)),  # 91 / 65, 48 / 41
        (515, 4, 16, 2048, 1408, 64, (PAIRS, PAIRS)),  # 32.6 / 30.7, 24.4 / 21.0
        (1024, 4, 8, 2048, 1024, 64, (PAIRS, ONE_CTA)),  # 27.7 / 24.7, 19.2 / 20.0
        (4096, 4, 32, 2048, 768, 128, (PAIRS, ONE_CTA)),  # 64.1 / 63.1, 43.0 / 51.2
        (32, 2, 8, 4096, 2048, 16, (TWO_TILES, TWO_TILES)),  # other routing blocks have a kernel of their own
    ],
)
def test_measured_sizes(tokens, topk, experts, model, inter, tile_m, forms):
    assert tuple(_lib.moe_form(s, tokens, topk, experts, model, inter, tile_m) for s in (1, 2)) == forms


@pytest.mark.parametrize(
    "tokens,topk,local,experts,model,inter",
    [  # one CTA / pairs, us
        (74, 8, 4, 16, 2048, 3712),  # 21.1 / 29.7
        (313, 8, 16, 64, 1280, 3072),  # 31.8 / 45.6
        (890, 4, 32, 128, 1280, 2304),  # 36.4 / 48.1
        (6692, 1, 64, 128, 1280, 1024),  # 46.4 / 62.3
    ],
)
def test_a_ranks_share_of_the_experts_gets_its_share_of_the_routes(tokens, topk, local, experts, model, inter):
    assert _lib.moe_form(1, tokens, topk, local, model, inter, 64, all_experts=experts) == ONE_CTA
    assert _lib.moe_form(1, tokens, topk, local, model, inter, 64) == PAIRS  # as many routes on these experts alone


def test_longer_lists_than_the_pair_form_holds():
    assert _lib.moe_form(1, 100000, 4, 8, 4096, 2048, 64) == PAIRS  # 6258 routing blocks
    assert _lib.moe_form(1, 120000, 4, 8, 4096, 2048, 64) == ONE_CTA  # 7508; the list has room for 7168


def test_arguments_out_of_range():
    assert _lib.moe_form(3, 64, 2, 8, 512, 512, 64) == 0 and _lib.moe_form(1, 64, 2, 8, 512, 512, 24) == 0
    assert _lib.moe_form(1, 64, 2, 8, 512, 512, 64, all_experts=4) == 0


def test_the_layer_tells_its_stages_how_many_experts_all_ranks_have():
    from flydsl_b200.expert_parallel import ExpertParallelMoe

    layer = ExpertParallelMoe(model_dim=256, inter_dim=128, experts=16, topk=2, rank=1, world=4)
    assert layer._g1.experts == layer._g2.experts == 4 and layer._g1.all_experts == layer._g2.all_experts == 16
