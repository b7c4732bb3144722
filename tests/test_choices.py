"""Which kernel a call takes, where that depends on sizes alone (no GPU)."""
from types import SimpleNamespace

import pytest
import torch

from lastengine_b200.ops import kernels


def test_pairs_take_many_rows_of_large_or_long_products():
    assert not kernels.pairs_take(1023, 8192, 8192)                        # too few rows, whatever the matrix
    assert kernels.pairs_take(1024, 4096, 64) and kernels.pairs_take(1024, 64, 4096)
    assert kernels.pairs_take(4096, 2048, 1024)                             # 128 tiles of a long K
    assert not kernels.pairs_take(4096, 2048, 1016)                         # ... of a short one
    assert not kernels.pairs_take(3840, 2048, 2048)                         # 120 tiles
    assert kernels.pairs_take(6144, 2048, 128) and not kernels.pairs_take(6143, 2048, 128)     # 192 whole tiles, whatever K
    assert not kernels.pairs_take(32768, 257, 256)                          # 256 tiles, half of them columns that are not there


@pytest.mark.parametrize("heads,seqs,length,pieces", [(16, 8, 64, 1), (16, 8, 65, 1), (16, 64, 128, 1), (16, 7, 128, 2), (8, 16, 100, 1),
                                                      (16, 8, 129, 3), (16, 64, 129, 2), (16, 1, 4096, 64), (16, 256, 4096, 1)])
def test_pieces_of_the_latent_decode_kernel_of_few_heads(monkeypatch, heads, seqs, length, pieces):
    """A piece is a tile of 64 rows as long as the blocks fit the SMs; two tiles stay together from 128 query vectors on."""
    monkeypatch.setattr(kernels, "sm_count", lambda: 148)
    step = SimpleNamespace(max_qlen=1, n_seqs=seqs, max_kvlen=length)
    assert kernels.latent_attention_splits(step, heads, True, 512, few=True) == pieces
    # a window of 128 reaches into a third tile, one of 65 into no more than two
    assert kernels.latent_attention_splits(SimpleNamespace(max_qlen=1, n_seqs=8, max_kvlen=4096), 16, True, 512, window=128, few=True) == 3
    assert kernels.latent_attention_splits(SimpleNamespace(max_qlen=1, n_seqs=8, max_kvlen=4096), 16, True, 512, window=65, few=True) == 1
    step.max_qlen = 2
    assert kernels.latent_attention_splits(step, heads, True, 512, few=True) == 1


@pytest.mark.parametrize("sms", [132, 148])
def test_every_kernel_of_the_32_bit_product_is_chosen_somewhere(sms):
    """... and only where it can run: the stream (6) takes up to 16 ungrouped rows of whole vectors, grouped products the
    tiles 1, 2 and 4 or the blocks of 64 x 64 (5)."""
    choice = kernels.lib().leb_gemm_f32_choice
    sizes = [1, 3, 9, 16, 17, 36, 130, 523, 1757, 2557, 4000]
    seen = {}
    for groups in (0, 1, 3, 64):
        for M in sizes:
            for N in sizes:
                for K in (4, 128, 132, 301, 1024, 5632):
                    for vec in (0, 1) if K % 4 == 0 else (0,):
                        k = choice(M, N, K, groups, vec, sms)
                        seen.setdefault((min(groups, 2), vec), set()).add(k)
                        assert 0 <= k <= 6 and (k != 6 or (groups == 0 and vec and M <= 16)) and (groups < 2 or k in (1, 2, 4, 5))
    assert seen[0, 1] == set(range(7)) and seen[0, 0] == set(range(6)) and seen[2, 0] == seen[2, 1] == {1, 2, 4, 5}
    assert choice(0, 1, 1, 0, 1, sms) == -1 and choice(1, 1, 0, 0, 1, sms) == -1


def test_products_wait_for_one_another_only_in_models_of_the_librarys_own_parts():
    """A part from elsewhere may touch its input or result without the library's kernels: its model launches every product at once."""
    import dataclasses
    from lastengine_b200.engine.model import Model
    from lastengine_b200.engine.workspace import Workspace
    from lastengine_b200.parts.base import BuildEnv, PartSpec
    from lastengine_b200.parts.ffn import SwiGLU
    from lastengine_b200.registry import FEED_FORWARDS, plan_from_config
    from tiny_configs import TINY_A
    cpu = torch.device("cpu")
    env = BuildEnv(device=cpu, dtype=torch.bfloat16, workspace=Workspace(cpu))
    plan = plan_from_config(TINY_A)
    assert Model(plan, env).chains

    @FEED_FORWARDS.register("swiglu_from_elsewhere", replace=True)
    class Elsewhere(SwiGLU):
        pass
    last = plan.layers[-1]
    layers = [*plan.layers[:-1], dataclasses.replace(last, ffn=PartSpec("swiglu_from_elsewhere", last.ffn.params))]
    assert not Model(dataclasses.replace(plan, layers=layers), env).chains
