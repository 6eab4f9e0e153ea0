"""What the greedy decoder and the entry points behind it refuse, and that they refuse it before anything is launched. No
device needed: the host-side checks are what is tested."""
import ctypes

import pytest

torch = pytest.importorskip("torch")

from nntrainer_b200 import build as nb_build  # noqa: E402
from nntrainer_b200 import capi  # noqa: E402
from nntrainer_b200.decoder import DecoderConfig, Qwen3Decoder  # noqa: E402

CFG = DecoderConfig(n_layers=1, hidden=512, n_heads=8, n_kv_heads=2, head_dim=64, inter=768, vocab=1024, max_seq=64)


@pytest.fixture(scope="module")
def L():
    nb_build.build()
    return capi.lib()


def _decoder(cfg):
    """A decoder whose passes only write down what they were asked for."""
    d = Qwen3Decoder.__new__(Qwen3Decoder)
    d.torch, d.cfg, d.dev, d.fed = torch, cfg, "cpu", []
    d._prompt = lambda ids, pos: d.fed.append(("rows", pos, len(ids)))
    d.step = lambda tok, pos, **kw: d.fed.append(("step", pos, 1))
    return d


@pytest.mark.parametrize("pos,tokens,max_rows", [(0, 65, 64), (60, 5, 64), (64, 1, 64), (1, 0xFFFFFFFF, 64), (0xFFFFFFFF, 1, 64)])
def test_rows_behind_the_caches_are_refused(L, pos, tokens, max_rows):
    a = capi.AttnDesc(8, 2, 64, 0xFFFFFFFF, None)
    p = 1 << 20  # aligned, and never looked at: the check comes before the first launch
    before = L.nntr_cuda_launch_count()
    rc = L.nntr_cuda_attention_rows_dev(ctypes.byref(a), pos, tokens, max_rows, p, p, p, 768, None, None, 0.0, p, p, p, p, p, 512,
                                        0, None)
    assert rc == capi.ERR_INVALID
    assert L.nntr_cuda_launch_count() == before


@pytest.mark.parametrize("n", [65, 66, 300])
def test_a_prompt_longer_than_the_caches_is_refused_before_the_first_pass(n):
    d = _decoder(CFG)
    with pytest.raises(ValueError):
        d.generate([1] * n, 1)
    assert d.fed == []


def test_a_prompt_that_fills_the_caches_is_fed():
    d = _decoder(CFG)
    d.generate([1] * 64, 0)
    assert d.fed == [("rows", 0, 63), ("step", 63, 1)]


@pytest.mark.parametrize("n_new", [1, 5])
def test_an_empty_prompt_is_refused(n_new):
    """There is no token to start from: nothing may be decoded from an uninitialised one."""
    d = _decoder(CFG)
    with pytest.raises(ValueError):
        d.generate([], n_new)
    assert d.fed == []


@pytest.mark.parametrize("prompt,n_new", [([], 0), ([], -1), ([3], 0), ([3], -1), ([3, 4], -7), ([1] * 8, -2)])
def test_no_new_tokens_feed_the_prompt_only(prompt, n_new):
    d = _decoder(CFG)
    assert d.generate(prompt, n_new) == []
    assert sum(n for _, _, n in d.fed) == len(prompt)
