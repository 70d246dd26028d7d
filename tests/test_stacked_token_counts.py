"""A stored segment has the number of tokens that its shape states: payloads whose arrays do not agree with it are refused
when they are stacked, on either device."""
import pytest
import torch

from nanokv_b200 import lingbot_codec, mg_codec

HEADS, HEAD_DIM, RANK, CLUSTERS = 2, 16, 8, 4


def _payload(form, tokens, ids, scales):
    joint = HEADS * HEAD_DIM
    gen = torch.Generator().manual_seed(tokens)
    codes = torch.randint(0, 256, (1, tokens, RANK // 2), generator=gen).to(torch.uint8)
    scale = torch.rand(1, scales, 1, generator=gen).to(torch.bfloat16)
    part = dict(layer=0, ids=torch.randint(0, CLUSTERS, (1, ids), generator=gen).to(torch.uint8),
                centers=torch.randn(1, CLUSTERS, joint, generator=gen).to(torch.bfloat16))
    if form == "lingbot":
        return dict(part, format=lingbot_codec.FORMAT, target="k", rank=RANK, shape=(1, tokens, HEADS, HEAD_DIM),
                    latent_packed=codes, latent_scale=scale)
    return dict(part, codec=mg_codec.CODEC, kind="k", shape=(1, tokens, joint), latent_shape=(1, tokens, RANK),
                packed_codes=codes, scale=scale)


def _stack(form, parts, device):
    return (lingbot_codec if form == "lingbot" else mg_codec).history_from_payloads(parts, device=device)


DEVICES = ["cpu", pytest.param("cuda", marks=pytest.mark.gpu)]


@pytest.mark.parametrize("device", DEVICES)
@pytest.mark.parametrize("form", ["lingbot", "matrix_game"])
@pytest.mark.parametrize("tokens,ids", [(1, 3), (1, 2), (5, 3), (5, 6)])
def test_ids_of_another_number_are_refused(form, tokens, ids, device):
    with pytest.raises((ValueError, RuntimeError)):
        _stack(form, [_payload(form, 4, 4, 4), _payload(form, tokens, ids, tokens)], device)


@pytest.mark.parametrize("device", DEVICES)
@pytest.mark.parametrize("form", ["lingbot", "matrix_game"])
def test_segments_that_agree_are_stacked(form, device):
    parts = [_payload(form, n, n, n) for n in (1, 7, 3)]
    hist = _stack(form, parts, device)
    assert hist.tokens == 11 and hist.seg_start.tolist() == [0, 1, 8, 11]
    assert torch.equal(hist.ids.cpu(), torch.cat([p["ids"][0] for p in parts]))
