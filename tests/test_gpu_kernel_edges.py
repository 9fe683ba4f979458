"""Tile edges, remainders and dispatch branches of the kernels, against the oracle."""
import math

import pytest
import torch

from helpers import TOL_BF16, maxabs
from oracle import conv_attn_oracle as orc

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("offset_causal", [False, True])
@pytest.mark.parametrize("B,H,q_len,Nk,d,cq,ck,k_splits", [
    (1, 2, 6, 31, 128, 6, 11, 1),      # less than one 32-key block
    (1, 2, 6, 33, 128, 6, 11, 1),      # one key past it
    (1, 1, 9, 515, 128, 9, 17, 2),     # 16-row fragments, widest filter; a split of 320 and one of 195 keys
    (1, 2, 16, 1040, 64, 16, 7, 3),    # 16 live rows, padded filter columns
    (2, 2, 5, 4097, 64, 5, 9, 1),      # one split over a cluster of eight CTAs, ragged end
    (1, 1, 3, 2050, 32, 3, 13, 2),     # two splits x sub-splits merged in one cluster
    (1, 1, 6, 1600, 64, 6, 11, 24),    # more splits than a cluster holds: combine launch
    (3, 8, 7, 129, 128, 7, 7, 129),    # one key per split: most splits are empty
])
def test_decode_blocks_splits_and_filters(B, H, q_len, Nk, d, cq, ck, k_splits, offset_causal):
    import fmta_b200 as F
    Q, K, V, _, theta = orc.make_inputs(B, H, 0, d, cq, ck, seed=Nk + d, dtype=torch.bfloat16, Nk=Nk, q_len=q_len)
    scale = 1.0 / math.sqrt(d)
    q, k, v = (t.cuda().to(torch.bfloat16).contiguous() for t in (Q, K, V))
    O, M, L = F.fwd_conv_attn_inference(q, k, v, theta.cuda(), k_splits, scale, cq - 1, (ck - 1) // 2, False, offset_causal=offset_causal)
    fn = orc.decode_last_row_offset_causal if offset_causal else orc.decode_last_row_streaming
    Or, Mr, Lr = fn(Q, K, V, theta, scale)
    # scores and probabilities are 32-bit here: far inside the bf16 bound
    assert maxabs(O, Or.reshape(O.shape)) <= 1e-4
    assert maxabs(M, Mr.reshape(M.shape)) <= 1e-4
    assert maxabs(M + torch.log(L), (Mr + torch.log(Lr)).reshape(M.shape)) <= 1e-4
    # the same cache through pages of 64 keys
    page, pages = 64, -(-Nk // 64)
    pad = pages * page - Nk
    pool = [torch.nn.functional.pad(t, (0, 0, 0, pad)).view(B, H, pages, page, d).transpose(1, 2).reshape(B * pages, H, page, d).contiguous()
            for t in (k, v)]
    table = torch.arange(B * pages, dtype=torch.int32, device="cuda").view(B, pages)
    Op, Mp, Lp = F.forward_inference_paged(q, pool[0], pool[1], table, theta.cuda(), k_splits, scale, cq - 1, (ck - 1) // 2,
                                           max_seq_len=Nk, offset_causal=offset_causal)
    assert torch.equal(Op[:, :, 0:1], O) and torch.equal(Mp[:, :, 0:1], M) and torch.equal(Lp[:, :, 0:1], L)
