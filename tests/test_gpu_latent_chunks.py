"""Attention on the latent in chunks of 64 and of 32 keys, against float64: shares of the keys, windows, sinks, ranks on both sides of
the column split, keys too long for the larger chunks and for two buffers."""
from types import SimpleNamespace

import pytest
import torch

from burn_lm_b200 import kernels as K

pytestmark = pytest.mark.gpu


# the last three: 64 keys no longer fit twice (32 do), 32 keys fit once, and once with sixteen rows only
@pytest.mark.parametrize("H,R,dr", [(1, 16, 0), (3, 48, 16), (16, 256, 32), (32, 272, 64), (40, 512, 64), (40, 512, 176), (20, 512, 512),
                                    (20, 512, 960)])
@pytest.mark.parametrize("splits,window,sink", [(1, 0, False), (3, 0, True), (5, 70, True), (1, 1, False)])
@pytest.mark.parametrize("lens,starts", [([1, 1, 1, 1], [0, 63, 64, 400]), ([3, 0, 2], [130, 5, 31])])
def test_latent_attention_in_chunks(H, R, dr, splits, window, sink, lens, starts):
    gen = torch.Generator(device="cuda")
    gen.manual_seed(R + dr + splits)
    rnd = lambda *shape: torch.randn(shape, generator=gen, device="cuda")
    i32 = lambda v: torch.tensor(v, dtype=torch.int32, device="cuda")
    D, cu = R + dr, [0]
    for m in lens:
        cu.append(cu[-1] + m)
    n, each = cu[-1], max(-(-(a + b) // K.PAGE) for a, b in zip(lens, starts))
    perm = torch.randperm(each * len(lens) + 1, generator=torch.Generator().manual_seed(2))[: each * len(lens)].to(torch.int32)
    table = perm.reshape(len(lens), each).cuda()
    pool = torch.full((each * len(lens) + 1, K.PAGE, D), float("nan"), dtype=torch.bfloat16, device="cuda")
    step = SimpleNamespace(n_tokens=n, n_seqs=len(lens), max_q_len=max(lens), max_kv_len=each * K.PAGE, cu_seqlens=i32(cu),
                           token_seq=i32([s for s, m in enumerate(lens) for _ in range(m)]),
                           token_pos=i32([a + t for m, a in zip(lens, starts) for t in range(m)]),
                           slot_of_seq=i32(list(range(len(lens)))), start_pos=i32(starts))
    q_lat, q_rot = rnd(H, n, R).bfloat16().float(), rnd(n, H, dr).bfloat16().float()      # (the kernel rounds them to bfloat16)
    logits = 2.0 * rnd(H)
    latents = [rnd(start + m, D).bfloat16() for m, start in zip(lens, starts)]
    for s, rows in enumerate(latents):
        for j in range(0, len(rows), K.PAGE):
            pool[int(table[s, j // K.PAGE]), : min(K.PAGE, len(rows) - j)] = rows[j:j + K.PAGE]
    scale = D ** -0.5
    for out_dtype in (torch.bfloat16, torch.float32):
        out = torch.full((H, n, R), float("nan"), dtype=out_dtype, device="cuda")
        partial = torch.full((max(1, K.latent_attention_scratch_floats(n, H, R, splits)),), float("nan"), device="cuda")
        K.latent_attention(q_lat, q_rot, pool, table, step, out, H, R, dr, scale, n_splits=splits, partial=partial, window=window,
                           sink=logits if sink else None)
        for s, (m, start) in enumerate(zip(lens, starts)):
            sl, keys = slice(cu[s], cu[s + 1]), latents[s].double()
            q = torch.cat([q_lat[:, sl].double(), q_rot[sl].double().transpose(0, 1)], -1)
            i, j = start + torch.arange(m, device="cuda")[:, None], torch.arange(start + m, device="cuda")[None]
            sc = torch.where((j <= i) & ((i - j < window) | (window == 0)), q @ keys.T * scale, -torch.inf)
            if sink:
                p = torch.softmax(torch.cat([sc, logits.double()[:, None, None].expand(H, m, 1)], -1), -1)[..., :-1]
            else:
                p = torch.softmax(sc, -1)
            want = p @ keys[:, :R]
            # the weights are rounded to bfloat16 (2^-8), bfloat16 outputs once more; the rest is float32
            room = 2.0 ** -8 * (p @ keys[:, :R].abs()) + (2.0 ** -8 * want.abs() if out_dtype == torch.bfloat16 else 0.0) + 1e-4
            assert ((out[:, sl].double() - want).abs() <= room).all()


@pytest.mark.parametrize("H,R,dr", [(16, 256, 32), (32, 512, 64), (20, 512, 512)])           # 64 keys twice, and 32
@pytest.mark.parametrize("splits", [1, 4])
def test_weights_are_kept_to_sixteen_bits(H, R, dr, splits):
    gen = torch.Generator(device="cuda")
    gen.manual_seed(R + dr)
    rnd = lambda *shape: torch.randn(shape, generator=gen, device="cuda")
    i32 = lambda v: torch.tensor(v, dtype=torch.int32, device="cuda")
    n, keys, D = 3, 700, R + dr
    pages = -(-keys // K.PAGE)
    step = SimpleNamespace(n_tokens=n, n_seqs=n, max_q_len=1, max_kv_len=keys, cu_seqlens=i32(list(range(n + 1))), token_seq=i32(list(range(n))),
                           token_pos=i32([keys - 1] * n), slot_of_seq=i32(list(range(n))), start_pos=i32([keys - 1] * n))
    latents = rnd(n, pages * K.PAGE, D).bfloat16()
    q_lat, q_rot = rnd(H, n, R).bfloat16().float(), rnd(n, H, dr).bfloat16().float()
    out = torch.empty((H, n, R), device="cuda")
    partial = torch.empty((max(1, K.latent_attention_scratch_floats(n, H, R, splits)),), device="cuda")
    scale = 2.0 * D ** -0.5
    K.latent_attention(q_lat, q_rot, latents.view(n * pages, K.PAGE, D), i32(list(range(n * pages))).view(n, pages), step, out, H, R, dr, scale,
                       n_splits=splits, partial=partial)
    seen = latents[:, :keys].double()
    p = torch.softmax(torch.einsum("nhd,ntd->nht", torch.cat([q_lat.transpose(0, 1), q_rot], -1).double(), seen) * scale, -1)
    want = torch.einsum("nht,ntd->nhd", p, seen[..., :R]).transpose(0, 1)
    terms = torch.einsum("nht,ntd->nhd", p, seen[..., :R].abs()).transpose(0, 1)
    # two bfloat16 numbers round a weight by 2^-17; fp32 scores of up to 10 and their exponentials by some 2^-19
    assert ((out.double() - want).abs() <= 2.0 ** -15 * terms).all()


@pytest.mark.parametrize("dtype,rank,rot,blocks", [(torch.bfloat16, 512, 64, 1), (torch.float32, 512, 64, 2), (torch.bfloat16, 500, 64, 2),
                                                   (torch.bfloat16, 640, 64, 2)])
@pytest.mark.parametrize("n_seqs", [1, 7, 32])
def test_shares_offer_every_multiprocessor_the_blocks_it_holds(dtype, rank, rot, blocks, n_seqs):
    """One block of the tensor-core kernel fills a multiprocessor, two of the CUDA-core kernel do (32-bit caches, ranks that are no
    multiples of 16 lanes or too long)."""
    heads, dev = 32, torch.device("cuda")
    splits = K.latent_attention_splits(dtype, heads, rank, rot, n_seqs, 1, 1 << 20, dev)
    tiles = -(-heads // K.latent_attention_tile_rows(dtype, heads, rank, rot, 1)) * n_seqs
    most = blocks * K.sm_count(dev)
    assert splits == 32 and tiles * splits <= most or most - tiles < tiles * splits <= most
