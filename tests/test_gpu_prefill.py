"""Chunked prefill on the decode tiles (one GPU, cp = 1): every query token of a
chunk against the CPU oracle's decode step at that token's causal length."""

import math

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.mark.parametrize("S,Tq,tile,K,bpc", [(4096, 32, 8, 512, 16), (8192, 24, 12, 2048, 32)])
def test_prefill_chunk_matches_oracle_per_query(S, Tq, tile, K, bpc):
    from dsa_inputs import indexer_case
    from mega_dsa_cp_b200.prefill import DsaPrefillChunk, causal_local_lens
    from oracle import dsa_oracle as orc

    P, H, DQK = 64, 128, 576
    case = indexer_case(1, S, P, "nvfp4", seed=14)          # one sequence's index cache and page table
    g = torch.Generator().manual_seed(15)
    q_idx = torch.randn(Tq, 64, 128, generator=g).bfloat16()
    w_idx = torch.randn(Tq, 64, generator=g) / 64
    q_mla = (torch.randn(Tq, 1, H, DQK, generator=g) * 0.5).bfloat16()
    kv = (torch.randn(S, 1, DQK, generator=g) * 0.5).bfloat16()
    # the chunk's tokens are the last Tq of the context, plus two early positions shorter than top-k
    pos = torch.arange(S - Tq, S)
    pos[0], pos[1] = 5, K // 2
    assert causal_local_lens(pos, 1, 0).tolist() == (pos + 1).tolist()
    pf = DsaPrefillChunk(tile, cp=1, top_k=K, max_pages=S // P, blocks_per_chunk=bpc, out_dtype=torch.float32, n_ctas=64)
    d = lambda t: t.to(DEV)
    pf.bind(d(case["fused"]), d(case["bt"][0]), d(kv))
    out = torch.zeros(Tq, H, 512, device=DEV)
    lse = torch.zeros(Tq, H, device=DEV)
    sel_i = torch.zeros(Tq, K, dtype=torch.int32, device=DEV)
    sel_c = torch.zeros(Tq, dtype=torch.int32, device=DEV)
    pf.run(d(q_idx), d(w_idx), d(q_mla), pos, out, lse, sel_i, sel_c)
    torch.cuda.synchronize()
    pf.check_status()
    data, sf = orc.split_index_pages(case["fused"], "nvfp4", P)
    kd = orc.dequant_fp4(data, sf, "nvfp4").reshape(-1, P, 128)[case["bt"][0].long()].reshape(S, 128)
    scale = 1 / math.sqrt(DQK)
    for j in range(Tq):
        n_ctx = int(pos[j]) + 1
        sel, _, _ = orc.decode_step_ref(q_idx[j].float(), w_idx[j], kd, q_mla[j, 0].float(), kv[:, 0].float(),
                                        n_ctx, K, scale)
        n = int(sel_c[j])
        got = sel_i[j, :n].cpu()
        assert n == sel.numel() == min(K, n_ctx), (j, n, sel.numel())
        assert int(got.max()) < n_ctx                     # causal: nothing after the query's own position
        overlap = len(set(got.tolist()) & set(sel.tolist())) / sel.numel()
        assert overlap >= 0.999, (j, overlap)
        o, l = orc.attend_selected_ref(q_mla[j, 0].float(), kv[:, 0].float(), got, scale)
        assert (out[j].cpu() - o).abs().max() < 2e-2, j
        assert (lse[j].cpu() - l).abs().max() < 1e-3, j


def _chunk(S, Tq, K, seed):
    """One sequence's caches and a chunk's inputs and results on the device."""
    from dsa_inputs import indexer_case

    case = indexer_case(1, S, 64, "nvfp4", seed=seed)
    g = torch.Generator().manual_seed(seed + 1)
    d = lambda t: t.to(DEV)
    caches = (d(case["fused"]), d(case["bt"][0]), d((torch.randn(S, 1, 576, generator=g) * 0.5).bfloat16()))
    pos = torch.arange(S - Tq, S)
    pos[0], pos[-1] = 7, K // 2
    x = (d(torch.randn(Tq, 64, 128, generator=g).bfloat16()), d(torch.randn(Tq, 64, generator=g) / 64),
         d((torch.randn(Tq, 1, 128, 576, generator=g) * 0.5).bfloat16()), d(pos))
    return caches, x


def _results(Tq, K, dtype=torch.bfloat16):
    return dict(out=torch.zeros(Tq, 128, 512, dtype=dtype, device=DEV), out_lse=torch.zeros(Tq, 128, device=DEV),
                sel_i=torch.zeros(Tq, K, dtype=torch.int32, device=DEV), sel_c=torch.zeros(Tq, dtype=torch.int32, device=DEV))


@pytest.mark.parametrize("device", ["cuda", "cuda:0"])
@pytest.mark.parametrize("tile,Tq,out_dtype", [(8, 32, torch.bfloat16), (8, 24, torch.float32), (4, 20, torch.bfloat16), (3, 39, torch.bfloat16)])
def test_results_in_place_and_copied_agree_with_the_oracle(device, tile, Tq, out_dtype):
    """Results that the launches write straight into the caller's tensors (of every launch size a chunk is split into)
    against the oracle, and bit for bit against copied ones: other types, rows apart, off a 16-byte boundary."""
    from mega_dsa_cp_b200.prefill import DsaPrefillChunk
    from oracle import dsa_oracle as orc

    S, K, scale = 4096, 512, 1 / math.sqrt(576)
    caches, x = _chunk(S, Tq, K, seed=71)
    pf = DsaPrefillChunk(tile, top_k=K, max_pages=S // 64, blocks_per_chunk=16, out_dtype=out_dtype, device=device)
    pf.bind(*caches)
    res = _results(Tq, K, out_dtype)
    own = [b for layer in pf._layers.values() for b in (layer.out, layer.out_lse, layer.sel_i, layer.sel_c)]
    pf.run(*x, **res)
    torch.cuda.synchronize()
    pf.check_status()
    assert not any(bool(b.any()) for b in own)                        # nothing went through the layers' own buffers
    kv = caches[2][:, 0].float().cpu()
    for j in (0, 1, tile, Tq - 2, Tq - 1):
        n, pos = int(res["sel_c"][j]), int(x[3][j])
        assert n == min(K, pos + 1)
        ids = res["sel_i"][j, :n].cpu()
        assert int(ids.max()) <= pos
        o, l = orc.attend_selected_ref(x[2][j, 0].float().cpu(), kv, ids, scale)
        assert (res["out"][j].float().cpu() - o).abs().max() < 2e-2 and (res["out_lse"][j].cpu() - l).abs().max() < 1e-3
    odd = torch.zeros(res["out"].numel() + 1, dtype=out_dtype, device=DEV)[1:].view(res["out"].shape)
    apart = torch.zeros(Tq, 2 * K, dtype=torch.int32, device=DEV)
    copied = dict(out=odd, out_lse=torch.zeros(Tq, 128, dtype=torch.float64, device=DEV), sel_i=apart[:, :K],
                  sel_c=torch.zeros(Tq, dtype=torch.int64, device=DEV))
    pf.run(*x, **copied)
    torch.cuda.synchronize()
    pf.check_status()
    assert all(torch.equal(copied[k], res[k].to(copied[k].dtype)) for k in res) and not apart[:, K:].any()


def test_chunks_on_new_tensors_on_another_stream():
    """Each chunk's tensors are made anew and dropped right after the call, on a stream that the launches do not run on."""
    from mega_dsa_cp_b200.prefill import DsaPrefillChunk

    S, K, tile, Tq = 4096, 512, 4, 12
    caches, x = _chunk(S, Tq, K, seed=73)
    pf = DsaPrefillChunk(tile, top_k=K, max_pages=S // 64, blocks_per_chunk=16)
    pf.bind(*caches)
    want = _results(Tq, K)
    pf.run(*x, **want)
    torch.cuda.synchronize()
    side = torch.cuda.Stream()
    for handle in (side, side.cuda_stream):
        got = []
        for _ in range(4):
            res = _results(Tq, K)
            y = tuple(t.clone() for t in x)
            side.wait_stream(torch.cuda.current_stream())
            pf.run(*y, **res, stream=handle)
            got.append(res)
            del y, res
            torch.full((8 << 20,), -1, dtype=torch.int32, device=DEV)   # (takes freed memory, were it free)
        torch.cuda.synchronize()
        pf.check_status()
        assert all(torch.equal(r[k], want[k]) for r in got for k in want)


def test_a_chunk_replays_from_a_cuda_graph():
    """A chunk of two launches captured by its first call: replays follow the contents of the captured tensors."""
    from mega_dsa_cp_b200.prefill import DsaPrefillChunk

    S, K, tile, Tq = 4096, 512, 16, 48
    caches, x = _chunk(S, Tq, K, seed=75)
    first, new = tuple(t.clone() for t in x), tuple(t.flip(0).contiguous() for t in x)
    wants = []
    for y in (x, new):
        pf = DsaPrefillChunk(tile, top_k=K, max_pages=S // 64, blocks_per_chunk=16)
        pf.bind(*caches)
        wants.append(_results(Tq, K))
        pf.run(*y, **wants[-1])
    torch.cuda.synchronize()
    pf = DsaPrefillChunk(tile, top_k=K, max_pages=S // 64, blocks_per_chunk=16)
    pf.bind(*caches)
    got = _results(Tq, K)
    got["out_lse"] = got["out_lse"].double()                # (one result copied inside the graph)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        pf.run(*x, **got)
    for want, y in ((wants[0], x), (wants[1], new), (wants[0], x)):
        for a, b in zip(x, y if y is new else first):
            a.copy_(b)
        for t in got.values():
            t.zero_()      # (a row's ids behind its count are not written)
        graph.replay()
        torch.cuda.synchronize()
        pf.check_status()
        assert all(torch.equal(got[k], want[k].to(got[k].dtype)) for k in want)
