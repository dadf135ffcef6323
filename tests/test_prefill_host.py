"""Host side of the chunked prefill on the CPU: where a chunk's launches read and write.  Both launches of a chunk are
replaced (the step by a recorder), so nothing reaches a device."""

import gc
import weakref

import pytest
import torch

from mega_dsa_cp_b200 import _native as N
from mega_dsa_cp_b200 import layer as layer_mod
from mega_dsa_cp_b200 import prefill as prefill_mod

H, DQK, K, TILE = 128, 576, 64, 2


@pytest.fixture
def launches(monkeypatch):
    seen = []

    def step(self, wait_budget_ns=0, stream=None, trace=None, _params=None):
        L = N.LayerParams.from_buffer_copy(_params or self._params)
        seen.append((self, L))
        self.out.fill_(1.0)    # what a launch would leave in the layer's own buffers
        self.out_lse.fill_(2.0)
        self.sel_i.fill_(3)
        self.sel_c.fill_(4)

    monkeypatch.setattr(layer_mod.DsaDecodeLayer, "step", step)
    monkeypatch.setattr(prefill_mod, "_device_lens", lambda *args: None)
    return seen


def _prefill(**kw):
    args = dict(top_k=K, max_pages=4, blocks_per_chunk=2, n_ctas=16, device="cpu")
    pf = prefill_mod.DsaPrefillChunk(TILE, **{**args, **kw})
    pf.bind(torch.zeros(4, 4608, dtype=torch.uint8), torch.arange(4), torch.zeros(256, 1, DQK, dtype=torch.bfloat16))
    return pf


def _inputs(Tq):
    return (torch.zeros(Tq, 64, 128, dtype=torch.bfloat16), torch.zeros(Tq, 64), torch.zeros(Tq, 1, H, DQK, dtype=torch.bfloat16),
            torch.arange(Tq))


def _results(Tq):
    return dict(out=torch.zeros(Tq, H, 512, dtype=torch.bfloat16), out_lse=torch.zeros(Tq, H), sel_i=torch.zeros(Tq, K, dtype=torch.int32),
                sel_c=torch.zeros(Tq, dtype=torch.int32))


def _targets(launches, name):
    return [getattr(L, name) for _, L in launches]


def _offset(t, elements):
    """A contiguous copy of t whose data starts `elements` elements behind a 16-byte boundary."""
    buf = torch.zeros(t.numel() + elements, dtype=t.dtype)
    return buf[elements:].view(t.shape)


def test_results_that_fit_are_written_in_place(launches):
    pf, res = _prefill(), _results(4)
    pf.run(*_inputs(4), **res)
    for name, t in res.items():
        assert _targets(launches, name)[0] == t.data_ptr() and not t.any(), name


@pytest.mark.parametrize("name,make", [
    ("out", lambda t: t.float()),                                            # another type
    ("out", lambda t: torch.zeros(4, H, 1024, dtype=t.dtype)[:, :, :512]),   # rows apart
    ("out", lambda t: _offset(t, 1)),                                        # contiguous, but not 16-byte aligned
    ("out_lse", lambda t: t.double()),
    ("sel_i", lambda t: t.long()),
    ("sel_i", lambda t: torch.zeros(4, 2 * K, dtype=t.dtype)[:, ::2]),
    ("sel_c", lambda t: t.long()),
])
def test_other_results_are_copied(launches, name, make):
    pf, res = _prefill(), _results(4)
    res[name] = make(res[name])
    pf.run(*_inputs(4), **res)
    value = dict(out=1, out_lse=2, sel_i=3, sel_c=4)[name]
    assert bool((res[name] == value).all())
    assert all(L_target == getattr(layer, name).data_ptr() for (layer, _), L_target in zip(launches, _targets(launches, name)))


def test_results_in_the_memory_of_an_input_are_copied(launches):
    """A caller may let the output take the place of the attention query: it is written once the step is through."""
    pf, res = _prefill(), _results(4)
    q_idx, w, q_mla, pos = _inputs(4)
    res["out"] = q_mla.view(-1)[:res["out"].numel()].view(res["out"].shape)
    pf.run(q_idx, w, q_mla, pos, **res)
    assert bool((res["out"] == 1).all()) and _targets(launches, "out")[0] == launches[0][0].out.data_ptr()


@pytest.mark.parametrize("name,shape", [("out", (4, H, 256)), ("out", (3, H, 512)), ("out", (4, H // 2, 512)), ("out", (4 * H, 512)),
                                        ("out_lse", (4, H // 2)), ("out_lse", (2, H)), ("sel_i", (4, K // 2)), ("sel_i", (1, K)),
                                        ("sel_c", (2,)), ("sel_c", (4, 1))])
def test_results_of_a_wrong_shape_are_refused(launches, name, shape):
    pf, res = _prefill(), _results(4)
    res[name] = torch.zeros(shape, dtype=res[name].dtype)
    with pytest.raises((RuntimeError, IndexError)):
        pf.run(*_inputs(4), **res)
    assert all(getattr(L, name) == getattr(layer, name).data_ptr() for layer, L in launches)


def test_every_call_reads_and_writes_its_own_tensors(launches):
    """Another view at the same address, and a new tensor at a freed one's address, are other tensors."""
    pf = _prefill()
    q_idx, w, q_mla, pos = _inputs(4)
    wide = torch.zeros(4, H, 1024, dtype=torch.bfloat16)
    pf.run(q_idx, w, q_mla, pos, wide[:, :, :512])
    assert bool((wide[:, :, :512] == 1).all()) and not wide[:, :, 512:].any()
    wide.zero_()
    every_other = wide.view(4, 2, H, 512)[:, 0]                        # same address and type, other strides
    pf.run(q_idx, w, q_mla, pos, every_other)
    assert bool((every_other == 1).all()) and not wide.view(4, 2, H, 512)[:, 1].any()
    wide.zero_()
    pf.run(q_idx, w, q_mla, pos, wide.view(8, H, 512)[:4])             # contiguous: in place
    assert not wide.any() and launches[-1][1].out == wide.data_ptr()
    for _ in range(3):
        x, res = _inputs(4), _results(4)
        x[1].fill_(1.0)
        pf.run(*x, **res)
        L = launches[-1][1]
        assert (L.logits.q, L.logits.weights, L.mla.q, L.out) == (x[0].data_ptr(), x[1].data_ptr(), x[2].data_ptr(), res["out"].data_ptr())


def test_tensors_of_a_call_are_not_kept(launches):
    pf = _prefill()
    x, res = _inputs(4), _results(4)
    pf.run(*x, **res)
    refs = [weakref.ref(t) for t in (*x, *res.values())]
    del x, res
    gc.collect()
    assert not any(r() is not None for r in refs)


def test_bind_wants_a_whole_row_of_the_page_table():
    pf = _prefill()
    for n in (1, 3, 8):
        with pytest.raises(AssertionError):
            pf.bind(torch.zeros(4, 4608, dtype=torch.uint8), torch.zeros(n, dtype=torch.int32), torch.zeros(256, 1, DQK, dtype=torch.bfloat16))


@pytest.mark.parametrize("tile,Tqs", [(2, (2, 4, 2)), (1, (3, 1, 4)), (4, (4, 8))])
def test_the_layers_are_built_with_the_object(launches, monkeypatch, tile, Tqs):
    """A call of a size not seen before lays out nothing: every launch runs on a layer that the constructor built."""
    monkeypatch.setattr(prefill_mod, "DsaDecodeLayer", _counted := _Counted(layer_mod.DsaDecodeLayer))
    pf = prefill_mod.DsaPrefillChunk(tile, top_k=K, max_pages=4, blocks_per_chunk=2, n_ctas=16, device="cpu")
    pf.bind(torch.zeros(4, 4608, dtype=torch.uint8), torch.arange(4), torch.zeros(256, 1, DQK, dtype=torch.bfloat16))
    built = _counted.n
    for Tq in Tqs:
        del launches[:]
        pf.run(*_inputs(Tq), **_results(Tq))
        assert sum(L.B for _, L in launches) == Tq
    assert _counted.n == built


class _Counted:
    def __init__(self, cls):
        self.cls, self.n = cls, 0

    def __call__(self, *a, **kw):
        self.n += 1
        return self.cls(*a, **kw)


@pytest.mark.parametrize("tile", [1, 2, 3, 5, 8, 37])
def test_chunks_of_every_size_are_covered_by_the_layers(launches, tile):
    """Few launches, each of at most what fills the blocks, together exactly the chunk."""
    pf = _prefill_of(tile, 148)
    assert pf.max_tiles == 37 // tile and len(pf._layers) <= 17
    for tiles in (1, 2, 3, 7, 8, 11, 12, 13, 17, 18, 23, 30, 31, 36, 37, 38, 75):
        parts = list(pf._split(tiles))
        assert sum(parts) == tiles and all(n in pf._layers for n in parts)
        assert len(parts) <= -(-tiles // pf.max_tiles) + 2 and max(parts) <= pf.max_tiles


def _prefill_of(tile, n_ctas):
    return prefill_mod.DsaPrefillChunk(tile, top_k=K, max_pages=4, blocks_per_chunk=2, n_ctas=n_ctas, device="cpu")


def test_a_device_without_an_index_is_the_current_one(monkeypatch):
    monkeypatch.setattr(torch.cuda, "current_device", lambda: 3)
    assert layer_mod.resolve_device("cuda") == torch.device("cuda", 3)
    assert layer_mod.resolve_device("cuda:1") == torch.device("cuda", 1) and layer_mod.resolve_device("cpu") == torch.device("cpu")
