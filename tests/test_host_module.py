"""CPU checks of the native host module (csrc/host_bindings.cpp): what the runners refuse comes back as a Python
error, before anything reaches a device."""

import os
import subprocess
import sys

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def _errors_of(bodies):
    """Names of the exceptions that the pieces of code raise in a fresh interpreter (a crash there fails the test, not
    the session)."""
    code = "import sys\nsys.path.insert(0, %r)\nimport torch\n" % ROOT
    for body in bodies:
        code += "try:\n" + "".join("    " + line + "\n" for line in body.strip().splitlines())
        code += "    print('NONE')\nexcept Exception as e:\n    print(type(e).__name__)\n"
    r = subprocess.run([sys.executable, "-c", code], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, (r.returncode, r.stderr[-1000:])
    return r.stdout.split()


MLA = """
from mega_dsa_cp_b200.tiles.hca import run_sparse_mla
B, H, D = %(B)s, 128, 576
q, kv = torch.zeros(B, 1, H, D, dtype=torch.bfloat16), torch.zeros(4, 1, D, dtype=torch.bfloat16)
pt, n = torch.zeros(B, 4, dtype=torch.int32), torch.zeros(0, dtype=torch.int32)   # (no lengths: the launcher refuses every call)
run_sparse_mla(q, None, kv, None, pt, %(o)s, %(lse)s, n, None, None, 0.04, n_splits=%(splits)s, stream=0)
"""
O, LSE = "torch.zeros(B, 1, H, 512, dtype=torch.bfloat16)", "torch.zeros(B, 1, H)"


def test_an_empty_batch_is_refused():
    assert _errors_of(MLA % dict(B=0, o=O, lse=LSE, splits=splits) for splits in (1, 2)) == ["MdcError"] * 2


def test_outputs_that_do_not_hold_the_rows_are_refused():
    fits = [(O, LSE), ("torch.zeros(3, H, 512)", "None"), ("torch.zeros(B, 2, H, 512)[:, :1]", LSE), ("torch.zeros(B, 1, H * 512)", LSE)]
    assert _errors_of(MLA % dict(B=2, o=o, lse=l, splits=1) for o, l in fits) == ["MdcError"] * len(fits)   # (as far as the launcher)
    small = [(o, LSE) for o in ("torch.zeros(1, 1, H, 512)", "torch.zeros(1, H, 512)", "torch.zeros(B, H // 2, 512)", "torch.zeros(B, H, 256)",
                                "torch.zeros(B, 1, H, 256)", "torch.zeros(B, H * 512)", "torch.zeros(B, H, 1024)[:, :, :512]")]
    small += [(O, "torch.zeros(1, 1, H)"), (O, "torch.zeros(B, 1, H // 2)")]
    got = _errors_of(MLA % dict(B=2, o=o, lse=l, splits=1) for o, l in small)
    assert all(e in ("AssertionError", "RuntimeError") for e in got), list(zip(small, got))


LOGITS = """
from mega_dsa_cp_b200.tiles.logits import run_fp4_paged_mqa_logits
B, pages = 2, 4
run_fp4_paged_mqa_logits(torch.zeros(8, 4608, dtype=torch.uint8), torch.zeros(B, 64, 128, dtype=torch.bfloat16), None, torch.zeros(B, 64),
                         torch.zeros(B, pages, dtype=torch.int32), torch.zeros(B, pages * 64), %d, fmt="nvfp4", page_tokens=64, stream=0)
"""


def test_chunks_of_no_pages_are_refused():
    assert _errors_of(LOGITS % pages_per_chunk for pages_per_chunk in (0, -1)) == ["AssertionError"] * 2


FINALIZE = """
from mega_dsa_cp_b200.comm.buffers import alloc_arena
from mega_dsa_cp_b200.events.symm import alloc_event_buffer
from mega_dsa_cp_b200.tiles.compress import CompressorState, launch_finalize, stats_bytes
st = CompressorState(1, 1, 0, 4, 0, device="cpu")   # (no entries: the launcher refuses every call)
f = torch.zeros(512)
launch_finalize(st, torch.zeros(1, dtype=torch.int32), alloc_arena({"stats": stats_bytes(4)}, 1, device="cpu"), "stats",
                alloc_event_buffer(1, device="cpu"), 0, f, f, 1e-6, torch.zeros(4, 64), fp8_scale=%s, stream=0)
"""


def test_a_zero_fp8_scale_is_refused():
    assert _errors_of(FINALIZE % scale for scale in ("0.02", "0.0")) == ["MdcError", "ZeroDivisionError"]


TEMPORARY = FINALIZE.replace("f = torch.zeros(512)", """f = torch.zeros(512)
class Fresh(type(st)):   # attributes that exist only while they are read
    attn_pool = property(lambda self: torch.zeros(1, 1, 512, dtype=torch.float8_e4m3fn), lambda self, v: None)
    k_valid = property(lambda self: torch.zeros(1, dtype=torch.int32), lambda self, v: None)
st = Fresh(1, 1, 0, 4, 0, device="cpu")""")


def test_attributes_made_on_the_fly_are_held_while_they_are_read():
    assert _errors_of([TEMPORARY % "0.02"] * 20) == ["MdcError"] * 20


def test_a_launch_leaves_the_shared_parameters_alone():
    """Threads that launch one layer share its MegaParams: a launch takes a copy, its own layer, trace and budget in it."""
    import pytest
    import torch

    from mega_dsa_cp_b200 import _native as N
    from mega_dsa_cp_b200.schedule.device import launch_params

    p = N.MegaParams(row_words=1, n_ctas=0, wait_budget_ns=7)   # (no blocks: the launcher refuses every call)
    p.layer.B = 3
    before, layer = bytes(p), N.LayerParams(B=5)
    with pytest.raises(N.MdcError):
        launch_params(p, layer, 0, torch.zeros(12, dtype=torch.int64), wait_budget_ns=9)
    assert bytes(p) == before
