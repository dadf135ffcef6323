"""CPU checks of the native host module (csrc/host_bindings.cpp): what the runners refuse comes back as a Python
error, before anything reaches a device."""

import os
import subprocess
import sys

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def _error_of(body):
    """Name of the exception that `body` raises in a fresh interpreter (a crash there fails the test, not the session)."""
    code = "import sys\nsys.path.insert(0, %r)\nimport torch\ntry:\n" % ROOT
    code += "".join("    " + line + "\n" for line in body.strip().splitlines())
    code += "    print('NONE')\nexcept Exception as e:\n    print(type(e).__name__)\n"
    r = subprocess.run([sys.executable, "-c", code], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, (r.returncode, r.stderr[-1000:])
    return r.stdout.split()[-1]


MLA = """
from mega_dsa_cp_b200.tiles.hca import run_sparse_mla
B, H, D = %(B)s, 128, 576
q, kv = torch.zeros(B, 1, H, D, dtype=torch.bfloat16), torch.zeros(4, 1, D, dtype=torch.bfloat16)
pt, n = torch.zeros(B, 4, dtype=torch.int32), torch.zeros(B, dtype=torch.int32)
run_sparse_mla(q, None, kv, None, pt, %(o)s, %(lse)s, n, None, None, 0.04, n_splits=%(splits)s, stream=0)
"""


def test_an_empty_batch_is_refused():
    o, lse = "torch.zeros(B, 1, H, 512, dtype=torch.bfloat16)", "torch.zeros(B, 1, H)"
    for splits in (1, 2):
        assert _error_of(MLA % dict(B=0, o=o, lse=lse, splits=splits)) == "MdcError"


LOGITS = """
from mega_dsa_cp_b200.tiles.logits import run_fp4_paged_mqa_logits
B, pages = 2, 4
run_fp4_paged_mqa_logits(torch.zeros(8, 4608, dtype=torch.uint8), torch.zeros(B, 64, 128, dtype=torch.bfloat16), None, torch.zeros(B, 64),
                         torch.zeros(B, pages, dtype=torch.int32), torch.zeros(B, pages * 64), %d, fmt="nvfp4", page_tokens=64, stream=0)
"""


def test_chunks_of_no_pages_are_refused():
    for pages_per_chunk in (0, -1):
        assert _error_of(LOGITS % pages_per_chunk) == "AssertionError"
