"""The self-checking build (-DMK_CHECK): which barriers it looks at, and the kernels under it on a GPU."""
import os
import pathlib
import re
import subprocess
import sys

import pytest

ROOT = pathlib.Path(__file__).resolve().parent.parent
CSRC = ROOT / "megacute_b200" / "csrc"


def barriers(text, call):
    """Name of the barrier in every `call(...)`: `&c->name[...]` / `&a->name` / a local pointer `full + sl`."""
    out = set()
    for m in re.finditer(call + r"\(", text):
        args = text[m.end():m.end() + 80]
        b = re.search(r"(?:&[ac]->|\b)(\w*(?:full|empty|free|done)\w*)\b", args)
        out.add(b.group(1) if b else args)
    return out


def test_every_barrier_armed_for_bulk_copies_is_checked():
    for f in sorted(CSRC.glob("op_*.cuh")):
        text = f.read_text()
        armed = barriers(text, "mbar_arrive_expect_tx")
        assert armed <= barriers(text, "check_phase(?:_warp)?"), f.name


def test_every_barrier_the_issuer_releases_is_checked():
    for name in ("op_gemm_tc_wide.cuh", "op_attention_tc.cuh", "op_gemm_tc.cuh"):
        text = (CSRC / name).read_text()
        released = barriers(text, "tc_commit") - {"acc_full"}          # (acc_full: two arrivals per instruction, the epilogue waits for both)
        assert released and released <= barriers(text, "check_phase(?:_warp)?") | barriers(text, "released"), name


@pytest.mark.gpu
def test_kernels_run_clean_under_the_self_check(cuda):
    """Tile linears of both heights, prefill attention of both head sizes, decode and streaming linears with the checks compiled in."""
    env = dict(os.environ, MEGACUTE_B200_CHECK="1")
    picks = ["tests/test_tiles.py", "tests/test_gpu_models.py::test_wide_tiles_many_per_cta_and_slot_kinds",
             "tests/test_gpu_models.py::test_streaming_and_tile_linears_alternate", "tests/test_gpu_models.py::test_batched_decode_small"]
    r = subprocess.run([sys.executable, "-m", "pytest", "-x", "-q", "-m", "gpu", *picks], cwd=ROOT, env=env, capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout[-3000:]
