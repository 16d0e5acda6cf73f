"""Tensor parallelism on >= 2 GPUs: column/row-parallel shards, NVLink peer-memory all-reduce
written in this repo (no NCCL), vocab-parallel arg-max — against the CPU oracle.  t=4 runs the per-rank head layout of Qwen2.5-32B TP=4,
t=8 that of Llama-3-70B TP=8 (tests/tp_worker.py).  Skipped on a box with fewer GPUs — `bench.py --gpus N` runs the same check at t=N."""
import os
import subprocess
import sys

import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu
ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.mark.parametrize("t,extra", [(2, "{}"), (2, '{"tp_nvls": 1}'), (2, '{"tp_ar_bf16": 0}'), (4, "{}"), (8, "{}")])
def test_tensor_parallel_matches_oracle(t, extra):
    """default: bf16 peer-memory one-shot all-reduce for decode steps, two-shot for prefill-sized chunks; tp_nvls=1: the in-switch (multimem)
    decode all-reduce where the box offers multicast; tp_ar_bf16=0: fp32 partials"""
    if torch.cuda.device_count() < t:
        pytest.skip(f"needs {t} GPUs")
    cmd = [sys.executable, "-u", "-m", "torch.distributed.run", "--nnodes=1", f"--nproc-per-node={t}", "--master-addr", "127.0.0.1",
           "--master-port", str(29600 + t), os.path.join(ROOT, "tests", "tp_worker.py"), extra]
    r = subprocess.run(cmd, capture_output=True, text=True, timeout=600)
    sys.stdout.write(r.stdout[-3000:])
    assert r.returncode == 0 and "TP_OK" in r.stdout, r.stdout[-2000:] + r.stderr[-2000:]
