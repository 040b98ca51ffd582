"""Which kernels a piece of work launches and how long they take, by torch's profiler in a child process."""
import json
import os
import subprocess
import sys
from pathlib import Path

ROOT = Path(__file__).resolve().parent.parent
PROLOGUE = f"""
import json, sys
sys.path[:0] = [{str(ROOT / "tsne-h2pack-python_b200")!r}, {str(ROOT / "oracle")!r}, {str(ROOT / "tests")!r}]
import numpy as np
import torch
from torch.profiler import ProfilerActivity, profile
import oracle as O
from helpers import Engine
from test_gpu_lists import _ring_P
torch.zeros(1, device="cuda")
with profile(activities=[ProfilerActivity.CUDA]) as prof:
"""
EPILOGUE = """
    torch.cuda.synchronize()
print("KERNELS" + json.dumps({e.key: e.device_time_total / e.count for e in prof.key_averages()}))
"""


def kernels_of(code, **env):
    """The kernels that `code` launches: name (with template arguments) -> mean microseconds of a
    launch; env: environment variables, None to leave one unset."""
    e = dict(os.environ)
    for k, v in env.items():
        e.pop(k, None)
        if v is not None:
            e[k] = v
    src = PROLOGUE + "".join(f"    {line}\n" for line in code.strip().splitlines()) + EPILOGUE
    r = subprocess.run([sys.executable, "-c", src], env=e, capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout + r.stderr
    return {k: t for k, t in json.loads(r.stdout[r.stdout.rindex("KERNELS") + 7:]).items() if "k_" in k}
