"""Which kernels a call launched: (name, template arguments, grid) in order, from torch's device activity records."""
import json
import os
import re
import tempfile

import pytest


def launched(backend, call):
    import torch
    from torch.profiler import ProfilerActivity, profile

    backend.sync()
    with profile(activities=[ProfilerActivity.CUDA]) as prof:
        call()
        backend.sync()
        torch.cuda.synchronize()
    with tempfile.TemporaryDirectory() as d:
        path = os.path.join(d, "trace.json")
        prof.export_chrome_trace(path)
        with open(path) as f:
            events = json.load(f)["traceEvents"]
    kernels = sorted((e for e in events if e.get("cat") == "kernel"), key=lambda e: e["ts"])
    if not kernels:
        pytest.skip("no device activity records on this machine")
    names = [re.search(r"(\w+_kernel)(?:<(.*?)>)?\(", e["name"].replace("(bool)1", "true").replace("(bool)0", "false").replace("(int)", "")) for e in kernels]
    return [(n.group(1), n.group(2) or "", tuple(e["args"]["grid"])) for n, e in zip(names, kernels) if n]
