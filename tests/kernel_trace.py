"""Which kernels a call launched, from torch's device activity records."""
import json
import os
import re
import tempfile
import time

import pytest


def _records(backend, call):
    import torch
    from torch.profiler import ProfilerActivity, profile

    backend.sync()
    with profile(activities=[ProfilerActivity.CUDA]) as prof:
        time.sleep(0.05)  # (records outside the window are dropped, and the device's clock is not the host's)
        call()
        backend.sync()
        torch.cuda.synchronize()
        time.sleep(0.05)
    with tempfile.TemporaryDirectory() as d:
        path = os.path.join(d, "trace.json")
        prof.export_chrome_trace(path)
        with open(path) as f:
            events = json.load(f)["traceEvents"]
    for e in sorted((e for e in events if e.get("cat") == "kernel"), key=lambda e: e["ts"]):
        m = re.search(r"(\w+_kernel)(?:<(.*?)>)?\(", e["name"].replace("(bool)1", "true").replace("(bool)0", "false").replace("(int)", ""))
        if m:
            yield m.group(1), m.group(2) or "", tuple(e["args"]["grid"])


def launched(backend, call, *groups):
    """(name, template arguments, grid) of the kernels named in groups, in order.  Each group is a tuple of names, one of which the call launches.  Now and then the
    records of a call are lost, so it is repeated until every group has one; without any the test is skipped."""
    for _ in range(8):
        seen = [r for r in _records(backend, call) if any(r[0] in g for g in groups)]
        if all(any(r[0] in g for r in seen) for g in groups):
            return seen
    pytest.skip("no device activity records on this machine")
