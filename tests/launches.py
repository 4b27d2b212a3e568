"""What a call puts on the GPU: its kernel launches as the profiler lists them."""
import json

import torch


def launches(fn, tmp_path):
    """[(kernel name, grid, block)] of fn()'s launches, in their order."""
    fn()                                   # (whatever is made once)
    torch.cuda.synchronize()
    with torch.profiler.profile(activities=[torch.profiler.ProfilerActivity.CUDA]) as prof:
        fn()
        torch.cuda.synchronize()
    path = str(tmp_path / "trace.json")
    prof.export_chrome_trace(path)
    with open(path) as f:
        events = [e for e in json.load(f)["traceEvents"] if e.get("cat") == "kernel"]
    return [(e["name"], tuple(e["args"]["grid"]), tuple(e["args"]["block"])) for e in sorted(events, key=lambda e: e["ts"])]
