"""The bench's reference arm where Remora's CPU path is not built: one line that says so, and success."""
from __future__ import annotations

import io
import json
import os
import sys
from contextlib import redirect_stdout
from pathlib import Path

ROOT = Path(__file__).resolve().parent.parent


def test_unavailable_reference_is_reported(monkeypatch):
    sys.path.insert(0, str(ROOT))
    import bench
    import oracle

    def missing(*args, **kwargs):
        raise FileNotFoundError("libremora_ref.so not built")

    monkeypatch.setattr(oracle, "Reference", missing)
    monkeypatch.delenv("RANK", raising=False)

    class Args:
        ref_n, n, nrhs, steps, warmup, gpus = 96, 32768, 4, 2, 1, 1

    buf = io.StringIO()
    with redirect_stdout(buf):
        bench.run_reference_arm(Args())
    line = json.loads(buf.getvalue())
    assert line == {"impl": "reference", "unavailable": "libremora_ref.so not built"}
