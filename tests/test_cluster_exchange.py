"""The exchange of a column's candidates between the CTAs of the LU panel's cluster, as a model whose
interleavings are all walked: warps publish for their CTA, meet at its barrier, each sends what was
published to the CTA that it serves, and waits until one warp of every CTA has sent to its own. The
number of copies of each buffer is taken from the kernel's source."""
from __future__ import annotations

import re
from pathlib import Path

SOURCE = (Path(__file__).resolve().parents[1] / "remora_b200" / "csrc" / "lu.cu").read_text()
LOCAL = ["mine", "top", "whi", "wlo", "widx"]  # written before the CTA's barrier, read by every warp after it
REMOTE = ["cand_row", "crow", "cand_key"]      # written by other CTAs, read after the wait


def _copies(name: str) -> int:
    """2 where the buffer's first dimension is the column's parity in its declaration and at each use."""
    struct = re.search(r"struct ClusterSmem \{.*?\n\};", SOURCE, re.S).group(0)
    dims = re.search(rf"\b{name}((?:\[[^\]]+\])+)", struct).group(1)
    uses = re.findall(rf"\bsm\.{name}(\[[^\]]+\])?", SOURCE)
    assert len(uses) >= 2, name
    return 2 if dims.startswith("[2]") and all(u == "[par]" for u in uses) else 1


def _walk(local: int, remote: int, ctas: int = 2, columns: int = 5) -> bool:
    """Whether every warp always sends and reads its own column's values. Warp w of a CTA serves CTA w;
    a warp's place is 4 t + step: 0 publish, 1 barrier and send, 2 wait, 3 read."""
    warps = [(c, w) for c in range(ctas) for w in range(ctas)]
    start = (tuple(0 for _ in warps), tuple([-1] * local * len(warps)), tuple([-1] * remote * len(warps)))
    seen, todo = {start}, [start]
    while todo:
        places, published, received = todo.pop()
        for i, (c, w) in enumerate(warps):
            t, step = divmod(places[i], 4)
            if t == columns:
                continue
            pub, rec = list(published), list(received)
            if step == 0:
                pub[(t % local) * len(warps) + i] = t
            elif step == 1:  # all of the CTA's warps have published this column: the barrier
                if any(places[j] < 4 * t + 1 for j, (d, _) in enumerate(warps) if d == c):
                    continue
                if any(pub[(t % local) * len(warps) + j] != t for j, (d, _) in enumerate(warps) if d == c):
                    return False
                rec[(t % remote) * len(warps) + w * ctas + c] = t
            elif step == 2:  # warp c of every CTA has sent this column's message to CTA c
                if any(places[d * ctas + c] < 4 * t + 2 for d in range(ctas)):
                    continue
            elif any(rec[(t % remote) * len(warps) + c * ctas + d] != t for d in range(ctas)):
                return False
            now = (places[:i] + (places[i] + 1,) + places[i + 1:], tuple(pub), tuple(rec))
            if now not in seen:
                seen.add(now)
                todo.append(now)
    return True


def test_one_copy_would_race():
    assert not _walk(1, 2) and not _walk(2, 1)


def test_the_kernel_has_two_copies_and_none_is_overwritten_early():
    copies = {name: _copies(name) for name in LOCAL + REMOTE}
    assert set(copies.values()) == {2}, copies
    assert _walk(2, 2)
