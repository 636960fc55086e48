"""shapes_collide_noalloc clears at the start of every call all that it counts on being zero.

Its scratch outlives the calls.  Calls that overlap (the caller's fault) can leave the scans' tile
counters of several launches mixed; that must end with them and not reach later calls.  Running
overlapping calls would be a race on the GPU, so the cleared range is read from the source: counters
and scan words are members of one struct, and the call's first operation clears the struct.
"""
import re
from pathlib import Path

SOURCE = (Path(__file__).resolve().parent.parent / "shapes_gb300" / "csrc" / "shapes_gpu.cu").read_text()


def test_counters_and_scan_words_are_cleared_together():
    members = set(re.findall(r"(\w+)\[", re.search(r"struct NaWords \{(.*?)\n\};", SOURCE, re.S).group(1)))
    body = SOURCE[SOURCE.index('extern "C" int shapes_collide_noalloc'):]
    words = re.search(r"NaWords\* const (\w+) = ", body).group(1)
    state = re.search(r"ScanState \w+\{(.*?)\}", body, re.S).group(1).split(",")
    used = {m.strip() for m in state if not m.strip().startswith("k")}
    used.add(re.search(r"d\.counters = (.*?);", body).group(1))
    assert used == {f"{words}->{m}" for m in members}
    clear = body.index(f"cudaMemsetAsync({words}, 0, sizeof(NaWords), st)")
    assert clear < body.index("<<<") and clear < body.index("launch_chained(true, shapes::k_init_extents")
