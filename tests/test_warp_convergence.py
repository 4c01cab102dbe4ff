"""Instructions that a whole warp has to reach together (tcgen05.ld and .st are .sync.aligned), by the kernels' source: accesses of tensor
memory converge their warp, and waits before them give all lanes one answer."""
import re
from pathlib import Path

KERNELS = Path(__file__).parent.parent / "ksanallm_b200" / "csrc" / "kernels"


def test_accesses_of_tensor_memory_converge():
    source = (KERNELS / "sm100_ptx.cuh").read_text()
    bodies = dict(re.findall(r"void (tmem_(?:ld|st)\d+)\([^)]*\)[^)]*\) \{\n(.*?)\n\}", source, re.S))
    assert set(bodies) == {"tmem_ld16", "tmem_ld32", "tmem_st16", "tmem_st32"}
    assert all(b.lstrip().startswith("__syncwarp();") for b in bodies.values())
    used = {f.name for f in KERNELS.glob("*.cu*") if re.search(r"tcgen05\.(ld|st)\.sync", f.read_text())}
    assert used == {"sm100_ptx.cuh"}                  # ... and there is no other way to them


def test_waits_of_a_warp_have_one_answer():
    # barriers that whole warps wait for and go on from only where the wait succeeded: accumulators, outputs, and scales packed by a warp
    lone = re.compile(r"(?<!__all_sync\(0xffffffffu, ok && )\bmbar_wait\(&?(tfull_bar|done_bar|o_full|o_done|pv_done|sf_empty|xs_ready)\b")
    assert [(f.name, m[0]) for f in KERNELS.glob("*.cu") for m in lone.finditer(f.read_text())] == []
