"""Rules that the CUDA sources keep and no run on one GPU would show broken: checked on
the text of the sources (no GPU)."""
import re

from conftest import ROOT

CSRC = ROOT / "beamz_b200" / "csrc"


def _functions(text):
    """Bodies of the functions at namespace level (they end in a brace in column 0)."""
    for m in re.finditer(r"^[^\s#/}][^;{}]*\([^;{}]*\)\s*\{\n(.*?)^\}", text, re.M | re.S):
        yield m.group(0).split("(")[0].split()[-1], m.group(1)


def test_warp_wide_tensor_memory_instructions_follow_a_warp_barrier():
    """tcgen05.ld, tcgen05.dealloc and the aligned cluster barrier need the whole warp at
    once. Lanes that skip a store (rows or pixels past the end) leave it split, so the
    function that issues one of them has to bring the lanes together first."""
    found = 0
    for path in sorted(CSRC.glob("*.cu")):
        for name, body in _functions(path.read_text()):
            code = re.sub(r"//[^\n]*", "", body)
            for m in re.finditer(r"tcgen05\.ld\.|tcgen05\.dealloc\.|barrier\.cluster\.arrive", code):
                found += 1
                before = code[:m.start()]
                assert "__syncwarp();" in before, f"{path.name}: {name}"
                between = before[before.rindex("__syncwarp();"):]
                assert "?" not in between and "&&" not in between, f"{path.name}: {name} branches after the barrier"
    assert found >= 5


def test_pair_epilogue_waits_as_one_warp():
    """The epilogue warps of the CTA-pair GEMM leave their loop together: a lane whose
    bounded wait ran out alone would miss the warp-wide accumulator loads of the others."""
    code = (CSRC / "bz_gemm.cu").read_text()
    body = code[code.index("gemm_pair_kernel(const __grid_constant__"):]
    body = body[body.index("warp >= 2"):body.index("arrive_rank0(tempty0")]
    assert re.findall(r"\w+\(0xffffffffu, tc_wait\(tfull0", body) == ["__all_sync(0xffffffffu, tc_wait(tfull0"]


def test_launch_settings_are_kept_per_device():
    """What a launcher sets on a kernel holds for the device that was current, and launchers
    run on several host threads: nothing remembers it in a plain static."""
    for path in sorted(CSRC.glob("*.cu*")):
        assert not re.findall(r"^\s+static (?:bool|int|unsigned|long long) .*", path.read_text(), re.M), path.name
