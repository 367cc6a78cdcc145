"""Read off the kernels' sources. Kernels that may start before the ones ahead of them have ended wait for those, and nothing that
those may write is read through the non-coherent path, which const __restrict__ parameters and __ldg ask for; shared arrays
are aligned for their accesses."""
import re
from pathlib import Path

import ml_framework_b200

CSRC = Path(ml_framework_b200.__file__).parent / "csrc"


def _kernels():
    """(name, parameters, body) of every __global__ function."""
    for path in sorted(CSRC.rglob("*.cu")):
        text = re.sub(r"//[^\n]*", "", path.read_text())
        for m in re.finditer(r"__global__", text):
            depth, i = 0, text.index("{", m.end())
            head, j = text[m.end():i], i
            while True:
                depth += {"{": 1, "}": -1}.get(text[j], 0)
                if depth == 0:
                    break
                j += 1
            name, params = re.search(r"(\w+)\s*\(((?:[^()]|\([^()]*\))*)\)\s*$", head).groups()
            yield name, params, text[i:j]


def test_no_non_coherent_reads_under_overlap():
    seen = 0
    for name, params, body in _kernels():
        if "pdl_wait()" not in body:
            continue
        seen += 1
        assert not re.search(r"const[^,]*__restrict__", params), name
        assert "__ldg" not in body, name
    assert seen >= 12


def _given(text, name):
    """What a variable, an array or an array of function pointers of that name is given: (where, what)."""
    return [(m.start(), m.group(1)) for m in re.finditer(r"\b" + name + r"(?:\[[^\]]*\])*(?:\)\([^)]*\))?\s*=(?!=)([^;]*);", text)]


def _launched(text, name, kernels):
    """Kernels that `name` stands for at the end of this text."""
    if name in kernels:
        return {name}
    given = _given(text, name)
    if not given:
        return set()
    at, what = given[-1]
    return set().union(*(_launched(text[:at], word, kernels) for word in set(re.findall(r"[A-Za-z_]\w*", what)) - {name}))


def test_every_overlapped_launch_waits():
    waits = {name for name, _, body in _kernels() if "pdl_wait()" in body}
    kernels = {name for name, _, _ in _kernels()}
    launched = set()
    for path in CSRC.rglob("*.cu"):
        text = re.sub(r"//[^\n]*", "", path.read_text())
        for m in re.finditer(r"launch_pdl\(\s*(\w+)", text):
            found = _launched(text[:m.start()], m.group(1), kernels)
            assert found, (path.name, m.group(1))
            launched |= found
    assert {"norm_bwd_cta_kernel", "norm_fwd_row_kernel", "rope_kv_write_kernel", "paged_decode_kernel", "flash_fwd_ws_kernel"} <= launched
    assert launched <= waits


def test_shared_arrays_are_aligned_for_their_widest_access():
    """An array that is also read or written 16 bytes at a time says so where it is declared."""
    seen = 0
    for name, _, body in _kernels():
        for array in re.findall(r"reinterpret_cast<(?:const )?(?:uint4|int4|float4)\s*\*>\(&?(\w+)\b", body):
            declared = re.search(r"__shared__([^;]*?)\b" + array + r"\s*\[", body)
            if declared:
                seen += 1
                assert re.search(r"__align__\(\d*(16|32|64|128|1024)\)|\b(uint4|int4|float4)\b", declared.group(1)), (name, array)
    assert seen >= 1
