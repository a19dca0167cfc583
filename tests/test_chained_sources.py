"""Chained kernels (csrc/chained.cuh) live from before the kernels ahead of them end, so what those
wrote must not come through the read-only path: in the sources of such kernels and of the device
functions beside them no __ldg, and no pointer to const declared __restrict__."""
import re
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parent.parent / "lbm3d_bb_b200" / "csrc"
READ_ONLY = re.compile(r"const\s+(?:typename\s+)?[\w:]+\s*\*\s*__restrict__\s*(\w+)")


def _strip(text):
    return re.sub(r"//[^\n]*|/\*.*?\*/", "", text, flags=re.S)


def _kernels(text):
    """(name, parameters, body) of every __global__ function with a body."""
    for m in re.finditer(r"__global__\s+void\s", text):
        p = m.end()
        while True:  # past the launch bounds to the parameter list
            name = re.compile(r"\s*(\w+)\s*\(").match(text, p)
            q = name.end()
            depth = 1
            while depth:
                depth += {"(": 1, ")": -1}.get(text[q], 0)
                q += 1
            params = text[name.end():q - 1]
            p = q
            if name.group(1) != "__launch_bounds__":
                break
        brace = text.index("{", q)
        if text[q:brace].strip():
            continue  # a declaration
        e, depth = brace + 1, 1
        while depth:
            depth += {"{": 1, "}": -1}.get(text[e], 0)
            e += 1
        yield name.group(1), params, text[brace:e]


def _chained():
    out = []
    for path in sorted(CSRC.iterdir()):
        if path.suffix in (".cu", ".cuh"):
            out += [(path.name, *k) for k in _kernels(_strip(path.read_text())) if re.search(r"\bchain_(begin|wait)\(", k[2])]
    return out


def test_the_chained_kernels_are_found():
    names = {k[1] for k in _chained()}
    assert {"aa_step_kernel", "aa_rows_kernel", "ref_step_kernel", "body_flags_kernel", "conv_halo_kernel", "conv_bwdw_tc_kernel",
            "mse_kernel", "adam_kernel", "up2_concat8_kernel"} <= names


@pytest.mark.parametrize("kernel", _chained(), ids=lambda k: k[1])
def test_chained_kernels_read_with_ordinary_loads(kernel):
    _, _, params, body = kernel
    assert READ_ONLY.findall(params) == []
    assert "__ldg" not in body


def test_device_functions_beside_them():
    for name in ("unet3d.cu", "aa_impl.cuh", "ref_impl.cuh", "geometry.cu"):
        text = _strip((CSRC / name).read_text())
        assert "__ldg" not in text, name
        for m in re.finditer(r"__device__\s[^{;]*?\(([^{;]*?)\)\s*\{", text):
            if "__global__" not in m.group(0):
                assert "flags" not in READ_ONLY.findall(m.group(1)), (name, m.group(0)[:80])
                assert not {"Fp", "Rp"} & set(READ_ONLY.findall(m.group(1))), (name, m.group(0)[:80])
