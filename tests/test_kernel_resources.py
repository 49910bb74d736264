"""Registers and spills of the built kernels (the assembler's resource report, kept by the
build beside each object) against what their launches count on."""
import re


def resources(unit):
    """{mangled kernel name: (registers, spill store bytes, spill load bytes)} of one unit."""
    from gturbo3d_gb300 import build
    build.build()
    out, name, spills = {}, None, (0, 0)
    for line in (build.BUILD / f"{unit}.log").read_text().splitlines():
        if m := re.search(r"Compiling entry function '(\S+)'", line):
            name = m.group(1)
        elif m := re.search(r"(\d+) bytes spill stores, (\d+) bytes spill loads", line):
            spills = (int(m.group(1)), int(m.group(2)))
        elif (m := re.search(r"Used (\d+) registers", line)) and name:
            out[name] = (int(m.group(1)), *spills)
    return out


def kernels(unit, prefix):
    found = {k: v for k, v in resources(unit).items() if k.startswith(prefix)}
    assert found
    return found


def test_inverse_y_pass_spills(lib):
    """The step's inverse y pass is held to 64 registers for four blocks per SM; what does not
    fit stays within 32 bytes of stores and 40 of loads, and lines of up to 64 points fit."""
    found = {k: v for k, v in kernels("gt_kernels_f32.cu", "_ZN2gt8k_spass2ILi1E").items()
             if re.match(r"_ZN2gt8k_spass2ILi1ELi\d+ELb[01]ELb0E", k)}
    assert len(found) == 16   # 8 to 1024 points, launched alone or dependent
    for name, (regs, stores, loads) in found.items():
        short = re.match(r"_ZN2gt8k_spass2ILi1ELi[3-6]E", name)
        assert regs <= 64 and stores <= (0 if short else 32) and loads <= (0 if short else 40), (name, stores, loads)
