"""What the kernels of chained launches (chain.cuh) read through the read-only path.

Such a kernel exists while its predecessor still writes, so only data that no kernel
of the chain writes may be read by __ldg or through a const __restrict__ pointer:
bases, mode weights, twiddles and slice transforms.  The sources are read as text,
since a GPU that happens to order such a load shows nothing."""
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "picard_b200", "csrc")

# kernel (or the device function that is its body) -> names it may read so
CHAINED = {
    "grid.cu": {"zero_kernel": set(), "finish_deposit_kernel": set(), "efield_kernel": set()},
    "outflow.cuh": {"outflow_mark_kernel": set(), "outflow_mark_quad_kernel": set(), "outflow_fill_kernel": set()},
    "particles_exact.cu": {"produce_count_kernel": set(), "produce_emit_kernel": set(), "inflow_stage_kernel": set(),
                           "inflow_place_kernel": set(), "add_count_kernel": set()},
    "particles_fast.cu": {"scan_tiles_kernel": set(), "scan_add_kernel": set(), "deposit_tile_c32_kernel": set(),
                          "load_group": set(), "load_species": set(), "load_pos": set()},
    "spectral.cu": {"spec_begin_kernel": set(), "spec_axis_kernel": {"Pe", "Po"},
                    "spec_norms_kernel": {"omx", "omy", "omz"}, "spec_scale_kernel": {"omx", "omy", "omz"}},
    "bcpot_fft.cu": {"fft_pass": {"tw"}, "fft_block": {"tw"}, "bcfft_rows_body": {"tw"},
                     "bcfft_cols_body": {"tw", "d0", "d1"}, "bcfft_invq_body": {"tw"}, "bcfft_invp_body": {"tw"},
                     "bcfft_stage": set(), "bcfft_run_kernel": set()},
}


def source(name):
    with open(os.path.join(CSRC, name)) as f:
        return re.sub(r"//[^\n]*", "", f.read())


def definition(text, name):
    """Parameters and body of the function `name`."""
    for m in re.finditer(rf"\b{name}\s*\(", text):
        depth, i = 1, m.end()
        while depth:
            depth += {"(": 1, ")": -1}.get(text[i], 0)
            i += 1
        params, rest = text[m.end():i - 1], text[i:].lstrip()
        if not rest.startswith("{"):
            continue
        start = i + text[i:].index("{")
        depth, j = 0, start
        while True:
            depth += {"{": 1, "}": -1}.get(text[j], 0)
            j += 1
            if depth == 0:
                return params, text[start:j]
    raise AssertionError(f"{name} not found")


@pytest.mark.parametrize("unit,name", [(u, n) for u, ns in CHAINED.items() for n in ns])
def test_read_only_loads_are_of_constant_data(unit, name):
    params, body = definition(source(unit), name)
    read = {re.search(r"(\w+)\s*$", p).group(1) for p in params.split(",")
            if "__restrict__" in p and re.search(r"\bconst\b[^*]*\*", p)}
    read |= set(re.findall(r"__ldg\(\s*(?:reinterpret_cast<[^>]*>\()?(\w+)", body))
    assert read <= CHAINED[unit][name]


def test_every_chained_kernel_is_listed():
    listed = {n for ns in CHAINED.values() for n in ns}
    for name in sorted(os.listdir(CSRC)):
        if not name.endswith((".cu", ".cuh")) or name == "chain.cuh":
            continue
        text = source(name)
        for m in re.finditer(r"__global__[^;{(]*?(?:__launch_bounds__\([^)]*\)\s*)?(\w+)\s*\(", text):
            if "chain_begin();" in definition(text, m.group(1))[1]:
                assert m.group(1) in listed, f"{name}: {m.group(1)}"
