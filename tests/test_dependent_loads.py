"""Kernels launched as programmatic dependents (pdl_enter) are resident while
the previous kernel on the stream still writes their inputs.  ld.global.nc is
defined for data that is read-only for the kernel's lifetime, so in the sources
of these kernels it may only load what is complete since finalize: through
ld4_nc or __ldg of the reference records and the bond lists, or through a
const __restrict__ kernel parameter (which lets the compiler choose it) of the
masses."""
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "peridyn_b200", "csrc")
UNITS = ["pd_exact.cu", "pd_fast.cu", "pd_solver.cu", "pd_contact.cu"]


def _code(unit):
    s = open(os.path.join(CSRC, unit)).read()
    return re.sub(r"//[^\n]*|/\*.*?\*/", "", s, flags=re.S)


def _body(s, at):
    """Text from `at` (a function's parameter list) to the end of its body."""
    i = s.index("{", at)
    depth = 0
    for j in range(i, len(s)):
        depth += {"{": 1, "}": -1}.get(s[j], 0)
        if depth == 0:
            return s[i:j + 1]


def test_non_coherent_loads_read_finalized_data_only():
    users = 0
    for unit in UNITS:
        s = _code(unit)
        for m in re.finditer(r"ld\.global\.nc", s):
            owner = re.findall(r"(\w+)\(const double4 \*p\) \{", s[:m.start()])
            assert owner and owner[-1] == "ld4_nc", f"{unit}: ld.global.nc outside ld4_nc"
        for arg in re.findall(r"\bld4_nc\(([^()]*)\)", s):
            if arg != "const double4 *p":
                assert arg.startswith("g.x4 +"), f"{unit}: ld4_nc({arg})"
                users += 1
        for arg in re.findall(r"__ldg\((?:reinterpret_cast<[^>]*>\()?(\w+)", s):
            assert arg in ("nb", "np", "spp", "p"), f"{unit}: __ldg({arg})"
    assert users


def test_dependent_kernels_take_written_arrays_without_restrict():
    kernels = []
    for unit in UNITS:
        s = _code(unit)
        for m in re.finditer(r"__global__[^;{]*?\b(k_\w+)\(([^{;]*)\)\s*\{", s):
            name, params = m.group(1), m.group(2)
            if "pdl_enter()" not in _body(s, m.end() - 1):
                continue
            kernels.append(name)
            for par in re.findall(r"const \w+ \*__restrict__ (\w+)", params):
                assert par == "mass", f"{name}: const __restrict__ {par}"
    assert {"k_theta_slice", "k_force_slice", "k_advance", "k_qs_apply", "k_fc12", "k_step", "k_theta", "k_td"} - set(
        kernels) <= {"k_step", "k_theta", "k_td"}  # (those enter through their bodies and take one struct)
