"""Loads of the kernels that a dependent launch may start while their predecessor still writes.

Such a kernel's lifetime overlaps its predecessor's, and a non-coherent load (`ld`, `__ldg`) is defined
only for data that stay unwritten for the kernel's lifetime. So in every kernel that calls
`pdl_enter` a non-coherent load may address an array that is constant over the loop, and nothing else: the root of
each such load is looked up here. CPU only."""
import glob
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "femtools.jl_b200", "csrc")

# Fields of the kernels' arguments that no kernel of a solver loop writes between two synchronisations:
# connectivity, geometry, phases, materials, history, prescribed data, preconditioners, scratch of the setup.
# (Not: v, P, temp, lam_v, lam_P, Tn, src_ip, dv, dP, Rv, R, RP, rate, mean.)
CONSTANT = set("""el2n dofsP geo_v geo_P geo_c geo phv php ph phases gammaP MP told eta_ip P0 P_old_ip temp0 Q Pf Pnum_in
    lin tile_list group T0 src mass grad diag load mask PC Rfill
    el2n_t dofs_t geo_t phase_t base_t apex_t eta_t pscale_t""".split())
# a scalar nodal field of the heat diffusion that is constant over the loop, under a name that others write
CONSTANT_IN = {"thermal3d_kernel": {"P"}}

NC = re.compile(r"(?<![\w:])(ld|__ldg|ldg_stream|load10)\s*\(")


def matching(s, i, pair):
    depth = 0
    for j in range(i, len(s)):
        depth += (s[j] == pair[0]) - (s[j] == pair[1])
        if depth == 0:
            return j
    raise AssertionError("unbalanced " + pair)


def kernels():
    out = {}
    for path in sorted(glob.glob(os.path.join(CSRC, "*.cu"))):
        with open(path) as f:
            s = re.sub(r"//[^\n]*", "", f.read())
        for m in re.finditer(r"__global__\s+void", s):
            i = m.end()
            b = re.compile(r"\s*__launch_bounds__\s*\(").match(s, i)
            if b:
                i = matching(s, b.end() - 1, "()") + 1
            name = re.compile(r"\s*(\w+)\s*\(").match(s, i)
            start = s.index("{", matching(s, name.end() - 1, "()"))
            body = s[start:matching(s, start, "{}") + 1]
            if "pdl_enter()" in body:
                out[name.group(1)] = body
    return out


KERNELS = kernels()


def roots(body, expr, seen=()):
    """Argument fields an address expression starts from, through local pointers."""
    fields = set(re.findall(r"\ba\.(\w+)", expr.split("+")[0]))
    if fields:
        return fields
    name = re.match(r"\W*(?:reinterpret_cast<[^(]*\()?\s*(\w+)", expr).group(1)
    found = set()
    for d in re.findall(r"\*\s*(?:const\s+)?%s\s*=\s*([^;]*);" % re.escape(name), body):
        if name not in seen:
            found |= roots(body, d, seen + (name,))
    return found or {"?" + name}


def test_the_loops_kernels_are_found():
    assert {"hex27_residual_kernel", "hex27_incr_kernel", "q9_residual_kernel", "hex27_adjoint_tile_kernel",
            "thermal3d_kernel", "thermal3d_tile_kernel", "cp_tile_kernel", "node_update_kernel"} <= set(KERNELS)


@pytest.mark.parametrize("name", sorted(KERNELS))
def test_non_coherent_loads_address_constant_arrays(name):
    body = KERNELS[name]
    allowed = CONSTANT | CONSTANT_IN.get(name, set())
    for m in NC.finditer(body):
        arg = body[m.end():matching(body, m.end() - 1, "()")]
        arg = re.sub(r"^ht_at\(", "", arg.strip())
        bad = roots(body, arg) - allowed
        assert not bad, "%s: non-coherent load of %s: %s(%s)" % (name, sorted(bad), m.group(1), arg)
