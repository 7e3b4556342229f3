"""Which loads of the step kernels take the read-only path (__ldg).

A step's passes start while their predecessor drains (programmatic dependent
launch), so a field that some pass of the step or of the substep writes may
change while they run.  CUDA allows the read-only path only for data that
nothing writes during the kernel's life: the static fields, and any field in
k_fluid, which is launched after its predecessor in full.
"""
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "mpcns_mercury_b200", "csrc")
# the fields that a solve's preparation sets and no pass of a step writes
STATIC = {"cAMB", "cBAX", "cBAY", "cBAZ", "cDRX", "cDRY", "cDRZ", "cLEX", "cTPX", "cWB", "cWJ", "cALX", "cALY", "cALZ",
          "cBFX", "cBFY", "cBFZ", "cRW", "cETAR", "cFNX", "cFNY", "cFNZ", "cUCK", "cFM", "cIHX", "cIHY", "cIHZ"}
# locals that name one of them
LOCAL = {"cd": {"cDRX", "cDRY", "cDRZ"}, "ci": {"cIHX", "cIHY", "cIHZ"}}


def source():
    with open(os.path.join(CSRC, "mhd_kernels.cu")) as f:
        return re.sub(r"//[^\n]*", "", f.read())


def body(s, head):
    """The brace block that follows `head`."""
    i = s.index("{", s.index(head))
    depth = 0
    for q in range(i, len(s)):
        depth += {"{": 1, "}": -1}.get(s[q], 0)
        if depth == 0:
            return s[i:q + 1]
    raise AssertionError(head)


def test_ldg_only_in_the_static_accessors():
    s = source()
    for head in ("R fixed1(int comp", "double ldm(int comp", "static void load(T *to", "Vc fixed(int comp", "Vc stat(int comp",
                 "R stat1(int comp", "Vc lm(int comp"):
        s = s.replace(body(s, head), "{}")
    assert "__ldg" not in s
    for head in ("Vc lv(int comp", "R ld(int comp"):
        assert "load(" not in body(s, head)


def test_static_accessors_only_on_static_fields():
    s = source()
    fluid = s[s.index("struct FluidCell"):s.index("void flip_solve")]
    rest = s.replace(fluid, "")
    found = set()
    for m in re.finditer(r"\bB\.(?:fixed|fixed1|stat|stat1)\((\w+)", rest):
        found.add(m.group(1))
    for m in re.finditer(r"\bB\.fixed_upper\(\w+, (\w+)", rest):
        found.add(m.group(1))
    assert found and found <= STATIC | set(LOCAL), found - STATIC - set(LOCAL)
    for name, fields in LOCAL.items():
        for m in re.finditer(r"const int %s = ([^;]*);" % name, rest):
            assert set(re.findall(r"\bc[A-Z]\w+", m.group(1))) <= fields


@pytest.mark.parametrize("static", sorted(STATIC))
def test_static_fields_are_not_stored_by_a_step(static):
    """No pass but the preparation's (k_face_normals, k_res_w, k_sing_setup) stores one."""
    s = source()
    for head in (" k_face_normals(Dir", " k_res_w(Dir", " k_sing_setup(Dir"):
        s = s.replace(body(s, head), "{}")
    assert not re.search(r"\bB\.st\(%s\b|\bput\(%s\b|B\.c\(%s\b[^;]*\]\s*=[^=]|AT\(%s\b[^;]*\)\s*=[^=]" % ((static,) * 4), s)


def test_fluid_pass_is_launched_in_full():
    with open(os.path.join(CSRC, "mhd_ctx.cu")) as f:
        s = re.sub(r"//[^\n]*", "", f.read())
    assert re.search(r"b->after_flip \|\| k == SK_FLUID\b", body(s, "void launch(mhd_batch *b"))
    direct = re.findall(r"launch_step_kernel\(SK_FLUID[^;]*;", s)
    assert direct and all(c.rstrip(";").endswith(", true)") for c in direct)
