"""The sweep solve's steps are dependent launches: step k + 1 is resident while
step k still writes the pending right-hand sides A and the finished tiles F, so
nothing of these two arrays may be read with the non-coherent load (__ldg),
which is defined only for data that no running kernel writes.  Checked in the
source, since a stale read shows up on the device by timing alone."""
import os
import re

SRC = os.path.join(os.path.dirname(os.path.abspath(__file__)), os.pardir, "hmatrix.jl_b200", "csrc", "hm_lu.cu")


def sweep_functions():
    """{name: body} of the device functions a sweep step runs."""
    text = re.sub(r"//[^\n]*", "", open(SRC).read())
    out = {}
    for m in re.finditer(r"\b(sweep_z|sweep_z1|sweep_update|sweep_finish|lu_sweep_kernel)\s*\([^;{]*\)\s*\{", text):
        depth, i = 1, m.end()
        while depth:
            depth += {"{": 1, "}": -1}.get(text[i], 0)
            i += 1
        out[m.group(1)] = text[m.end():i]
    return out


def test_sweeps_read_what_a_step_writes_with_plain_loads():
    bodies = sweep_functions()
    assert set(bodies) == {"sweep_z", "sweep_z1", "sweep_update", "sweep_finish", "lu_sweep_kernel"}
    for name, body in bodies.items():
        # names bound to A or F, directly or through one another
        written = {"A", "F", "ys"}
        for _ in range(4):
            for var, rhs in re.findall(r"double\s*\*\s*(\w+)\s*=\s*([^;]+);", body):
                if re.match(r"\s*(%s)\b" % "|".join(written), rhs):
                    written.add(var)
        for arg in re.findall(r"__ldg\(\s*-?\s*(\w+)", body):
            assert arg not in written, "%s: non-coherent load of %s" % (name, arg)
