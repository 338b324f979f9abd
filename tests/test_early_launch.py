"""Early placement of small launches (programmatic stream serialization),
checked on the source: what a run cannot show without a race.

Every kernel waits for its predecessor before anything else, and releases its
successor only after that, so that at most one kernel of a stream is resident
and waiting; kernels launched that way do not take step data as read-only."""
import glob
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "turbid_b200", "csrc")
SOURCES = {os.path.basename(f): re.sub(r"//[^\n]*", "", open(f).read())
           for f in sorted(glob.glob(os.path.join(CSRC, "*.cu*")))}
TABLES = {"tw"}   # twiddles: written at set-up only


def kernels():
    for name, src in SOURCES.items():
        for m in re.finditer(r"__global__", src):
            brace = src.index("{", m.start())
            head = src[m.start():brace]
            params = max(re.finditer(r"(\w+)\(([^()]*)\)\s*$", head.rstrip() + " "), key=lambda k: k.end(), default=None)
            yield name, params.group(1), params.group(2), src[brace + 1:brace + 200].strip()


def test_wait_comes_before_release():
    body = re.search(r"void pdl_begin\(\) \{(.*?)\n\}", SOURCES["tg_common.cuh"], re.S).group(1)
    order = re.findall(r"griddepcontrol\.(\w+)", body)
    assert order == ["wait", "launch_dependents"]
    # and nowhere else, so no kernel releases its successor earlier
    assert sum(s.count("griddepcontrol") for s in SOURCES.values()) == 2


def test_every_kernel_begins_with_the_wait():
    found = list(kernels())
    assert len(found) > 30
    assert [k[:2] for k in found if not k[3].startswith("pdl_begin();")] == []


def test_early_kernels_read_no_step_data_as_constant():
    early = set()
    for src in SOURCES.values():
        early |= set(re.findall(r"launch_pdl\((\w+_kernel|k_\w+)\s*[<,]", src))
    # the z-operator products go through a local launch wrapper
    early |= {"zgemm_dense_kernel", "zgemm_sym_kernel"}
    params = {k[1]: k[2] for k in kernels()}
    assert early <= set(params) and len(early) > 15
    for k in sorted(early):
        for p in params[k].split(","):
            if "__restrict__" in p:
                assert re.search(r"(\w+)\s*$", p).group(1) in TABLES, (k, p)
