"""Source rules of the programmatic dependent launches (csrc/pdl.cuh), read from
the CUDA sources: a kernel that waits for the grids before it may not let the
compiler load what they write ahead of the wait.  A latent race of this kind
shows in no result until a compiler or a register count changes, so the rule is
checked where it can be broken.
"""
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))),
                    "distributednavierstokes_b200", "csrc")

# tables of a context, written when it is created and by no kernel of a step
TABLES = {"twz", "twy", "twM", "twN", "twn", "lam1", "lam2", "lam3", "ymet", "cin", "ay", "by", "cy",
          "xph", "yph", "zph", "ph"}
# outputs that a kernel only writes, from values loaded past its wait
OUTPUTS = {"k_rfftx_any": {"S"}, "k_irfftx_any": {"out"}, "k_rfftx4": {"S"}, "k_irfftx4": {"out"},
           "k_gradmom_pipe": {"p_out"}, "k_ls_xsums": {"A"}, "k_ls_sums": {"out"}}
# read-only loads of tables, and of a closure's biases and scales (written by
# ordinary launches before the first convolution of a pass)
LDG = {"g.rdy", "g.rdyu", "lam1", "lam2", "lam3", "ay", "by", "cy", "cin", "twM", "twN", "a.bias", "a.oscale"}


def source(name):
    with open(os.path.join(CSRC, name)) as f:
        return re.sub(r"//[^\n]*", "", f.read())


def closing(text, i):
    """Index past the bracket that closes the one at i."""
    pair = {"(": ")", "{": "}"}[text[i]]
    depth = 0
    for j in range(i, len(text)):
        depth += (text[j] == text[i]) - (text[j] == pair)
        if depth == 0:
            return j + 1
    raise AssertionError("unbalanced source")


def kernels(text):
    """(name, parameters, body) of every __global__ function."""
    for m in re.finditer(r"__global__\s+void\b", text):
        i = m.end()
        bounds = re.match(r"\s*__launch_bounds__\s*", text[i:])
        if bounds:
            i = closing(text, i + bounds.end())
        name = re.match(r"\s*(\w+)\s*", text[i:])
        i += name.end()
        j = closing(text, i)
        k = text.index("{", j)
        if text[j:k].strip():
            continue  # a declaration
        yield name.group(1), text[i + 1:j - 1], text[k:closing(text, k)]


def dependents():
    for f in sorted(os.listdir(CSRC)):
        if f.endswith((".cu", ".cuh")):
            for name, params, body in kernels(source(f)):
                if "pdl_wait(" in body or "griddepcontrol.wait" in body:
                    yield name, params, body


DEPENDENTS = list(dependents())


def test_the_parser_sees_them():
    names = {k[0] for k in DEPENDENTS}
    assert {"k_momentum_march", "k_gradmom_pipe", "k_fftz_any", "k_y_any", "k_rfftx_any", "k_irfftx_any",
            "k_fftz4", "k_rfftx4", "k_irfftx4", "k_ythomas", "k_cn", "k_grad", "k_sfs_stage", "k_les_dt",
            "k_maxabs3", "k_conv", "k_wgrad", "k_infer_in", "k_sp_stage", "k_ls_modes"} <= names


@pytest.mark.parametrize("name,params,body", DEPENDENTS, ids=[k[0] for k in DEPENDENTS])
def test_what_other_kernels_write_is_read_through_plain_pointers(name, params, body):
    restricted = set(re.findall(r"__restrict__\s+(\w+)", params))
    assert restricted <= TABLES | OUTPUTS.get(name, set()), name
    assert set(re.findall(r"__ldg\(\s*&?([\w.]+)", body)) <= LDG, name
    # nothing is loaded through an output
    for out in OUTPUTS.get(name, set()):
        assert not re.search(rf"=\s*{out}\s*\[", body), (name, out)


def test_tensor_memory_is_taken_before_the_dependents_may_start():
    """A dependent block allocates tensor memory before it waits for the grid
    ahead of it.  Were it let in before that grid's blocks hold theirs, it could
    take the columns of an SM that one of them still needs, and neither would end."""
    text = source("cnn.cuh")
    helper = text[text.index("void tmem_alloc_then_trigger("):]
    helper = helper[helper.index("{"):closing(helper, helper.index("{"))]
    assert 0 <= helper.index("tmem_alloc(") < helper.index("griddepcontrol.launch_dependents")
    assert text.count("griddepcontrol.launch_dependents") == 1
    users = {k[0]: k[2] for k in kernels(text) if "tmem_free(" in k[2]}
    assert set(users) == {"k_conv", "k_wgrad"}
    for name, body in users.items():
        assert body.count("tmem_alloc_then_trigger(") == 1 and "tmem_alloc(" not in body, name
        assert "pdl_trigger(" not in body, name
        assert body.index("tmem_alloc_then_trigger(") < body.index("griddepcontrol.wait"), name


def test_shared_memory_limits_are_only_raised():
    """A kernel's dynamic shared-memory limit belongs to the kernel on the device:
    set to one context's size, it could drop below another's between that one's
    own set and its launch.  Only raise_smem (launch.h), which keeps the largest,
    sets it."""
    for f in sorted(os.listdir(CSRC)):
        if f.endswith((".cu", ".cuh", ".h")) and f != "launch.h":
            assert "cudaFuncAttributeMaxDynamicSharedMemorySize" not in source(f), f


def test_weights_ahead_of_the_wait():
    """k_conv copies its weights before it waits.  They are complete then as long as
    what runs between k_update, which writes them, and a convolution are ordinary
    launches without a trigger, or let their dependents start past their own wait."""
    host, device = source("cnn.cu"), source("cnn.cuh")
    bodies = {name: body for text in (host, device) for name, _, body in kernels(text)}
    conv = bodies["k_conv"]
    assert conv.index("bulk_load(wsm, a.wpack") < conv.index("griddepcontrol.wait")
    # nothing else that another kernel writes is touched before it
    ahead = conv[:conv.index("griddepcontrol.wait")]
    assert not re.search(r"a\.(bias|zin|target|out|zout|infer_out|oscale|loss_part)\b|tma4\(", ahead)
    ordinary = {"k_update", "k_tail", "k_crops", "k_batch_in"}
    for name in ordinary:
        assert re.search(rf"\b{name}<<<", host), name
        assert not re.search(rf"launch_(as|pdl)\([^;]*\b{name}\b", host), name
        assert "pdl_trigger(" not in bodies[name] and "launch_dependents" not in bodies[name], name
    body = bodies["k_infer_in"]
    assert body.index("pdl_wait(") < body.index("pdl_trigger(")
    # every kernel of the closure is one of these
    assert set(bodies) == ordinary | {"k_infer_in", "k_conv", "k_wgrad"}
