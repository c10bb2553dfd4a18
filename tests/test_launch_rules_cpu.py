"""Rules of programmatic launches (csrc/common/pdl.cuh) that the sources can be held to by reading: the launch
trigger of a kernel that allocates tensor memory comes behind the barrier after the allocation, and no
block leaves a kernel before it has waited for the kernels ahead of it. And which weights may be read ahead of the wait."""

import glob
import os
import re

import pytest
import torch

from arcticinference_b200 import ops

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "arcticinference_b200", "csrc")


def _kernels():
    """(file and name, body without comments) of every kernel that uses either instruction."""
    out = []
    for path in sorted(glob.glob(os.path.join(CSRC, "**", "*.cu*"), recursive=True)):
        text = re.sub(r"//[^\n]*", "", open(path).read())
        for m in re.finditer(r"__global__", text):
            name = re.compile(r"(\w+)\s*\((?=[^()]*(?:const|\*))").search(
                re.sub(r"__launch_bounds__\([^)]*\)", lambda x: " " * len(x.group()), text[m.end():]))
            at = text.index("{", m.end() + name.start())
            end, depth = at, 0
            while True:
                depth += {"{": 1, "}": -1}.get(text[end], 0)
                end += 1
                if depth == 0:
                    break
            body = text[at:end]
            if "pdl_wait()" in body or "pdl_trigger()" in body:
                out.append(("%s:%s" % (os.path.basename(path), name.group(1)), body))
    return out


KERNELS = _kernels()


def test_every_source_is_seen():
    assert len(KERNELS) >= 40 and sum("tmem_alloc" in b for _, b in KERNELS) >= 8


@pytest.mark.parametrize("name,body", [k for k in KERNELS if "tmem_alloc" in k[1]], ids=lambda v: v.split("{")[0])
def test_successors_start_after_tensor_memory_is_owned(name, body):
    owned = body.index("__syncthreads()", re.search(r"tmem_alloc\w*\(", body).start())
    triggers = [m.start() for m in re.finditer(r"pdl_trigger\(\)", body)]
    assert any(t > owned for t in triggers)
    for t in triggers:
        if t < owned:      # a block that allocates nothing: it leaves
            assert "return;" in body[t:body.index("}", t)], name


@pytest.mark.parametrize("name,body", KERNELS, ids=lambda v: v.split("{")[0])
def test_no_block_leaves_before_it_has_waited(name, body):
    first_wait = body.index("pdl_wait()")
    for m in re.finditer(r"\breturn;", body):
        assert m.start() > first_wait, name


def test_storages_are_known_by_identity():
    """A parameter that is gone is no parameter any more, whatever is allocated where it lay; views of one are."""
    known, w = ops.StorageSet(), torch.empty(1 << 20)
    known.add(w)
    assert w in known and w[3:7].view(1, -1) in known and torch.empty(8) not in known
    again = []
    del w
    for _ in range(64):
        again.append(torch.empty(1 << 20))
        assert again[-1] not in known
    for i in range(64):        # (addresses of the objects behind the storages are not used again either)
        t = torch.empty(16 + i)
        known.add(t)
        del t
        assert torch.empty(16 + i) not in known
    known.add(again[0])
    assert again[0] in known and len(known) <= 64 + 2
    known.clear()
    assert again[0] not in known
