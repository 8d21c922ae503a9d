"""Orders in the kernels' sources that no run on one GPU shows to be missing: what has to have happened before another
block's shared memory is touched, and before a chained kernel reads what an earlier kernel writes."""
import glob
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "cupythia_b200", "csrc")


def _closing(s, i):
    """Index of the bracket that closes s[i]."""
    pair = {"(": ")", "{": "}"}[s[i]]
    depth = 0
    for k in range(i, len(s)):
        depth += (s[k] == s[i]) - (s[k] == pair)
        if not depth:
            return k
    raise ValueError("unbalanced source")


def _kernels():
    """name -> (parameters, body) of every kernel in csrc, comments removed."""
    out = {}
    for f in sorted(glob.glob(os.path.join(CSRC, "*.cu"))):
        s = re.sub(r"//[^\n]*|/\*.*?\*/", "", open(f).read(), flags=re.S)
        for m in re.finditer(r"__global__\s+(?:void\s+)?(?:__cluster_dims__\([^()]*\)\s*)?"
                             r"(?:__launch_bounds__\([^()]*(?:\([^()]*\))?[^()]*\)\s*)?(?:void\s+)?", s):
            n = re.match(r"\w+", s[m.end():])
            if n is None:
                continue
            i = s.index("(", m.end())
            j = _closing(s, i)
            k = re.match(r"\s*\{", s[j + 1:])
            if k is None:
                continue
            b = j + k.end()
            out[n.group()] = (s[i + 1:j], s[b + 1:_closing(s, b)])
    return out


KERNELS = _kernels()


def test_every_kernel_is_found():
    n = sum(len(re.findall(r"^\s*(?:template <[^>]*>\s*)?(?:static )?__global__", open(f).read(), flags=re.M))
            for f in glob.glob(os.path.join(CSRC, "*.cu")))
    assert len(KERNELS) == n >= 30


CLUSTERED = sorted(k for k, (_, b) in KERNELS.items() if "map_shared_rank" in b)


@pytest.mark.parametrize("name", CLUSTERED)
def test_no_block_touches_another_s_shared_memory_before_the_cluster_runs(name):
    """A pointer from map_shared_rank is used only after a cluster barrier that the block's start arrives at."""
    body = KERNELS[name][1]
    for m in re.finditer(r"(\w+)\s*=\s*\w+\.map_shared_rank", body):
        use = re.search(r"\b%s\b" % m.group(1), body[m.end():])
        assert use, m.group(1)
        assert re.search(r"\.(barrier_wait|sync)\(\)", body[:m.end() + use.start()]), (name, m.group(1))


# written once, when the handle is created
CONSTANT = {"cteq_g"}
CHAINED = sorted(k for k, (_, b) in KERNELS.items() if "cp_wait_previous()" in b)


@pytest.mark.parametrize("name", CHAINED)
def test_no_chained_kernel_touches_global_memory_before_its_wait(name):
    """Ahead of cp_wait_previous a kernel names none of its pointer parameters, and of a launch record's members only
    whether a pointer is null."""
    params, body = KERNELS[name]
    head = body[:body.index("cp_wait_previous()")]
    names = set(re.findall(r"\*\s*(?:__restrict__\s*)?(\w+)\s*(?:,|$)", params)) - CONSTANT
    assert not {n for n in names if re.search(r"\b%s\b" % n, head)}
    for rec in re.findall(r"(?:HadLaunch|UnwLaunch|FlowTrainBufs)\s+(\w+)", params):
        used = set(re.findall(r"(?<!if \()\b%s\.(\w+)" % rec, head))
        assert used <= {"nb", "n"}, (name, used)


def test_chained_kernels_are_launched_as_such():
    """Every kernel that a chained launch starts has the wait."""
    for f in glob.glob(os.path.join(CSRC, "*.cu")):
        for n in re.findall(r"cp_launch_chained(?:_smem)?\((k_\w+)", open(f).read()):
            assert n in CHAINED
