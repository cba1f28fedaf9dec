"""Rules of the kernels' sources that no run can show to be broken: a load on the wrong side of the wait for the launch before
reads the right values nearly always.  The sources are read as text, without comments."""
import glob
import os
import re

import pytest

from poor_mans_mamba_b200.kernels.build import CSRC_DIR


def source(path):
    with open(path) as fh:
        text = fh.read()
    return re.sub(r"//[^\n]*", "", re.sub(r"/\*.*?\*/", "", text, flags=re.S))


def closing(text, at, pair="{}"):
    """The place of the bracket that closes the one at `at`."""
    depth = 0
    for i in range(at, len(text)):
        depth += (text[i] == pair[0]) - (text[i] == pair[1])
        if depth == 0:
            return i
    raise AssertionError("unbalanced brackets")


def kernels():
    """(file:kernel, parameters, body) of every __global__ function."""
    out = []
    for path in sorted(glob.glob(os.path.join(CSRC_DIR, "*.cu"))):
        text = source(path)
        for m in re.finditer(r"__global__\s+void\s*(__launch_bounds__\s*)?", text):
            at = m.end()
            if m.group(1):
                at = closing(text, at, "()") + 1
            name = re.compile(r"\s*(\w+)\s*\(").match(text, at)
            end = closing(text, name.end() - 1, "()")
            body = re.compile(r"\s*\{").match(text, end + 1)
            if body:
                stop = closing(text, body.end() - 1)
                out.append((f"{os.path.basename(path)}:{name.group(1)}", text[name.end():end], text[body.end():stop]))
    assert len(out) > 60
    return out


KERNELS = kernels()


def marked(body):
    return {p.strip() for group in re.findall(r"\bpdl_written\(([^)]*)\)", body) for p in group.split(",")}


def uses(text, name):
    return re.search(rf"(?<![.\w]){name}\b(?!\s*\?)", text) is not None   # (neither a member, threadIdx.x, nor the question whether it is null)


def ahead_of_wait(body):
    """What a kernel runs before it has waited for the launch before it: the text up to the wait, named lambdas only where they are
    called there; a block with a wait of its own counts up to that wait."""
    ahead, at = "", 0
    while True:
        found = re.compile(r"\bpdl_wait\(\)").search(body, at)
        assert found, "a kernel that marks pointers waits"
        ahead += body[at:found.start()]
        depth, i = 0, found.start()
        while i >= 0 and depth >= 0:   # to the bracket that opens the block around this wait
            depth += (body[i] == "}") - (body[i] == "{")
            i -= 1
        if depth >= 0:
            break
        at = closing(body, i + 1)
    named = {}
    while True:
        m = re.search(r"\bauto (\w+) = \[[^\]]*\]\s*\([^)]*\)[^{};]*\{", ahead)
        if not m:
            break
        stop = closing(ahead, m.end() - 1)
        named[m.group(1)] = ahead[m.end():stop]
        ahead = ahead[:m.start()] + ahead[stop + 1:]
    called = True
    while called:
        called = [n for n in named if re.search(rf"\b{n}\(", ahead)]
        for n in called:
            ahead += named.pop(n)
    return ahead


@pytest.mark.parametrize("name,body", [pytest.param(n, b, id=n) for n, _, b in KERNELS if marked(b)])
def test_results_of_a_launch_are_read_behind_the_wait(name, body):
    """What a kernel marks as written by the launches before it, it does not touch before it has waited for them."""
    ahead = ahead_of_wait(body)
    assert [p for p in sorted(marked(body)) if uses(ahead, p)] == []


# Weights, and inputs of the step that are written before its first launch: no launch's result, so on neither side of a wait.
CONSTANT = {"w", "w_t", "bias", "norm_w", "gate_w", "w_gate", "w_proj", "w_proj_t", "mix", "in_w", "out_w", "post_w", "post_b", "post_alpha", "alpha", "sink", "mu",
            "correction", "pre_scale", "pre_bias", "dt_shift", "a_log", "d_skip", "z_bias", "table",
            "cu", "slots", "seq_of", "positions", "block_table", "rows", "tokens"}
# Read by asynchronous copies only (the compiler leaves them where they stand), or finished before the launch before let this one go.
OTHERWISE = {"attention_mma.cu:flash_paged_kernel": {"q", "pool"}, "ssd_tc.cu:ssd_tc_output_kernel": {"xbc", "z_raw"}}


def works_ahead(body):
    """Whether a kernel has code, not only declarations, ahead of its wait."""
    if not uses(body, "pdl_wait"):
        return False
    ahead = re.sub(r"(extern\s+)?__shared__[^;]*;|constexpr[^;]*;|using[^;]*;", "", ahead_of_wait(body))
    return re.search(r"\b(if|for|while)\b|__syncthreads|\bldf|\w\[", ahead) is not None


@pytest.mark.parametrize("name,params,body", [pytest.param(n, p, b, id=n) for n, p, b in KERNELS if works_ahead(b)])
def test_results_of_a_launch_are_marked_behind_the_wait(name, params, body):
    """The compiler may move what is read through a `const T* __restrict__` parameter above the wait once there is code in front
    of it: every such parameter is a constant of the step or is marked."""
    pointers = re.findall(r"\bconst\s+[\w:]+\s*\*\s*__restrict__\s+(\w+)", params)
    assert [p for p in pointers if p not in CONSTANT | marked(body) | OTHERWISE.get(name, set())] == []


@pytest.mark.parametrize("name,body", [pytest.param(n, b, id=n) for n, _, b in KERNELS if re.search(r"auto sync_\w+ = \[&\]\(\) \{ asm", b)])
def test_a_wait_that_gives_up_leaves_no_barrier_to_the_others(name, body):
    """Where the warps of a part of the block meet at a barrier of their own, a warp whose bounded wait gave up walks on with them:
    it leaves neither a loop nor the kernel on its own wait's answer, which the other warps' need not share."""
    body = body[re.search(r"auto sync_\w+ = \[&\]\(\) \{ asm", body).start():]
    answers = re.findall(r"\b(\w+) = (?:__all_sync\(0xffffffffu, )?mbar_wait\w*\(", body)
    failed = r"if \(!(?:mbar_wait\w*\(|" + "|".join(rf"{a}\b" for a in answers + ["wait_all"]) + ")"
    for m in re.finditer(failed, body):
        then = closing(body, body.index("(", m.start()), "()") + 1
        rest = body[then:].lstrip()
        end = closing(rest, 0) if rest.startswith("{") else rest.index(";")
        assert not re.search(r"\b(return|break)\b", rest[:end]), body[m.start():then]


def test_no_state_of_a_launcher_outlives_a_call():
    """Attributes, residency and SM counts belong to the current device, and calls come from several threads: what a launcher keeps
    for the calls after it is one atomic word that names its device, or the address of a driver function."""
    for path in sorted(glob.glob(os.path.join(CSRC_DIR, "*.cu*"))):
        for line in re.findall(r"^\s*static\s+[^;({]*[;={\[]", source(path), flags=re.M):
            assert re.search(r"static (constexpr|std::atomic<|EncodeTiledFn )", line), f"{os.path.basename(path)}: {line.strip()}"
