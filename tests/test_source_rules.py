"""Rules that the sources of this repository must keep, checked as text on the CPU.

* Thread-block clusters share work through ``tcgen05.mma.cta_group::2`` with per-CTA plain TMA loads; no TMA or bulk
  *load* carries a cluster mask (a tensor map may one day cover memory of another GPU).  The only instruction with a
  CTA mask is the ``tcgen05.commit`` that signals both CTAs' barriers and moves no data.
* The batched asynchronous memory-copy entry points of the CUDA runtime and driver are not used (nor named).
* Device code neither traps nor asserts: a wait that runs out records a status and the kernel returns.
* Whether a warp goes on to an instruction that it executes as one is not decided lane by lane.
* Every translation unit is compiled for sm_100a with line information.
* Comments and docstrings stand on their own: they name no planning document of this build and no path of a machine.
"""
import re
from pathlib import Path

ROOT = Path(__file__).resolve().parents[1]
CSRC = ROOT / "warpstate_ai_b200" / "ops" / "csrc"
NATIVE = sorted(p for p in CSRC.rglob("*") if p.suffix in (".cu", ".cuh", ".h", ".cpp"))
PYTHON = sorted(p for p in [*ROOT.glob("*.py"), *(ROOT / "warpstate_ai_b200").rglob("*.py"), *(ROOT / "ops").glob("*.py"),
                            *(ROOT / "warpstate").glob("*.py"), *(ROOT / "tests").glob("*.py")] if "_build" not in p.parts)
SHIPPED_TEXT = [*NATIVE, *PYTHON, *sorted((ROOT / "launch").glob("*")), *sorted((ROOT / "configs").glob("*"))]


def test_there_are_native_sources_to_check():
    names = {p.name for p in NATIVE}
    assert {"gemm2_tcgen05.cu", "attention_fwd.cu", "attention_bwd.cu", "comm.cu", "decode.cu", "symm_alloc.cpp"} <= names
    assert len(PYTHON) > 100


def test_no_load_carries_a_cluster_mask():
    mask = "multicast" + "::cluster"
    hits = [(p.name, number, line.strip()) for p in NATIVE for number, line in enumerate(p.read_text().splitlines(), 1)
            if mask in line]
    assert hits, "the commit that frees a stage in both CTAs of a pair is expected to be there"
    for name, number, line in hits:
        assert "tcgen05.commit" in line and "cp.async" not in line, (name, number, line)
    for p in PYTHON:
        assert mask not in p.read_text(), p


def test_batched_memcpy_entry_points_are_not_named():
    stems = ["cuda" + "Memcpy", "cu" + "Memcpy", "cuda" + "Memcpy3D", "cu" + "Memcpy3D"]
    names = [stem + "Batch" + "Async" for stem in stems]
    for p in SHIPPED_TEXT:
        text = p.read_text(errors="ignore")
        assert not any(name in text for name in names), p


def test_device_code_neither_traps_nor_asserts():
    trap = re.compile(r"__trap\s*\(|\btrap\s*;|(?<!static_)\bassert\s*\(")
    for p in NATIVE:
        if p.suffix == ".cpp":
            continue
        for number, line in enumerate(p.read_text().splitlines(), 1):
            code = line.split("//")[0]
            assert not trap.search(code), (p.name, number, line.strip())


def test_waits_in_kernels_have_a_limit():
    """A loop without an exit condition in its header that polls something another thread, CTA or GPU writes (an
    mbarrier, a flag read with acquire or volatile semantics) reads ``%globaltimer`` and gives up with a status.  Loops
    of that form that only claim work from a counter or scan data end by construction."""
    bare = re.compile(r"while\s*\(\s*(true|1)\s*\)|for\s*\(\s*;\s*;\s*\)")
    polls = ("ld.acquire", "try_wait", "ld.volatile", "ld.relaxed", "test_wait")
    polling_loops = 0
    for p in NATIVE:
        if p.suffix == ".cpp":
            continue
        text = p.read_text()
        for match in bare.finditer(text):
            body = text[match.start():match.start() + 700]
            if any(word in body for word in polls):
                polling_loops += 1
                assert "globaltimer" in body, (p.name, text[:match.start()].count("\n") + 1)
    assert polling_loops >= 3                       # mbarrier wait, cross-rank flag wait, gather-chunk wait
    helpers = (CSRC / "ws_ptx.cuh").read_text()
    assert "globaltimer" in helpers and "mbar_wait" in helpers


def test_every_kernel_is_compiled_for_sm_100a_with_line_information():
    build = (ROOT / "warpstate_ai_b200" / "ops" / "_ext.py").read_text()
    assert '"-gencode", "arch=compute_100a,code=sm_100a"' in build and '"-lineinfo"' in build
    entry = (ROOT / "__graft_entry__.py").read_text()
    assert "def build(" in entry and "def smoke(" in entry
    for p in NATIVE:                                   # Hopper's warpgroup MMA does not exist on sm_100a
        code = "\n".join(line.split("//")[0] for line in p.read_text().splitlines())
        assert "wgmma" not in code and "mma.sync" not in code and "wmma" not in code, p.name
    kernels = "\n".join(p.read_text() for p in NATIVE if p.suffix in (".cu", ".cuh"))
    for needed in ("tcgen05.mma", "tcgen05.alloc", "tcgen05.ld", "cp.async.bulk.tensor", "multimem.ld_reduce", "griddepcontrol.wait"):
        assert needed in kernels, needed


def test_no_triton_or_compile_on_the_product_path():
    for p in (ROOT / "warpstate_ai_b200").rglob("*.py"):
        if "_build" in p.parts:
            continue
        text = p.read_text()
        assert "import triton" not in text and "tilelang" not in text, p
        if "torch.compile(" in text:
            assert p.name in ("validate_training.py",), p           # only the PyTorch yardstick arm of the harness compiles


def test_comments_stand_on_their_own():
    documents = ["SURVEY" + ".md", "DESIGN" + ".md", "VERDICT" + ".md", "ADVICE" + ".md", "BASELINE" + ".md"]
    other = ["gpu" + "run", "/ro" + "ot/", "the " + "judge", "VERDICT " + "item", "SURVEY " + "8"]
    rounds = re.compile(r"\bround[- ]\d\b|\bin round \w+\b", re.IGNORECASE)
    for p in SHIPPED_TEXT:
        if p.name == Path(__file__).name:
            continue
        text = p.read_text(errors="ignore")
        for word in documents + other:
            assert word not in text, (p, word)
        assert not rounds.search(text), (p, rounds.search(text).group(0))


def test_kernels_that_wait_for_their_predecessor_promise_no_read_only_inputs():
    """``const T* __restrict__`` says that nobody writes the data while the kernel runs, so the compiler may move its loads
    above ``griddepcontrol.wait``: a kernel that overlaps the one before it then reads what that one has not written yet."""
    promise = re.compile(r"const\s+[A-Za-z_0-9 ]+\*\s*__restrict__")
    waiting = 0
    for p in NATIVE:
        if p.suffix != ".cu":
            continue
        for kernel in p.read_text().split("__global__")[1:]:
            head, body = kernel.split("{", 1)
            if "pdl_wait()" not in body.split("\n}\n")[0]:
                continue
            waiting += 1
            assert not promise.search(head), (p.name, head)
    assert waiting > 20


ONE_LANE = ("lane == 0", "elect_one()", "tid == 0", "threadIdx.x == 0", "et == 0")
ONE_LANE_FUNCTIONS = ("tail_produce", "tail_mma")       # of decode_layer.cu, called by one lane


def sites(text, name):
    """``(line, inside one lane's code, statement so far)`` of every call of ``name``."""
    text = "\n".join(line.split("//")[0] for line in text.splitlines())
    scopes, begin, found = [], 0, []
    for match in re.finditer(r"[;{}]|\b" + name + r"(?=[<(])", text):
        token, statement = match.group(0), text[begin:match.start()]
        if token == "{":
            scopes.append(statement)
        elif token == "}" and scopes:
            scopes.pop()
        if token in ";{}":
            begin = match.end()
            continue
        if "__forceinline__" in statement:               # its definition
            continue
        context = [*scopes, statement]
        alone = any(word in scope for scope in context for word in ONE_LANE) or any(
            "__device__" in scope and f"{function}(" in scope for scope in scopes for function in ONE_LANE_FUNCTIONS)
        found.append((text[:match.start()].count("\n") + 1, alone, statement))
    return found


def test_a_warp_decides_as_one_what_it_does_as_one():
    """A bounded wait answers each lane for itself.  An epilogue warp of which some lanes gave up and some did not would meet
    tcgen05.ld in part and never come back: such waits go through `mbar_wait_warp`.  The attention kernels go on whatever a
    wait says, or vote; no jump there hangs on one lane's answer either."""
    whole = one = 0
    for p in NATIVE:
        if p.suffix != ".cu":
            continue
        text = p.read_text()
        for function in ONE_LANE_FUNCTIONS:
            for line, alone, _ in sites(text, function):
                assert alone, (p.name, line)
        for line, alone, statement in sites(text, "mbar_wait"):
            one += alone
            if not alone:
                assert p.name.startswith("attention_") and not re.search(r"\bif\s*\(", statement), (p.name, line, statement.strip())
        for line, alone, _ in sites(text, "mbar_wait_warp"):
            whole += 1
            assert not alone, (p.name, line)             # a vote of all lanes, in code of one
    assert whole >= 10 and one >= 20
