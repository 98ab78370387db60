"""A kernel that waits for the one in front (``pdl_wait``) is resident while that one still writes, so what it reads has to
come through coherent loads that stay behind the wait.  Read from the sources: the order of loads cannot be seen in results."""
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "flashrt_b200", "csrc")


def source(name):
    text = open(os.path.join(CSRC, name)).read()
    return re.sub(r"//[^\n]*|/\*.*?\*/", "", text, flags=re.S)


WAITING = sorted(f for f in os.listdir(CSRC) if f.endswith((".cu", ".cuh")) and "pdl_wait()" in source(f))


@pytest.mark.parametrize("name", WAITING)
def test_kernels_that_wait_read_coherently(name):
    text = source(name)
    for word in ("ld.global.nc", "__ldg(", "__ldlu(", "ld_global_nc"):
        assert word not in text, f"{name}: {word}"
    text = re.sub(r"__launch_bounds__\s*\((?:[^()]|\([^()]*\))*\)", "", text)
    kernels = re.findall(r"__global__\s+void\s+(\w+)\s*\(([^{;]*)\)\s*\{", text)
    assert len(kernels) == text.count("__global__")
    for kernel, params in kernels:
        for p in params.split(","):
            assert not ("const" in p and "*" in p and "__restrict__" in p), f"{name}: {kernel}: {' '.join(p.split())}"


def test_split_k_counters_end_at_zero_when_a_wait_gives_up():
    """The counters of the split-K product belong to the caller, who zeroes them once.  Every unit of a launch has to arrive
    exactly once with an operation that wraps at S, on the path of a warp whose wait gave up as well: a count left between
    0 and S would make the first arrival of the next launch take itself for the last and add a stale partial."""
    text = source("gemm_pair.cuh")
    uses = re.findall(r"[^\n]*split_cnt[^\n]*", text)
    assert len(uses) == 1 and re.search(r"atomicInc\(p\.split_cnt \+ .*, \(unsigned\)\(S - 1\)\)", uses[0]), uses
    gave_up = re.search(r"ERR_EPILOGUE(.*?)break;", text, flags=re.S).group(1)
    assert re.search(r"if constexpr \(SPLIT\)\s+for \(; t < total; t \+= npairs\)\s+if \(lane == 0\) split_k_arrive\(p, t, S, ",
                     gave_up), gave_up
    assert text.count("split_k_arrive(") == 3          # the definition, the sum, the path that gave up


@pytest.mark.parametrize("name", ["attention.cu", "attention_d256.cuh"])
def test_attention_counters_count_every_cta(name):
    """A tile's arrival counter stands at a multiple of 256 behind every launch: each CTA arrives, whether its waits returned
    or gave up."""
    text = re.sub(r"\s*ATT_STAMP\(\d+\);", "", source(name))
    found = re.findall(r"__threadfence\(\);\s*__syncthreads\(\);\s*if \(threadIdx\.x == 0\) \{\s*asm volatile\(\"red\.relaxed\.gpu", text)
    assert len(found) == text.count("red.relaxed.gpu") == 1


def test_lanes_that_skip_stores_meet_before_the_next_collective_load():
    """tcgen05.ld is executed by a whole warp: the loop around one whose lanes may take a ``continue`` starts with a warp
    barrier."""
    text = source("gemm_persistent.cuh")
    head = text[:text.index("if (m >= p.M) continue;")]
    head = head[head.rindex("for (int c"):]
    assert 0 < head.find("__syncwarp();") < head.index("tmem_ld") and text.count("continue;") == 1


def test_shared_memory_limit_of_a_kernel_does_not_follow_the_launch():
    """A kernel's limit of dynamic shared memory is one value per kernel: a size raised from launch to launch is set back when
    another thread's smaller launch sets its own between the check and the call."""
    values = []
    for name in sorted(f for f in os.listdir(CSRC) if f.endswith((".cu", ".cuh"))):
        values += re.findall(r"cudaFuncAttributeMaxDynamicSharedMemorySize,\s*([^;]*)\);", source(name))
    assert len(values) > 10
    for v in values:                   # no name of a variable: constants and what they make up
        words = set(re.findall(r"[A-Za-z_]\w*", v)) - {"int", "sizeof", "float", "el", "Cfg", "smem_bytes", "ragged_smem_bytes", "true"}
        assert all(w.isupper() for w in words), v


def _block(text, at):
    """The braces that open behind `at`, with what is between them."""
    start = i = text.index("{", at)
    depth = 0
    while True:
        depth += {"{": 1, "}": -1}.get(text[i], 0)
        i += 1
        if depth == 0:
            return text[start:i]


LANE_CONDITION = re.compile(r"if \((?:row (?:<|>=) (?:Mt|rows_valid)|m (?:<|>=) p\.M|n < p\.N|store|!lines && m < p\.M)\b")


@pytest.mark.parametrize("name", sorted(f for f in os.listdir(CSRC) if f.endswith((".cu", ".cuh")) and f != "tc05.cuh" and "tmem_ld32(" in source(f)))
def test_lanes_with_stores_of_their_own_meet_before_the_next_collective_load(name):
    """tcgen05.ld is an aligned instruction.  A block that loads and then lets some lanes store and others not, and comes round to
    the load again (a loop, or a function called in one), has a warp barrier in front of the load."""
    text = source(name)
    heads = [m.start() for m in re.finditer(r"for \(int c\w* = ", text)]
    heads += [m.start() for m in re.finditer(r"void epilogue_(?:geglu|rope)_rows\(", text)]
    for at in heads:
        body = _block(text, at)
        load = body.find("tmem_ld")
        if load < 0 or not LANE_CONDITION.search(body, load) or "for (int c" in body[:load]:
            continue
        assert "__syncwarp();" in body[:load], body[:400]
    for m in re.finditer(r"auto emit = \[&\]", text):      # stores of some lanes between two loads
        assert re.search(r"__syncwarp\(\);\s*\}$", _block(text, m.start())), name


def test_aligned_cluster_barriers_stand_behind_a_warp_or_block_barrier():
    """barrier.cluster's aligned forms want the warp together: __syncwarp or __syncthreads comes last in front of each, with no
    branch between."""
    for name in sorted(f for f in os.listdir(CSRC) if f.endswith((".cu", ".cuh"))):
        text = source(name)
        for helper in ("cluster_arrive_release", "cluster_wait_acquire"):      # their callers are looked at instead
            text = re.sub(r"void %s\(\) \{[^}]*\}" % helper, "", text)
        for m in re.finditer(r"barrier\.cluster\.(?:arrive|wait)[.\w]*aligned|cluster_(?:arrive_release|wait_acquire)\(\);", text):
            front = text[:m.start()]
            at = max(front.rfind("__syncwarp();"), front.rfind("__syncthreads();"))
            between = re.sub(r"if (?:constexpr )?\((?:XC|!XC|EPI == [^()]*)\)", "", front[at:])     # compile-time conditions
            assert at >= 0 and not re.search(r"\b(?:if|for|while)\b", between), (name, between)
