"""What the host code enqueues, on a recording stand-in for the CUDA runtime (tests/fake_cuda): streams,
order, launch attributes and graphs of the API's calls, without a GPU."""
import os
import shutil
import subprocess

import pytest

from conftest import ROOT

CSRC = os.path.join(ROOT, "gpuowl_b200", "csrc")
FAKE = os.path.join(ROOT, "tests", "fake_cuda")
NVCC = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"


@pytest.fixture(scope="module")
def host_log(tmp_path_factory):
    if not os.path.exists(NVCC):
        pytest.skip("no nvcc")
    d = tmp_path_factory.mktemp("host_log")
    src = d / "csrc"
    shutil.copytree(CSRC, src)
    for body in ("owl_pass1_body.inc", "owl_pass2_body.inc"):  # the kernels do not run: 20 s instead of minutes
        (src / body).write_text("")
    exe = str(d / "host_log")
    subprocess.run([NVCC, "-gencode", "arch=compute_100a,code=sm_100a", "-std=c++17", "-w", "-cudart", "none",
                    "--expt-relaxed-constexpr", "-I", str(src), "-I", os.path.join(ROOT, "include"), "-o", exe,
                    os.path.join(FAKE, "host_log.cu"), os.path.join(FAKE, "fake_cuda.cpp")],
                   check=True, capture_output=True)

    def run(*args):
        r = subprocess.run([exe] + [str(a) for a in args], capture_output=True, text=True, timeout=120)
        assert r.returncode == 0, (r.stdout[-2000:], r.stderr[-2000:])
        sections, name = {}, ""
        for line in r.stdout.splitlines():
            if line.startswith("== "):
                name = line[3:]
                while name in sections:
                    name += "'"
                sections[name] = []
            else:
                sections.setdefault(name, []).append(line)
        return sections
    return run


def test_a_new_plan_is_ready(host_log):
    """Tables and cleared scratch are there when the call returns: the plan's stream does not wait for the
    default stream, on which an upload or a memset may still be under way."""
    ops = host_log("create")["create"]
    assert [x for x in ops if x.startswith("stream ")] == ["stream 1 non-blocking"]
    moves = [i for i, x in enumerate(ops) if x.startswith(("memset", "copy"))]
    assert len(moves) >= 2 and all(ops[i] in ("memset stream=1", "copy stream=1") for i in moves), ops
    assert "wait stream=1" in ops[moves[-1]:], ops


def test_reset_after_a_timeout_is_ordered(host_log):
    """The control word and the carry words of a plan whose wait ran out are cleared on its own stream, and
    the call returns once they are (a launch between the two would take old carry words for new ones)."""
    ops = host_log("reset")["sync"]
    assert ops[-1] == "status -4"
    sets = [i for i, x in enumerate(ops) if x.startswith("memset")]
    assert len(sets) >= 2 and all(ops[i] == "memset stream=1" for i in sets), ops
    assert "wait stream=1" in ops[sets[-1]:], ops


@pytest.mark.parametrize("W,H,split", [(64, 64, 0), (2048, 64, 0), (64, 2560, 0), (64, 2048, 1), (64, 2560, 1)])
def test_a_kept_spectrum_is_complete_before_the_pass_that_reads_it_starts(host_log, W, H, split):
    """The product pass declares the kept spectrum read-only while it runs, so it must not be a programmatic
    dependent of the pass that writes it."""
    log = host_log("power", W, H, split)
    for name, muls in (("power", 5), ("product", 1), ("product'", 1)):  # 0xb5 has four bits below its top
        k = [x for x in log[name] if x.startswith("launch k_pass")]
        mode = [int(x.split("<")[1].split(">")[0].split(",")[2]) for x in k]
        at = [i for i, x in enumerate(k) if x.startswith("launch k_pass2") and mode[i] == 2]
        assert len(at) == muls, k
        for i in at:
            after_writer = k[i - 1].startswith("launch k_pass2") and mode[i - 1] == 1
            assert not (after_writer and "pdl=1" in k[i]), k[i - 1:i + 1]


def test_cached_graphs_follow_the_wait_limit(host_log):
    """A block, a profiled block, a product and a batch that run as cached graphs wait as long as the last
    set limit says, and a limit that comes back finds its graphs again."""
    log = host_log("timeouts")
    graphs = []
    for name, batch, limit in (("limit 7", "batch", 7), ("limit 9", "batch'", 9), ("limit 7'", "batch''", 7)):
        k = [x for x in log[name] if x.startswith("launch k_pass")]
        assert len(k) > 70 and all(" timeout=%d " % limit in x + " " for x in k), (name, k[:2])
        kb = [x for x in log[batch] if x.startswith("launch k_pass")]
        assert {x.split("timeout=")[1].split()[0] for x in kb} == {"%d,2000000000" % limit, str(limit + 1)}, kb[:2]
        graphs.append([x for x in log[name] + log[batch] if x.startswith("graph ")])
    assert graphs[0] != graphs[1]
    # a product becomes a graph on the second call with its buffers, so limit 7 ran one on its first call here
    assert set(graphs[0]) <= set(graphs[2])


def test_batch_graph_follows_the_plans_settings(host_log):
    """A batch that was captured before a plan's split form or column variant changed is captured again."""
    log = host_log("settings")
    runs = [[x.split()[1] for x in log[s] if x.startswith("launch k_pass2")] for s in ("plain", "split", "variant")]
    assert not any("k_pass2_tc" in x for x in runs[0])
    assert any("k_pass2_tc" in x for x in runs[1])
    assert any(x.startswith("k_pass2") and ",8," in x for x in runs[2])


@pytest.mark.parametrize("W,H,line_few,column_few", [
    (256, 64, False, False), (512, 64, True, False), (512, 128, True, False), (512, 256, False, False),
    (1024, 64, True, False), (1024, 128, False, False), (64, 1024, False, True), (128, 1024, False, True),
    (256, 1024, False, False), (2048, 64, False, False)])
def test_passes_of_few_threads_run_the_unbounded_builds(host_log, W, H, line_few, column_few):
    """Line passes of 64 and 128 threads and 1024-point columns are bounded to 128 registers, but for the fused
    line pass without the round-off measurement below 8,192 threads and columns below 16,384."""
    log = host_log("power", W, H, 0)
    few = set()
    for section in ("square", "square without round-off", "power", "product"):
        k = [x.split()[1].rstrip(">") for x in log[section] if x.startswith("launch k_pass")]
        lines = {x for x in k if x.startswith("k_pass1<")}
        columns = {x for x in k if x.startswith("k_pass2<")}
        assert lines and columns
        few |= {x.split("<")[1].split(",", 2)[2] for x in lines if x.endswith(",true") and x.count(",") == 5}
        assert {x.split(",")[4] == "1" for x in columns} == {column_few}, columns
    assert few == ({"0,false,false,true"} if line_few else set())
