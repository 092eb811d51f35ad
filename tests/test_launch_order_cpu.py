"""Order of waits in the kernels, read from the sources: those that start while the kernel ahead drains, and clusters.

The GEMVs stream their weights before they wait for the kernel ahead, so a weight must be complete by the time
the kernel ahead of the GEMV lets it in.  A kernel that lets its dependents in only behind its own wait vouches
for everything before itself; one that does so earlier lets them reach further back."""
import glob
import os
import re

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
TRIGGER, WAIT = "griddepcontrol.launch_dependents", "griddepcontrol.wait"

# Let their dependents in ahead of their own wait.  The two GEMVs do it from the producer warp.  The two reductions only
# ever follow their own split kernel, which lets them in behind ITS wait and writes nothing but their partials.
EARLY = {"nvfp4_gemv_mma_kernel", "nvfp4_matvec_kernel", "attention_splitk_reduce_kernel", "attention_few_splits_reduce_kernel"}


def kernels():
    """name -> body of every __global__ function under csrc (bodies end at a closing brace in the first column)."""
    found = {}
    for path in sorted(glob.glob(os.path.join(ROOT, "speedoza_b200", "csrc", "*.cu"))):
        text = re.sub(r"//[^\n]*", "", open(path).read())
        for m in re.finditer(r"__global__\s+void\s+(?:__launch_bounds__\([^\n]*\)\s+)?(\w+)\s*\(", text):
            found[m.group(1)] = text[m.end():text.index("\n}", m.end())]
    return found


def test_dependents_are_let_in_behind_the_wait():
    bodies = kernels()
    assert {"nvfp4_gemm_tc_kernel", "nvfp4_gemm_splitk_kernel", "nvfp4_gemm_pair6_kernel"} <= set(bodies) and EARLY <= set(bodies)
    early = {name for name, body in bodies.items()
             if TRIGGER in body and WAIT in body and body.index(TRIGGER) < body.index(WAIT)}
    assert early == EARLY


def test_writers_of_weight_format_are_complete_first():
    """Row quantisers let the next kernel in early only for fewer rows than a GEMV that starts early takes."""
    bodies = kernels()
    for name in ("nvfp4_quantize_kernel", "nvfp4_quantize_fast_kernel", "swiglu_nvfp4_quantize_rows_kernel"):
        lines = [line.strip() for line in bodies[name].splitlines() if TRIGGER in line]
        assert all(line.startswith("if (rows < q36::kWeightRows)") for line in lines), name
    launch = open(os.path.join(ROOT, "speedoza_b200", "csrc", "nvfp4_matvec.cu")).read()
    assert "cfg.numAttrs = N < q36::kWeightRows ? 0 : 1;" in launch


def test_remote_shared_memory_only_once_the_cluster_runs():
    """Stores into another CTA's shared memory come behind a cluster barrier: all CTAs of the cluster have started."""
    remote = re.compile(r"map_to_cta\(|cluster_rank_address\(|mapa\.shared|map_shared_rank\(")
    barrier = re.compile(r"cluster_sync_all\(|barrier\.cluster\.wait")
    found = {}
    for name, body in kernels().items():
        if remote.search(body):
            first = barrier.search(body)
            found[name] = first is not None and first.start() < remote.search(body).start()
    assert len(found) >= 6 and all(found.values()), found


def test_every_bounded_wait_of_the_w4a4_products_is_recorded():
    """A wait of nvfp4_gemm_tc.cu that gives up sets the error that qwen36_nvfp4_gemm_last_error returns: a loop that
    counts up to kSpinLimit stands only in a function that sets it once the loop has run out."""
    text = re.sub(r"//[^\n]*", "", open(os.path.join(ROOT, "speedoza_b200", "csrc", "nvfp4_gemm_tc.cu")).read())
    starts = [m.start() for m in re.finditer(r"\bfor \([^;{}]*;[^;{}]*kSpinLimit[^;{}]*;", text)]
    assert starts and len(starts) == text.count("kSpinLimit") - 1       # the other one is the constant
    for at in starts:
        rest = text[at:text.index("\n}", at)]
        assert "atomicExch(&g_gemm_error, 1u);" in rest and rest.rstrip().endswith("return false;"), text[at:at + 120]
