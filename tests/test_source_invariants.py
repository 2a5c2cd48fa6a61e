"""Properties of the source tree that the design relies on, checked by reading the files."""
import pathlib
import re

ROOT = pathlib.Path(__file__).resolve().parent.parent
KERNELS = sorted((ROOT / "csrc" / "kernels").rglob("*.cu")) + sorted((ROOT / "csrc" / "kernels").rglob("*.cuh"))


def _code_lines(path):
    """(line number, text) without // comments (good enough for these checks: no block comments in the kernels)."""
    for i, line in enumerate(path.read_text().splitlines(), 1):
        yield i, line.split("//", 1)[0]


def test_no_load_uses_cluster_multicast():
    """Operand tiles are fetched by each CTA itself; the qualifier may only appear on tcgen05.commit."""
    needle = "multicast" + "::cluster"
    bad = [(p.name, i) for p in KERNELS for i, line in _code_lines(p) if needle in line and "tcgen05.commit" not in line]
    assert not bad, bad


def test_kernels_never_trap_or_assert():
    """Problems are reported through the status page and the kernel returns; nothing traps the GPU."""
    pat = re.compile(r"__trap\s*\(|(?<![_a-zA-Z])assert\s*\(")
    bad = [(p.name, i) for p in KERNELS for i, line in _code_lines(p) if pat.search(line)]
    assert not bad, bad


def test_tensor_core_path_is_tcgen05_only():
    text = "\n".join(line for p in KERNELS for _, line in _code_lines(p))
    assert "tcgen05.mma" in text and "cp.async.bulk.tensor" in text
    for legacy in ("wgmma", "mma.sync", "wmma::"):
        assert legacy not in text, legacy


def test_every_device_wait_goes_through_the_bounded_helpers():
    """Acquire loads in a loop live in ptx.cuh (wait_flag_ge, mbar_wait) or sit next to a globaltimer limit."""
    for p in KERNELS:
        lines = list(_code_lines(p))
        for idx, (i, line) in enumerate(lines):
            if re.search(r"while\s*\(", line) and "ld_acquire" in line:
                window = " ".join(t for _, t in lines[idx: idx + 8])
                assert "globaltimer_ns" in window or "limit" in window, f"{p.name}:{i}: unbounded wait"


def test_cluster_barriers_are_reached_by_whole_warps():
    """barrier.cluster is used in its aligned form, which a split warp must not execute: the statement in front of every one
    brings the warp (or the block) together."""
    bad = []
    for p in KERNELS:
        prev = ""
        for i, line in _code_lines(p):
            if re.search(r"(?<!void )\bcluster_sync_all\(\)", line) and not re.search(r"__sync(threads|warp)\(\);\s*$", prev):
                bad.append((p.name, i))
            if line.strip():
                prev = line.rstrip()
    assert not bad, bad


def test_kernels_that_load_in_bulk_let_their_copies_land():
    """A CTA that leaves after a wait ran out must not hand its shared memory on while copies into it are under way: every
    kernel that starts such copies has the bounded pause of settle_copies() on that path."""
    loads = re.compile(r"\b(bulk_load_g2s|tma_load_2d\w*|ag_push_bulk\w*)\(")
    bad = []
    for p in KERNELS:
        text = "\n".join(line for _, line in _code_lines(p))
        for body in text.split("__global__")[1:]:
            if loads.search(body) and "settle_copies()" not in body:
                bad.append((p.name, body.split("(", 3)[0].split()[-1], body[:80]))
    assert not bad, bad


def test_waits_of_whole_warps_end_alike_in_all_lanes():
    """The roles that read accumulators or take tile numbers run as whole warps. Their bounded waits (places 4 and 6 of the status
    page, and 11 in the fp8 product) may run out in one lane only, so the lanes vote, or the threads pass the word on before a
    named barrier."""
    bad = []
    for p in KERNELS:
        lines = [line for _, line in _code_lines(p)]
        for i, line in enumerate(lines):
            places = "4|6|11" if p.name == "gemm_fp8.cuh" else "4|6"
            if re.search(rf"(mbar_wait\w*|wait_flag_ge)\(.*\bst, ({places}),", line):
                voted = "__all_sync" in line or re.search(r"mbar_wait\w*_warp\(", line)
                # or the lane goes on without leaving the loop, and the vote comes at its end
                kept = "part_phase |= 1u << 31;" in line and any("ok = __all_sync(0xffffffffu, static_cast<int>(part_phase) >= 0);" in t for t in lines[i: i + 30])
                if not voted and not kept and not any("epi_fail" in t for t in lines[i: i + 8]):
                    bad.append((p.name, i + 1))
    assert not bad, bad


def test_split_products_store_nothing_after_a_wait_that_ran_out():
    """The kernels that split a product along K over a cluster store through one function, which asks every CTA of the cluster
    whether it gave up before it adds or stores anything."""
    common = ROOT / "csrc" / "kernels" / "common"
    text = {p.name: "\n".join(line for _, line in _code_lines(p)) for p in common.glob("*.cuh")}
    body = text["cluster_sum.cuh"].split("void cluster_add_store", 1)[1]
    order = [body.index(s) for s in ("cluster_sync_all()", "ld_cluster_u32", "__any_sync", "return;", "ld_cluster_f32x4", "<uint2*>(C")]
    assert order == sorted(order)
    for name in ("gemm_ks.cuh", "gemm_fp8_pair.cuh"):
        kernel = text[name].split("ksplit_kernel", 1)[1]
        assert "cluster_add_store(sums, fail_slot" in kernel and "ld_cluster_f32x4" not in kernel, name


def test_chained_kernels_promise_nothing_about_their_inputs():
    """A kernel that waits for its predecessor inside (griddep_wait) runs while that one still writes: none of its pointers may be
    declared __restrict__, which says that the data does not change during the kernel's life."""
    seen, bad = 0, []
    for p in KERNELS:
        text = "\n".join(line for _, line in _code_lines(p))
        for kernel in text.split("__global__")[1:]:
            signature, body = kernel.split("\n{", 1)
            if "griddep_wait()" in body:
                seen += 1
                if "__restrict__" in signature:
                    bad.append((p.name, signature[:120]))
    assert seen >= 6 and not bad, (seen, bad)


def test_function_attributes_are_remembered_per_device():
    """A function attribute belongs to one device's copy of the kernel, and a process may drive several devices: what remembers
    that it has been set is an array over devices, never one word for the process."""
    bad = [(p.name, i) for p in KERNELS for i, line in _code_lines(p) if re.search(r"static\s+bool\s+\w+\s*(=|;|\{)", line)]
    assert not bad, bad


def test_c_api_header_and_library_agree():
    """Every function declared in the public C headers is exported by the built kernel library."""
    from dlslime_b200 import _lib

    if not _lib.available():
        import pytest

        pytest.skip("kernel library not built")
    lib = _lib.load()
    names = set()
    for h in ("slime_cuda.h", "slime_noalloc.h"):
        text = (ROOT / "csrc" / "include" / h).read_text()
        text = re.sub(r"//[^\n]*", "", text)
        names.update(re.findall(r"\b(slime_[a-z0-9_]+)\s*\(", text))
    assert len(names) > 40
    missing = [n for n in sorted(names) if not hasattr(lib, n)]
    assert not missing, missing


def test_baseline_arms_import_nothing_of_the_package():
    """The reference arm and the tuned arm of bench.py must not load this repository's package or libraries: their
    modules import only the standard library, torch and each other, and bench.py imports the package inside run_ours
    only."""
    import ast

    for name in ("reference_arm.py", "tuned_arm.py", "torch_moe.py"):
        tree = ast.parse((ROOT / "baseline" / name).read_text())
        for node in ast.walk(tree):
            mods = []
            if isinstance(node, ast.Import):
                mods = [a.name for a in node.names]
            elif isinstance(node, ast.ImportFrom):
                mods = [node.module or ""]
            assert not any(m.split(".")[0] == "dlslime_b200" for m in mods), (name, mods)
    tree = ast.parse((ROOT / "bench.py").read_text())
    for fn in [n for n in tree.body if isinstance(n, (ast.FunctionDef, ast.ClassDef))]:
        uses = [n for n in ast.walk(fn) if isinstance(n, ast.ImportFrom) and (n.module or "").startswith("dlslime_b200")]
        assert not uses or fn.name == "run_ours", fn.name
    top = [n for n in tree.body if isinstance(n, (ast.Import, ast.ImportFrom))]
    assert not any("dlslime_b200" in ast.dump(n) for n in top)
