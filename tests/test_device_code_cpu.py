"""Rules of the device code that no run can show to hold (a break of one may
give right results for years), read off the sources."""
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "openmp-blas_gb300", "csrc")


def sources():
    """{file name: its text without comments}"""
    out = {}
    for f in sorted(os.listdir(CSRC)):
        if f.endswith((".cu", ".cuh")):
            out[f] = re.sub(r"//[^\n]*", "", open(os.path.join(CSRC, f)).read())
    return out


def block(text, start):
    """The {...} that opens at or after `start`."""
    i = text.index("{", start)
    depth = 0
    for j in range(i, len(text)):
        depth += {"{": 1, "}": -1}.get(text[j], 0)
        if depth == 0:
            return text[i:j + 1]
    raise ValueError("unbalanced braces")


def test_aligned_cluster_barriers_follow_a_warp_barrier():
    """barrier.cluster.*.aligned is undefined for a diverged warp: each function
    that issues one brings the warp together first."""
    found = 0
    for name, text in sources().items():
        for m in re.finditer(r"barrier\.cluster\.arrive[a-z.]*\.aligned", text):
            body = text[text.rindex("__device__", 0, m.start()):m.start()]
            assert "__syncwarp();" in body, f"{name}: {body}"
            found += 1
    assert found == 2


def kernels(text):
    """(name, parameters, body) of each __global__ function."""
    for m in re.finditer(r"__global__\s+void\s+(?:__launch_bounds__\([^)]*(?:\([^)]*\)[^)]*)*\)\s*)?(\w+)\s*\(", text):
        depth, i = 1, m.end()
        while depth:
            depth += {"(": 1, ")": -1}.get(text[i], 0)
            i += 1
        yield m.group(1), text[m.end():i - 1], block(text, i)


def test_chained_kernels_take_the_chains_results_by_plain_loads():
    """A kernel launched behind the one before it (grid_wait) is resident while
    that one writes: what it reads of it must not be promised constant for the
    kernel's lifetime (const __restrict__, __ldg, ld_stream), or the loads may
    be served from the read-only path or moved ahead of the wait.  The caller's
    operands, reached through a job's or an operand's `src`, may be."""
    found = []
    for name, text in sources().items():
        assert not re.search(r"\b(TcProblem|SplitJob|SplitReduce)\s*\*\s*__restrict__", text), name
        for kernel, params, body in kernels(text):
            if "grid_wait()" not in body:
                continue
            found.append(kernel)
            assert not re.search(r"const\s+[\w:]+\s*\*\s*__restrict__", params), f"{kernel}({params})"
            operands = {"j.src", "src"}
            for local, value in re.findall(r"const\s+[\w:]+\s*\*\s*__restrict__\s+(\w+)\s*=\s*([\w.]+)", body):
                assert value in ("j.src", "o.src"), f"{kernel}: {local} = {value}"
                operands.add(local)
            for local, value in re.findall(r"const\s+(?:float|double)\s*\*\s*(\w+)\s*=\s*([\w.]+)", body):
                if value in operands:
                    operands.add(local)
            for arg in re.findall(r"(?:__ldg|ld_stream)\(\s*(?:reinterpret_cast<[^>]*>\(\s*)?\(?\s*([\w.]+)", body):
                assert arg in operands, f"{kernel}: read-only load of {arg}"
    assert len(found) >= 12 and {"gemm_split_kernel", "dgemm_digits_kernel", "finish_splits_kernel"} <= set(found)


def test_digit_gemm_looks_at_the_abort_flag_behind_a_barrier():
    """A role that gives up after the others have finished must still find its
    copies and MMAs waited for before the CTA leaves: the teardown reads the
    flag after a barrier of the whole CTA."""
    body = dict((k, b) for k, _, b in kernels(sources()["gemm_f64_tc.cu"]))["dgemm_digits_kernel"]
    checks = [m.start() for m in re.finditer(r"if \([^)]*lane == 0 && \*abort_flag\)", body)]
    assert len(checks) == 1
    stores = body.rindex("crow[")  # the epilogue's last store into C
    assert stores < body.index("__syncthreads();", stores) < checks[0]
