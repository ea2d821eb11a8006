"""Kernels that start while the kernel ahead still runs (programmatic dependents), held to what makes that sound, by reading the
sources: every block waits, nothing returns before the wait, and data of earlier launches is read by ordinary loads or TMA.  A
load of the non-coherent path (__ldg, or a const __restrict__ pointer, which the compiler may read that way) can hit a line that
an earlier kernel left in L1; only weights, which no kernel of a model writes, may be read like that."""
import glob
import os
import re
import subprocess

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "baranet_bdml_b200", "csrc")
WAIT = re.compile(r"grid_dependency_wait\(\)|griddepcontrol\.wait")

# what __ldg may read in a dependent: weights, biases, and the table of gemm_bf16_nt_kernel<EPI_QKV>, an ordinary launch
WEIGHTS = {
    "gemm_bf16_sm100.cu": {"p.bias + n0 + c", "cs + i"},
    "gemm_skinny.cu": {"p.bias + n"},
    "latent_decode.cu": {"reinterpret_cast<const uint4*>(w + (int64_t)k * p.kv_ld + c)", "reinterpret_cast<const uint4*>(w + (s + i) * 32)"},
    "mamba2.cu": {"p.conv_b + c", "reinterpret_cast<const float4*>(p.conv_w) + c", "p.conv_w + (int64_t)c * taps + taps - 1 - k"},
    "rmsnorm.cu": {"reinterpret_cast<const uint4*>(p.w) + c"},
}


def closing(text, at, pair):
    """index behind the bracket that closes the one at `at`"""
    depth = 0
    for i in range(at, len(text)):
        depth += (text[i] == pair[0]) - (text[i] == pair[1])
        if depth == 0:
            return i + 1
    raise AssertionError("unbalanced")


def kernels(text):
    """(name, parameters, body, start, end) of every __global__ function"""
    for m in re.finditer(r"__global__", text):
        at = re.compile(r"(\w+)\(").search(text, m.end())
        while at.group(1) in ("__launch_bounds__", "__maxnreg__"):
            at = re.compile(r"(\w+)\(").search(text, closing(text, at.end() - 1, "()"))
        params_end = closing(text, at.end() - 1, "()")
        body = text.index("{", params_end)
        end = closing(text, body, "{}")
        yield at.group(1), text[at.end():params_end - 1], text[body:end], m.start(), end


def sources():
    for path in sorted(glob.glob(os.path.join(CSRC, "*.cu"))):
        text = re.sub(r"//[^\n]*", "", open(path).read())
        yield os.path.basename(path), text, list(kernels(text))


def test_every_dependent_waits_first():
    seen = set()
    for name, text, found in sources():
        waiting = {k for k, _, body, _, _ in found if WAIT.search(body)}
        launched = {m for call in re.findall(r"launch_dependent\(([^;]*?)[,;]", text) for m in re.findall(r"\b(\w+_kernel)\b", call)}
        launched |= set(re.findall(r"cudaLaunchKernelEx\(&\w+, (\w+_kernel)", text))
        assert launched <= waiting, (name, launched - waiting)
        seen |= waiting
        for k, _, body, _, _ in found:
            m = WAIT.search(body)
            assert not m or not re.search(r"\breturn\b\s*;", body[:m.start()]), (name, k)
    assert len(seen) > 20


def test_dependents_read_what_others_wrote_by_ordinary_loads():
    for name, text, found in sources():
        # helpers belong to whoever calls them: only the bodies of ordinary kernels are left out
        rest, dependents = text, False
        for k, params, body, start, end in reversed(found):
            if not WAIT.search(body):
                rest = rest[:start] + rest[end:]
                continue
            dependents = True
            assert not re.search(r"const\s+\w+\*\s*__restrict__", params), (name, k)
        if dependents:
            reads = [rest[m.end():closing(rest, m.end() - 1, "()") - 1] for m in re.finditer(r"__ldg\(", rest)]
            assert set(reads) <= WEIGHTS.get(name, set()), (name, set(reads) - WEIGHTS.get(name, set()))


FAKE = r"""
#include <stdio.h>
#include "launch.cuh"
// The runtime's two calls, which refuse a programmatic dependence while `refuse` is set, and any launch without the cluster's size
// while `cluster` is
static int refuse, cluster, calls, kept;
static cudaError_t pending;
extern "C" cudaError_t cudaLaunchKernelExC(const cudaLaunchConfig_t* cfg, const void*, void** args) {
    bool dependent = false, size = false;
    for (unsigned i = 0; i < cfg->numAttrs; ++i) {
        dependent |= cfg->attrs[i].id == cudaLaunchAttributeProgrammaticStreamSerialization;
        size |= cfg->attrs[i].id == cudaLaunchAttributeClusterDimension;
    }
    ++calls;
    if ((refuse && dependent) || (cluster && !size) || *(int*)args[0] != 7) return pending = cudaErrorNotSupported;
    kept = cfg->numAttrs;
    return cudaSuccess;
}
extern "C" cudaError_t cudaGetLastError() { cudaError_t e = pending; pending = cudaSuccess; return e; }
static void kernel(int) {}
int main() {
    for (refuse = 0; refuse < 2; ++refuse) {
        calls = 0;
        bn::launch_dependent(kernel, dim3(3), 32, 0, (cudaStream_t)0, 7);
        if (calls != 1 + refuse || kept != 1 - refuse || cudaGetLastError() != cudaSuccess) return 1;
        cudaLaunchAttribute attr[2];
        attr[0].id = cudaLaunchAttributeClusterDimension;
        attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        cudaLaunchConfig_t cfg = {};
        cfg.attrs = attr;
        cfg.numAttrs = 2;
        calls = 0, cluster = 1;
        if (bn::launch_config(cfg, 1, kernel, 7) != cudaSuccess || calls != 1 + refuse || kept != 2 - refuse) return 2;
        cluster = 0;
        // what is refused for another reason stays refused, and says so
        if (bn::launch_config(cfg, 1, kernel, 8) == cudaSuccess || cudaGetLastError() == cudaSuccess) return 3;
    }
    return 0;
}
"""


def test_a_refused_attribute_costs_the_overlap_alone(tmp_path):
    """Against a fake runtime; and every launch with attributes goes that way, or has the fallback beside it."""
    src, exe = tmp_path / "launch.cpp", tmp_path / "launch"
    src.write_text(FAKE)
    cuda = os.environ.get("CUDA_HOME", "/usr/local/cuda")
    subprocess.run(["/usr/bin/g++", "-std=c++17", "-w", "-I" + CSRC, "-I" + os.path.join(cuda, "include"), str(src), "-o", str(exe)], check=True)
    assert subprocess.run([str(exe)]).returncode == 0
    for name, text, found in sources():
        waiting = {k for k, _, body, _, _ in found if WAIT.search(body)}
        assert set(re.findall(r"launch_config\(\w+, [^,]*, (\w+_kernel)", text)) <= waiting, name
        for m in re.finditer(r"cudaLaunchKernelEx\(&\w+, (\w+)", text):
            assert m.group(1) + "<<<" in text[m.end():m.end() + 200], name


def test_a_kernel_has_one_limit_of_shared_memory():
    """The limit that a kernel may ask for belongs to it in all threads: what sets it, outside allow_smem, is a constant of the kernel."""
    asked = 0
    for name, text, _ in sources():
        for m in re.finditer(r"cudaFuncSetAttribute\(", text):
            args = text[m.end():closing(text, m.end() - 1, "()") - 1]
            if "," not in args:                     # (the name in a message)
                continue
            assert re.search(r"(SMEM_\w+|\w+_SMEM|96 \* 1024)$", args.rsplit(",", 1)[1].strip()), (name, args)
            asked += 1
    assert asked > 5
