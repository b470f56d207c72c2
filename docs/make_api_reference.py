"""Regenerate docs/api.md from the package's docstrings:  python docs/make_api_reference.py"""

import importlib
import inspect
import os
import sys

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
sys.path.insert(0, ROOT)

MODULES = [
    ("bitscom_b200", ["init", "register_lowbit_backend", "is_extension_available", "LowBitGroup",
                      "SUPPORTED_BITWIDTHS", "shutdown"]),
    ("bitscom_b200.quantization", None),
    ("bitscom_b200.parallel.fused", ["FusedLowBitComm", "EmulatedWorld", "FusedCollectiveError",
                                     "FusedUnavailable", "traffic_bytes"]),
    ("bitscom_b200.parallel.hooks", None),
    ("bitscom_b200.parallel.zero", None),
    ("bitscom_b200.parallel.flat", None),
    ("bitscom_b200.parallel.pp_schedule", None),
    ("bitscom_b200.parallel.deferred", None),
    ("bitscom_b200.parallel.simulate", None),
    ("bitscom_b200.data", None),
    ("bitscom_b200.ops.gemm", ["gemm", "linear", "LinearFunction", "check_status", "variant",
                               "set_variant", "use_library_gemm"]),
    ("bitscom_b200.ops.attention", ["attention", "supported", "set_forward_variant",
                                    "set_backward_dq_variant", "check_status"]),
    ("bitscom_b200.ops.nn", ["rmsnorm", "rmsnorm_fork", "layernorm", "bias_gelu", "swiglu", "rope_qk_",
                             "rope_tables", "cross_entropy", "embedding", "FlatAdamW", "FlatSGD"]),
    ("bitscom_b200.utils.checkpoint", None),
    ("bitscom_b200.utils.graphs", None),
    ("bitscom_b200.utils.health", None),
    ("bitscom_b200.launch", ["run", "agent_store", "Generation"]),
    ("bitscom_b200.utils.timing", None),
    ("bitscom_b200.utils.clocks", None),
    ("bitscom_b200.utils.plot", ["save_line_plot"]),
    ("bitscom_b200.bench.allreduce_block", None),
]


ENVIRONMENT = [
    "## Environment variables", "",
    "| variable | effect |", "|---|---|",
    "| `BITSCOM_GEMM` | `auto` (default, by shape), `1cta` or `2cta`: the kernel `ops.gemm.gemm` launches |",
    "| `BITSCOM_ATTN_FWD`, `BITSCOM_ATTN_BWD_DQ` | attention kernel variants (`simple` / "
    "`pipelined` / `dual`; `atomic` / `tma` / `pipelined`) |",
    "| `BITSCOM_NVLS` | `1`: the all-gather half of the fused collective goes out as "
    "`multimem.st` through an NVLink multicast mapping (needs torch symmetric memory); "
    "default off |",
    "| `BITSCOM_MAX_CTAS` | grid cap of the fused collective (0 = as many CTAs as fit an empty "
    "GPU) |",
    "| `BITSCOM_LL_MAX_MB` | largest all-reduce (MiB of the tensor; 4- or 8-bit codes) that runs "
    "in the small-bucket form of the fused kernel (packed words that carry their own arrival "
    "flags), counted at four bytes per element; default 64 (16 Mi elements), 0 = never |",
    "| `BITSCOM_SYMM_MB` | size of each of the two data regions of a rank's symmetric block in MiB (default 256) |",
    "| `BITSCOM_TIMEOUT_MS` | limit of every in-kernel wait of the fused collective "
    "(default 30000) |",
    "| `BITSCOM_TIMING`, `BITSCOM_TIMING_DIR`, `BITSCOM_NVTX` | opt-in timing log, its "
    "directory, NVTX ranges |",
    "| `BITSCOM_COMM_DEBUG`, `TRACE_EXPLAIN` | the reference's debug switches: per-call log "
    "lines, path explanations |",
    "| `BITSCOM_UNSAFE_FULL_ASYNC_CHAIN` | the reference's switch: async Works that skip the "
    "final stream join |",
    "| `BITSCOM_CPU_CODEC` | `0`: CPU tensors are quantized with torch ops instead of the C++ "
    "codec |",
    "| `BITSCOM_ALLOW_FALLBACK` | `1`: on a machine with a GPU, a missing native library falls "
    "back to the host path instead of raising |",
    "| `BITSCOM_NO_BUILD`, `BITSCOM_NVCC` (`BITSCOM_CUDA_COMPILER`) | do not rebuild an "
    "existing extension; compiler to use |",
    "| `BITSCOM_AGENT_STORE`, `BITSCOM_RESTART_COUNT` | set by `bitscom_b200.launch` for its "
    "children: address of the agent's store, generation index |",
    "| `BITSCOM_INJECT_EXIT` | `rank:step[:generation]`: that rank of the Llama trainer exits "
    "before that step (host-side fault injection for recovery tests) |",
    "| `BITSCOM_RUN_PERF`, `BITSCOM_EXPERIMENTAL` | test tiers: timing tests, opt-in variants |",
    "",
]


def first_paragraph(doc):
    return inspect.cleandoc(doc).split("\n\n")[0].replace("\n", " ") if doc else ""


def signature(obj):
    try:
        return str(inspect.signature(obj)).replace("'", "")
    except (TypeError, ValueError):
        return "(...)"


def public_names(module, modname):
    return [n for n, o in vars(module).items()
            if not n.startswith("_") and (inspect.isfunction(o) or inspect.isclass(o))
            and getattr(o, "__module__", "").startswith("bitscom_b200")]


def render():
    out = ["# API reference", "",
           "Generated by `docs/make_api_reference.py` from the docstrings (first paragraph of "
           "each); public names only.", "`import bitscom_b200 as bitscom` gives the reference's "
           "names.", ""]
    for modname, names in MODULES:
        module = importlib.import_module(modname)
        out += [f"## `{modname}`", ""]
        if first_paragraph(module.__doc__):
            out += [first_paragraph(module.__doc__), ""]
        for name in names or public_names(module, modname):
            obj = getattr(module, name)
            if inspect.isclass(obj):
                out += [f"### class `{name}{signature(obj)}`", ""]
                if first_paragraph(obj.__doc__):
                    out += [first_paragraph(obj.__doc__), ""]
                for mname, member in vars(obj).items():
                    if mname.startswith("_"):
                        continue
                    if isinstance(member, property):
                        line, fn = f"* property `{mname}`", member.fget
                    elif isinstance(member, (staticmethod, classmethod)):
                        fn = member.__func__
                        line = f"* `{mname}{signature(fn)}`"
                    elif inspect.isfunction(member):
                        fn = member
                        line = f"* `{mname}{signature(fn)}`"
                    else:
                        continue
                    doc = first_paragraph(fn.__doc__)
                    out.append(line + (f" — {doc}" if doc else ""))
                out.append("")
            elif callable(obj):
                out += [f"### `{name}{signature(obj)}`", ""]
                if first_paragraph(obj.__doc__):
                    out += [first_paragraph(obj.__doc__), ""]
            else:
                out += [f"### `{name}` = `{obj!r}`", ""]
    out += ENVIRONMENT
    return "\n".join(out) + "\n"


if __name__ == "__main__":
    path = os.path.join(ROOT, "docs", "api.md")
    with open(path, "w", encoding="utf-8") as f:
        f.write(render())
    print("wrote", path)
