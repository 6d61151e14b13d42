"""Structural gates, run on the sources without a GPU: the Python side and the kernel library agree on the
exported entry points, the package keeps its layering, and nothing reaches for a tracing compiler or a
second backend (the reference keeps the same kind of gates in tests/test_backends.py and
tests/test_backends_purity.py)."""
import ast
import re
import subprocess
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parents[1]
PKG = ROOT / "coffin_b200"
PY = sorted(p for p in PKG.rglob("*.py"))
CU = sorted((PKG / "_C").glob("*.cu"))


def _exports() -> set[str]:
    out = set()
    for f in CU:
        out |= set(re.findall(r"CB_EXPORT\s+[\w\s\*]+?\bcb_(\w+)\s*\(", f.read_text()))
    return out


def _called() -> dict[str, set[str]]:
    """Kernel entry points named from Python: the first string argument of call / call_nostream, and cb_ attributes."""
    used: dict[str, set[str]] = {}
    for f in PY + [ROOT / "bench.py", ROOT / "__graft_entry__.py"] + sorted((ROOT / "tests").glob("*.py")):
        src = f.read_text()
        names = set(re.findall(r"\bcall(?:_nostream)?\(\s*\"(\w+)\"", src)) | set(re.findall(r"\.cb_(\w+)\b", src))
        if f.name == "_lib.py":
            names.discard("name")                      # the docstring's placeholder
        for n in names:
            used.setdefault(n, set()).add(f.relative_to(ROOT).as_posix())
    return used


def test_every_entry_point_named_from_python_is_exported_by_the_library():
    exports, used = _exports(), _called()
    assert len(exports) > 60, "the export scan found too few symbols: the pattern no longer matches the sources"
    missing = {n: sorted(fs) for n, fs in used.items() if n not in exports}
    assert not missing, f"called from Python but not exported by any .cu: {missing}"


def test_exported_entry_points_are_reachable_from_python():
    """An export nobody calls is either dead or untested; the few that exist for other runtimes are listed."""
    allow = {"argmax_static",            # allocation-free entry point for embedding runtimes (no_alloc.h)
             "trace_register", "trace_name",
             # introspection / tuning hooks for callers that size their own scratch or sweep a variant
             "set_stream_opts", "tp_os_rows"}
    unused = sorted(_exports() - set(_called()) - allow)
    assert not unused, f"exported but never called from Python or the tests: {unused}"


def _imports(path: Path) -> set[str]:
    """Absolute module names a file imports from inside the package (relative imports resolved)."""
    tree = ast.parse(path.read_text())
    pkg_parts = path.relative_to(ROOT).with_suffix("").parts[:-1]
    out = set()
    for node in ast.walk(tree):
        if isinstance(node, ast.ImportFrom):
            if node.level:
                base = list(pkg_parts[:len(pkg_parts) - node.level + 1])
                mod = ".".join(base + ([node.module] if node.module else []))
            else:
                mod = node.module or ""
            out.add(mod)
            for a in node.names:
                out.add(f"{mod}.{a.name}")
        elif isinstance(node, ast.Import):
            out |= {a.name for a in node.names}
    return out


def test_no_tracing_compiler_second_backend_or_working_files_in_the_package():
    banned = ("triton", "tilelang", "jax", "_work", "tests")
    for f in PY:
        mods = _imports(f)
        hit = sorted(m for m in mods if m.split(".")[0] in banned)
        assert not hit, f"{f.relative_to(ROOT)} imports {hit}"
        src = f.read_text()
        assert "torch.compile(" not in src and "@torch.compile" not in src, f"{f.relative_to(ROOT)} uses torch.compile"


def test_layering_lower_layers_do_not_import_upward():
    """ops / weights / cache know nothing of the engine; the engine nothing of serving or the entry points;
    the CPU oracle is a test oracle and the CPU twin, not something the device model leans on."""
    rules = {
        "ops": ("engine", "serving", "entrypoints", "models"),
        "weights": ("engine", "serving", "entrypoints"),
        "cache": ("engine", "serving", "entrypoints", "models"),
        "engine": ("serving", "entrypoints"),
        "serving": ("entrypoints",),
        "parallel": ("serving", "entrypoints"),
    }
    bad = []
    for f in PY:
        rel = f.relative_to(PKG).parts
        layer = rel[0]
        for m in _imports(f):
            parts = m.split(".")
            if parts[0] != "coffin_b200" or len(parts) < 2:
                continue
            if parts[1] in rules.get(layer, ()):
                bad.append(f"{f.relative_to(ROOT)} -> {m}")
    # lazy imports inside functions of the debugging switches are the one sanctioned exception
    bad = [b for b in bad if "engine.debug" not in b and "engine/debug.py" not in b]
    assert not bad, "upward imports:\n" + "\n".join(sorted(set(bad)))
    for f in sorted((PKG / "models").rglob("*.py")):
        if f.name == "oracle.py":
            continue
        # oracle.ops holds the host-side table builders (rotary rows) both sides share; the oracle MODELS stay out
        leaned = [m for m in _imports(f) if m.startswith("coffin_b200.oracle") and not m.startswith("coffin_b200.oracle.ops")
                  and m != "coffin_b200.oracle"]
        assert not leaned, f"{f.relative_to(ROOT)} imports the CPU oracle: {leaned}"


def test_every_preset_resolves_and_validates():
    from coffin_b200.config import preset
    for name in ("tiny", "qwen35-4b", "qwen35-27b", "qwen35-35b-a3b", "tiny-qwen4", "qwen4exp-a", "tiny-fasolorn", "fasolorn-4b", "fasolorn-35b-a3b",
                 "tiny-nodutar", "nodutar-35b-a3b", "nodutar-3b"):
        cfg = preset(name)
        assert cfg.num_hidden_layers == len(cfg.layer_types)
        if hasattr(cfg, "validate"):
            cfg.validate()


def test_kernel_sources_are_built_for_sm_100a_only():
    src = (PKG / "_C" / "build.py").read_text()
    assert "arch=compute_100a,code=sm_100a" in src and "-lineinfo" in src
    assert not re.search(r"sm_(8\d|9\d)\b", src), "another architecture crept into the build flags"


@pytest.mark.parametrize("arch", ["zufilorn", "sukisun", "fasolorn", "nodutar"])
def test_library_of_one_family_resolves_what_it_uses(arch, tmp_path):
    """A library of a family's kernel sources alone loads (no source refers to one that is left out) and exports the products of few
    rows, of many and in 32 bits that every such family calls."""
    import ctypes
    from coffin_b200._C import build as B
    from coffin_b200.models import kernel_sources
    objs = [str(B._compile(s, False)[0]) for s in B.sources() if s.name in kernel_sources(arch)]
    so = tmp_path / "family.so"
    subprocess.run([B.nvcc(), *B.ARCH, "-shared", "-o", str(so), *objs], check=True)
    lib = ctypes.CDLL(str(so))
    for name in ("cb_gemm_rows_bf16", "cb_gemm_bf16", "cb_gemm_bf16_f32out", "cb_gemm_bf16_xielu", "cb_gemm_f32", "cb_gemv_mma_bf16", "cb_settle"):
        assert hasattr(lib, name), name


def test_decode_attention_splits_cover_one_wave():
    """CTAs of a decode attention launch: about one wave where the splits are the grid, room for partials only where the batch kernel shares
    the tiles of few rows (heads of 256)."""
    from coffin_b200.ops import kernels as K
    for nkv in (1, 2, 4, 8, 16):
        for rows in (1, 2, 4, 8, 16, 32, 64, 128):
            pairs, ns = nkv * rows, K.decode_splits(nkv, rows)
            assert ns == max(1, min(32, (148 if pairs < 32 else 296) // pairs))
            few = 32 <= pairs <= 148 and rows <= 8
            assert K.decode_splits(nkv, rows, True) == (min(64, 2368 // pairs) if few else ns)
    assert K.attn_shares_tiles(16, 4, 256, 64) and not K.attn_shares_tiles(4, 2, 64, 16) and not K.attn_shares_tiles(64, 4, 256, 64)


def test_decode_projections_of_several_rows_by_size():
    """Short sums stay on the GEMV, long ones and wide weights take the products of few rows (sizes at which both were measured)."""
    from coffin_b200.ops.kernels import _rows_gemv
    for M in range(2, 9):
        assert not _rows_gemv(M, 4096, 1024, False) and not _rows_gemv(M, 256, 256, False)
        assert _rows_gemv(M, 512, 1536, False) and _rows_gemv(M, 16384, 1024, False)
        assert _rows_gemv(M, 5120, 6144, True) and _rows_gemv(M, 152064, 5120, True)
    assert not _rows_gemv(4, 4096, 1024, True) and not _rows_gemv(2, 4096, 4096, True) and _rows_gemv(5, 4096, 1024, True)
    assert not _rows_gemv(1, 16384, 4096, False) and not _rows_gemv(9, 16384, 4096, True)
