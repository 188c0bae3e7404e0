"""Kernels that are scheduled while the launch before them still runs (chain_begin,
kernels.cuh) must not read its output through the read-only path, which asks for memory that
stays as it is for the kernel's whole lifetime, nor through a pointer from which the compiler
may take a load ahead of the wait.  Checked in the sources: a race has no result to test."""
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "ctdm_gb300", "csrc")


def source(name):
    """The file without comments and launch bounds (whose expressions hold calls)."""
    text = re.sub(r"//[^\n]*", "", open(os.path.join(CSRC, name)).read())
    return re.sub(r"__launch_bounds__\((?:[^()]|\((?:[^()]|\([^()]*\))*\))*\)", "", text)


TEXT = {f: source(f) for f in sorted(os.listdir(CSRC)) if f.endswith((".cu", ".cuh"))}
# tables, and a tape's sample lists (complete when the tape is created)
COMPLETE = {"tw", "dtw", "dts", "dth", "eig", "egs", "a.tcount", "a.toff", "a.tmask", "a.tprefix", "a.yt", "a.rank"}


def body(text, at):
    """From the `{` at or after `at` to its partner."""
    start = text.index("{", at)
    depth = 0
    for i in range(start, len(text)):
        depth += {"{": 1, "}": -1}.get(text[i], 0)
        if depth == 0:
            return text[start:i]


def functions(text):
    """name -> (parameters, body) of the device functions of a file; loader structs by name."""
    out = {}
    for m in re.finditer(r"__(?:global|device)__[\w\s*&<>:]*?\b(\w+)\(([^{};]*)\)\s*\{", text):
        out.setdefault(m.group(1), []).append((m.group(2), body(text, m.end() - 1)))
    for m in re.finditer(r"struct (Load\w+) \{", text):
        out[m.group(1)] = [("", body(text, m.end() - 1))]
    return out


def chained():
    """(file, kernel, parameters, body with the bodies of the functions it calls)."""
    for f, text in TEXT.items():
        fns = functions(text)
        for name, forms in fns.items():
            for params, b in forms:
                if not re.search(r"\bchain_(begin\(\)|pass<\w+>\(a\));", b) or name == "chain_pass":
                    continue
                seen, todo = {name}, [b]
                while todo:
                    for callee in set(re.findall(r"\b(\w+)(?:<[^<>()]*>)?\(", todo.pop())) & set(fns) - seen:
                        seen.add(callee)
                        todo += [x for _, x in fns[callee]]
                yield f, name, params, b, [x for n in seen for _, x in fns[n]]


KERNELS = list(chained())


def test_kernels_are_found():
    assert {"rows_fn_kernel", "cols_kernel", "tv_kernel", "tape_z_kernel", "ewald_kernel", "prep_resize_kernel",
            "dct_unwrap_kernel", "qpi_rows_kernel", "qpib_rows_kernel", "pack_measured_kernel", "xpass_kernel",
            "ypass_kernel", "zpass_kernel", "zpass_packed_kernel"} <= {k[1] for k in KERNELS}


@pytest.mark.parametrize("f,name,params,own,bodies", KERNELS, ids=[k[1] for k in KERNELS])
def test_chained_kernel(f, name, params, own, bodies):
    for b in bodies:
        for arg in re.findall(r"__ldg\(([^;]*)", b):
            base = re.match(r"&?\s*(?:reinterpret_cast<[^>]*>\()?&?([\w.]+)", arg).group(1)
            assert base in COMPLETE, f"{f}: {name} reads {base} through the read-only path"
    for p in re.findall(r"const [\w]+ \*__restrict__ (\w+)", params):
        assert p in COMPLETE or f"{p} = fresh({p})" in own, f"{f}: {name}: {p} is not passed through fresh()"
    if name == "rows_fn_kernel":
        assert "ld.p = fresh(ld.p)" in own


def test_loaders_of_the_row_kernel():
    loaders = [(f, n, b) for f, text in TEXT.items() for n, forms in functions(text).items()
               if n.startswith("Load") for _, b in forms]
    assert len(loaders) >= 3
    for f, n, b in loaders:
        assert "__ldg" not in b, f"{f}: {n}"


def test_struct_pointers_read_by_intrinsics():
    for f, name, _, own, _ in KERNELS:
        for base in set(re.findall(r"__ldc[asg]\(&(a\.\w+)\[", own)):
            assert f"{base} = fresh({base})" in own or ("chain_pass<L>(a)" in own and base in ("a.G", "a.F2")), (f, name, base)
