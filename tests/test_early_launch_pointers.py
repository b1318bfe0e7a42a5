"""Kernels that start before their predecessor has ended (griddepcontrol.wait) take the data it
may still write through plain pointers: __restrict__ const promises the compiler that nothing
writes them while the kernel runs, which lets it use loads that are not kept coherent, or move
them above the wait."""
from __future__ import annotations

import re
from pathlib import Path

import anisotropicelastoplasticity_gb300 as pkg

CSRC = Path(pkg.__file__).parent / "csrc"
# the training records: written before the call that launches the kernels
CONSTANT = {("k_mlp_train_tile", "rec")}


def functions():
    """name -> (is a kernel, parameter list, body) of every device function and kernel."""
    out = {}
    for path in sorted(CSRC.glob("*.cu*")):
        text = re.sub(r"//[^\n]*|/\*.*?\*/", "", path.read_text(), flags=re.S)
        for m in re.finditer(r"__(global|device)__\s", text):
            close = text.find("{", m.end())
            head = text[m.end():close]
            if close < 0 or ";" in head:
                continue
            head = re.sub(r"__launch_bounds__\s*\((?:[^()]|\([^()]*\))*\)", "", head)
            name = re.search(r"(\w+)\s*\((.*)\)\s*$", head, flags=re.S)
            if not name:
                continue
            depth, end = 1, close + 1
            while depth:
                depth += {"{": 1, "}": -1}.get(text[end], 0)
                end += 1
            out[name.group(1)] = (m.group(1) == "global", name.group(2), text[close:end])
    return out


def test_waiting_kernels_take_no_restricted_pointers():
    fn = functions()
    waits = [k for k, (kernel, _, body) in fn.items()
             if kernel and re.search(r"pdl_wait\s*\(|pdl_entry\s*\(|griddepcontrol\.wait", body)]
    assert {"k_p2g", "k_normalize", "k_force", "k_force_fp64", "k_grid", "k_g2p", "k_mlp_finish", "k_cloth_g2p",
            "k_solve_dt", "k_mlp_train_tile", "k_mlp_reduce"} <= set(waits)
    bad = []
    for k in waits:
        seen, todo = set(), [k]
        while todo:  # the kernel and the device functions that it calls
            f = todo.pop()
            seen.add(f)
            for q in re.findall(r"__restrict__\s+(\w+)", fn[f][1]):
                if (f, q) not in CONSTANT:
                    bad.append((k, f, q))
            if re.search(r"__ldg\s*\(|ld\.global\.nc", fn[f][2]):
                bad.append((k, f, "__ldg"))
            todo += [c for c in set(re.findall(r"(\w+)\s*(?:<[^<>;]*>)?\s*\(", fn[f][2])) if c in fn and c not in seen]
    assert not bad, sorted(set(bad))
