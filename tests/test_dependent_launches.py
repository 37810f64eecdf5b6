"""Kernels that may start while the stream's previous kernel still runs read
what that kernel writes, so none of their pointers may promise the compiler
memory that stays unchanged while the kernel lives (const __restrict__, __ldg:
loads through the read-only path)."""
import re
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parents[1] / "eemd4cuda_b200" / "csrc"


def closing(text, i, pair):
    """The index after the bracket that closes text[i]."""
    depth = 0
    for j in range(i, len(text)):
        depth += (text[j] == pair[0]) - (text[j] == pair[1])
        if depth == 0:
            return j + 1
    raise ValueError("unbalanced")


def functions(text):
    """{name: (parameters, body)} of the device functions and kernels of a source."""
    text = re.sub(r"//[^\n]*", "", text)
    text = re.sub(r"__launch_bounds__\([^()]*\)", "", text)
    out = {}
    for m in re.finditer(r"__(?:global|device)__", text):
        head = re.compile(r"[\w\s*&:<>,]*?(\w+)\s*\(").match(text, m.end())
        if not head:
            continue
        p1 = closing(text, head.end() - 1, "()")
        b0 = re.compile(r"\s*\{").match(text, p1)
        if b0:
            out[head[1]] = (text[head.end():p1 - 1], text[b0.end() - 1:closing(text, b0.end() - 1, "{}")])
    return out


@pytest.mark.parametrize("source,some", [("spectra.cu", {"k_hil_cols", "k_hil_rows", "k_hil_out", "k_hil_small"}),
                                         ("surrogate.cu", {"k_conv_ws", "k_wgrad_ws", "k_loss", "k_adam", "k_sumsq",
                                                           "k_pack_layers"})])
def test_no_read_only_promise(source, some):
    fns = functions((CSRC / source).read_text())
    dependent = {n for n, (_, body) in fns.items() if "after_previous_kernel()" in body}
    assert some <= dependent
    # and what they call
    todo = list(dependent)
    while todo:
        body = fns[todo.pop()][1]
        for n in fns:
            if n not in dependent and re.search(r"\b%s\s*(<[^;{}]*>)?\s*\(" % n, body):
                dependent.add(n)
                todo.append(n)
    for n in sorted(dependent):
        params, body = fns[n]
        assert "__restrict__" not in params and "__restrict__" not in body, n
        assert "__ldg" not in body and "ld.global.nc" not in body, n
