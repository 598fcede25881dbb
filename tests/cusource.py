"""Reads the CUDA sources as text, for tests of what no run can show reliably: the order of stores and fences, and what a
kernel reads before it waits for the kernel before it."""
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "lethe_b200", "csrc")


def source(name):
    """The file without its comments."""
    with open(os.path.join(CSRC, name)) as f:
        text = f.read()
    return re.sub(r"//[^\n]*", "", re.sub(r"/\*.*?\*/", "", text, flags=re.S))


def block(text, start):
    """The braces that open at or after `start`: (contents, index behind the closing brace)."""
    i = text.index("{", start)
    depth = 0
    for j in range(i, len(text)):
        depth += {"{": 1, "}": -1}.get(text[j], 0)
        if depth == 0:
            return text[i + 1:j], j + 1
    raise ValueError("unbalanced braces")


def kernel_body(name, kernel):
    text = source(name)
    return block(text, re.search(r"\b%s\s*\(const " % kernel, text).start())[0]
