"""CPU test of the ids that the kernels' bounded waits leave in the status word: one per thing waited for."""
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "flash-attention-v100_b200", "csrc")
WAIT = re.compile(r"\b(?:mbar_wait|mbar_wait_warp|wait_full|global_flag_wait)\(")


def _arguments(text, start):
    """The call's arguments, from behind its opening bracket."""
    depth, args, last = 0, [], start
    for i in range(start, len(text)):
        if text[i] in "([{":
            depth += 1
        elif text[i] in ")]}":
            if depth == 0:
                return args + [text[last:i].strip()]
            depth -= 1
        elif text[i] == "," and depth == 0:
            args.append(text[last:i].strip())
            last = i + 1
    raise AssertionError("unbalanced call")


@pytest.mark.parametrize("kernel", ["fwd_kernel.cuh", "bwd_kernel.cuh"])
def test_an_id_names_one_wait(kernel):
    with open(os.path.join(CSRC, kernel)) as f:
        text = f.read()
    waits = {}
    for m in WAIT.finditer(text):
        args = _arguments(text, m.end())
        if args[-1].isdigit():  # (else a helper that passes its caller's id on)
            waits.setdefault(int(args[-1]), set()).add(args[0])
    assert len(waits) > 10
    assert [(i, w) for i, w in sorted(waits.items()) if len(w) > 1] == []
