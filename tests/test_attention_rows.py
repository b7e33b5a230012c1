"""Every row of a 16-position step of the decode attention's own-copy ring is written before it is read: copied, filled with zeros, or placed
once the preceding kernel is done.  A row that nothing writes holds whatever shared memory held, and a probability of zero times a NaN from
there is a NaN; no run shows that reliably, so the conditions are read from the source and tried over splits of all lengths."""
import os
import re

SOURCE = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "lighterpp_b200", "csrc", "attention.cuh")


def python(condition):
    return compile(condition.replace("||", " or ").replace("&&", " and "), SOURCE, "eval")


def test_every_row_of_a_step_is_written():
    text = open(SOURCE).read()
    requests = re.findall(r"if \((t != pos[^;{]*?)\) cp_async_16\(", text)
    assert len(requests) == 2  # K and V
    placed = python(re.search(r"auto holds_pos = \[&\]\(int base\) \{ return ([^;]*); \}", text).group(1))
    for condition in map(python, requests):
        for T in range(1, 200):
            pos = T - 1
            for n in range(1, min(T, 24) + 1):
                chunk = -(-T // n)
                for t0 in range(0, T, chunk):
                    t1 = min(T, t0 + chunk)
                    for base in range(t0, t1, 16):
                        for t in range(base, base + 16):
                            env = dict(t=t, pos=pos, t1=t1, base=base)
                            assert eval(condition, {}, env) or (t == pos and eval(placed, {}, env)), (T, n, t0, base, t)
