"""Loading on the GPU against the host reader, which a process that has not
used the GPU takes: every form of the Edge and ID files gives the same arrays
or the same error code, and plain files do take the GPU.  The sizes put lines
across the text's 64-byte and 16 KB pieces."""
import json
import os
import subprocess
import sys

import pytest

from small_graphs import grid, path, star

pytestmark = pytest.mark.gpu
HERE = os.path.dirname(os.path.abspath(__file__))


def _lines(n, edges):
    arcs = []
    for u, v, w in edges:
        arcs += [(u, v, w), (v, u, w + 1)]
    arcs.sort(key=lambda a: a[0])  # stable: a vertex keeps its arcs' order
    return ["a %d %d %d" % (u + 1, v + 1, w) for u, v, w in arcs], ["%d 1.5 -2 %d" % ((k * 7 + 3) % n, k) for k in range(n)]


def forms():
    """name: (Edge text, ID text, whether the GPU takes it)"""
    out = {}

    def put(name, n, arcs, ids, gpu, m=None, join="\n", end="\n", head=""):
        out[name] = ("%d %d%s\n" % (n, len(arcs) if m is None else m, head) + join.join(arcs) + end,
                     "%d%s\n" % (n, head) + join.join(ids) + end, gpu)

    for n, edges in (path(2), path(1200), grid(9, 9), grid(40, 53), grid(2, 1500)):
        if n % 7 == 0:
            continue
        arcs, ids = _lines(n, edges)
        put("plain%d" % n, n, arcs, ids, True)
        put("no_end%d" % n, n, arcs, ids, True, end="")
        put("reversed%d" % n, n, arcs[::-1], ids[::-1], True)
        put("blank_lines%d" % n, n, arcs, ids, True, join="\n\n\n")
        put("crlf%d" % n, n, arcs, ids, True, join="\r\n")
    n, edges = grid(9, 9)
    arcs, ids = _lines(n, edges)
    put("tabs", n, [a.replace(" ", "\t  ") + " \t" for a in arcs], ids, True)
    put("parallel", n, arcs + arcs[5:60:3], ids, True)
    put("heavy", n, [arcs[0].rsplit(" ", 1)[0] + " 2147483647"] + arcs[1:], ids, True)
    put("zero", n, [arcs[0].rsplit(" ", 1)[0] + " 0"] + arcs[1:], ids, True)
    put("overweight", n, [arcs[0].rsplit(" ", 1)[0] + " 2147483648"] + arcs[1:], ids, False)
    put("negative", n, [arcs[0].rsplit(" ", 1)[0] + " -1"] + arcs[1:], ids, False)
    put("plus", n, ["a +1" + arcs[0][3:]] + arcs[1:], ids, False)
    put("zeros", n, ["a 000000000001" + arcs[0][3:]] + arcs[1:], ids, False)
    put("id0", n, ["a 0 2 5"] + arcs[1:], ids, False)
    put("id_large", n, ["a 1 82 5"] + arcs[1:], ids, False)
    put("loop", n, arcs + ["a 3 3 1"], ids, False)
    put("one_way", n, arcs[:-1], ids, False)
    put("more_lines", n, arcs + ["a 1 2 3"], ids, False, m=len(arcs))
    put("fewer_lines", n, arcs, ids, False, m=len(arcs) + 1)
    put("two_a_line", n, [arcs[0] + " " + arcs[1]] + arcs[2:], ids, False, m=len(arcs))
    put("spread", n, [arcs[0].replace(" ", "\n")] + arcs[1:], ids, False, m=len(arcs))
    put("leading_blank", n, [" " + arcs[0]] + arcs[1:], ids, False)
    put("long_line", n, [arcs[0] + " " * 300] + arcs[1:], ids, False)
    put("header_blank", n, arcs, ids, False, head=" ")
    put("junk", n, ["x" + arcs[0][1:]] + arcs[1:], ids, False)
    put("trailing_word", n, [arcs[0] + " b"] + arcs[1:], ids, False)
    put("position_twice", n, arcs, ids[:-1] + [ids[0]], False)
    put("position_large", n, arcs, ids[:-1] + ["%d 1 2 80" % n], False)
    put("split", n + 2, arcs + ["a 82 83 1", "a 83 82 1"], ids + ["81 0 0 81", "82 0 0 82"], False)
    put("lonely", n + 1, arcs, ids + ["81 0 0 81"], False)
    put("split_and_bad_id", n + 2, arcs + ["a 82 83 1", "a 83 82 1"], ids + ["81 0 0 81", "81 0 0 82"], False)
    n, edges = star(511)
    put("star512", n, *_lines(n, edges), True)
    n, edges = star(514)
    put("star515", n, *_lines(n, edges), False)
    return out


def load_all(root, gpu):
    import gpuh2h
    got = {}
    if gpu:  # the process has used the GPU
        import torch
        torch.zeros(1, device="cuda").cpu()
    for name, (edge, ids, _) in forms().items():
        e, i, c = (os.path.join(root, name + x) for x in (".edge", ".id", ".cut"))
        n = int(edge.split()[0])
        for f, text in ((e, edge), (i, ids), (c, "1\n1 0 %d\n" % n)):
            with open(f, "w", newline="") as h:
                h.write(text)
        try:
            g = gpuh2h.Graph("g", 1, 1, 4, 1, files=(e, i, c))
            got[name] = [x.tolist() for x in (*g.input_arcs(), *g.partition())]
            g.close()
        except gpuh2h.H2HError as err:
            got[name] = err.code
    return got


def test_forms_match_host_reader(tmp_path, capfd, monkeypatch):
    monkeypatch.setenv("GPUH2H_TRACE", "1")
    capfd.readouterr()
    got = load_all(str(tmp_path), True)
    taken = capfd.readouterr().err.count("files parsed on the device")
    env = dict(os.environ, CUDA_VISIBLE_DEVICES="", PYTHONPATH=os.pathsep.join([HERE] + sys.path))
    out = subprocess.run([sys.executable, "-c", "import json, sys, test_load_forms_gpu as t; "
                          "json.dump(t.load_all(sys.argv[1], False), open(sys.argv[2], 'w'))",
                          str(tmp_path), str(tmp_path / "host.json")],
                         env=env, capture_output=True, text=True, timeout=300)
    assert out.returncode == 0, out.stderr
    assert "parsed on the device" not in out.stderr
    want = json.load(open(tmp_path / "host.json"))
    assert set(got) == set(want)
    for name in want:
        assert got[name] == want[name], name
    assert taken == sum(gpu for _, _, gpu in forms().values())


def test_load_and_read_back_during_a_capture(tmp_path):
    """Loading a graph and reading a built one back stay host calls: they run
    beside a graph capture (global mode) and do not spoil it."""
    import gpuh2h
    import torch

    from small_graphs import write
    n, edges = grid(9, 9)
    files = write(tmp_path, n, [(u, v, w, w) for u, v, w in edges], 2)
    ref = gpuh2h.Graph("g", 2, 1, 2, 1, files=files)
    arcs, built = ref.input_arcs(), ref.contraction_noHub(1)
    order = ref.order()
    other = gpuh2h.Graph("g", 2, 1, 2, 1, files=files).contraction_noHub(1)
    x = torch.zeros(4, device="cuda")
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, capture_error_mode="global"):
        x += 1
        g = gpuh2h.Graph("g", 2, 1, 2, 1, files=files)
        got = g.input_arcs()
        assert (other.order() == order).all()
        x += 1
    graph.replay()
    torch.cuda.synchronize()
    assert x.tolist() == [2.0] * 4
    assert all((a == b).all() for a, b in zip(arcs, got))
    for h in (g, built, other):
        h.close()
