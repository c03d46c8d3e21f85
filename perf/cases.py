"""The traversals that users of the engine run, as timed cases.

A case is one call path on one graph:

  call   "host"    the reference-shaped entry points GPU<alg>_{vertex,edge}(src, g, out): the graph
                   is resident, the result lands in a host array, the device time comes back
         "device"  DeviceGraph.run_device: graph and result stay on the device, the call is queued
                   on the caller's stream (analytics loops, queries from many sources)
         "batch"   Batch.run: many graphs traversed together, results in host arrays
         "coo"     an edge list in device memory becomes a graph, is traversed once and dropped
                   (edge lists that change from step to step)
         "upload"  a host CSR is uploaded, traversed once and dropped (one program run per file)
  algo   bfs, sssp, cc, mis
  family er (average degree 8), rmat (edge factor 16), grid (5% of the edges removed, 0.1%
         long-range edges added): the families and parameters of indigo2suite_b200/workloads.py
  n      vertices (grid: side ceil(sqrt(n)))
  style  the relax style or the selector; "edge" as style of a host call is the edge harness's entry point
  order  the traversals run on the degree-ordered copy (DeviceGraph.reorder)

Sources are each graph's highest-degree vertex, as in the benchmark's configurations. Values are
int32 levels, distances, labels or set membership: exact whatever the order of the relaxations.
"""
import math

import numpy as np
import torch

import indigo2suite_b200 as i2
from indigo2suite_b200 import selector, workloads

_ALGO = {"bfs": i2.I2_BFS, "sssp": i2.I2_SSSP, "cc": i2.I2_CC, "mis": i2.I2_MIS}
_FAMILIES = ("er", "rmat", "grid")
_BATCH_MIN, _BATCH_MAX = 1e3, 1e6  # vertices of a batch's graphs, as in workloads.batch_specs


def _case(name, call, algo, family, n, style="heuristic", order=False, count=1):
    c = {"call": call, "algo": algo, "family": family, "n": n, "style": style, "order": order, "count": count}
    if name:
        c["name"] = name
    return c


def listed():
    return [
        # the smallest queries: a few thousand vertices, one after another on a stream
        _case("sssp_rmat_3001_device", "device", "sssp", "rmat", 3001),
        # the suite's CPU configuration (ER 2^16 BFS) through the drop-in call
        _case("bfs_er_65536_host", "host", "bfs", "er", 65536),
        # road-network-like: many iterations with small frontiers
        _case("bfs_grid_4m_device", "device", "bfs", "grid", 4_000_000),
        # components of the 4096 x 4096 grid configuration
        _case("cc_grid_4096x4096_device", "device", "cc", "grid", 1 << 24),
        # the learned selector on a scale-20 social-network-like graph
        _case("bfs_rmat_2e20_learned", "device", "bfs", "rmat", 1 << 20, "learned"),
        # weighted uniform random graph, ragged size, the default style
        _case("sssp_er_2000003_vp_cta", "device", "sssp", "er", 2_000_003, "vp_cta"),
        # the benchmark's headline traversal (RMAT-22 SSSP, chosen by the rule)
        _case("sssp_rmat_2e22", "device", "sssp", "rmat", 1 << 22),
        # the largest: RMAT-25 on its degree-ordered copy, as the RMAT-26 configuration runs
        _case("sssp_rmat_2e25_ordered", "device", "sssp", "rmat", 1 << 25, order=True),
        # maximal independent set
        _case("mis_rmat_1000003", "device", "mis", "rmat", 1_000_003),
        # a batch as in the 512-graph configuration, a sixteenth of its size
        _case("sssp_batch_32", "batch", "sssp", "mixed", 0, "vp_cta", count=32),
        # components of an edge list that was made on the device
        _case("cc_coo_1000003", "coo", "cc", "coo", 1_000_003),
        # one program run per file: upload, SSSP, results back
        _case("sssp_upload_rmat_300007", "upload", "sssp", "rmat", 300_007),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    call = rng.choice(["host", "device", "device", "device", "batch", "coo", "upload"])
    algo = rng.choice(["bfs", "sssp", "cc"])
    if call == "batch":
        return _case(None, call, algo, "mixed", 0, rng.choice(["vp_cta", "heuristic"]), count=rng.randint(8, 32))
    if call == "coo":
        return _case(None, call, algo, "coo", _log(rng, 1e4, 1e6))
    family = rng.choice(_FAMILIES)
    if call == "upload":
        return _case(None, call, algo, family, _log(rng, 1e3, 3e5))
    if call == "host":
        return _case(None, call, algo, family, _log(rng, 1e3, 1e6), rng.choice(["vertex", "edge"]))
    if rng.random() < 0.15:
        return _case(None, call, "mis", family, _log(rng, 1e3, 1e6))
    n = _log(rng, 1e3, 3e7 if family == "rmat" else 8e6)
    # the degree-ordered copy is meant for large skewed graphs
    order = family == "rmat" and n > 500_000 and rng.random() < 0.4
    return _case(None, call, algo, family, n, rng.choice(["heuristic", "heuristic", "learned", "vp_cta"]), order)


def _pairs(n):
    return 8 * n  # edge-list cases: pairs given


def _batch_sizes(count):
    return [int(_BATCH_MIN * (_BATCH_MAX / _BATCH_MIN) ** ((k + 0.5) / count)) for k in range(count)]


def _entries(family, n):
    """CSR entries of a graph, near enough."""
    if family == "er":
        return 8 * n
    if family == "grid":
        return int(4 * n * 0.951)
    scale = max(1, math.ceil(math.log2(n)))  # 16 * 2^scale samples, both endpoints below n
    return int(32 * n * (n / 2**scale) * 0.93)


def _csr_bytes(algo, family, n):
    e = _entries(family, n)
    return 4 * (n + 1) + 4 * e + (4 * e if algo == "sssp" else 0)


def work(case):
    algo, n = case["algo"], case["n"]
    if case["call"] == "batch":
        sizes = _batch_sizes(case["count"])
        b = sum(_csr_bytes(algo, _FAMILIES[k % 3], m) + 4 * m for k, m in enumerate(sizes))
    elif case["call"] == "coo":
        b = _pairs(n) * (12 if algo == "sssp" else 8) + 4 * n
    else:
        b = _csr_bytes(algo, case["family"], n) + 4 * n
        if case["call"] == "upload" and algo != "sssp":
            b += 4 * _entries(case["family"], n)  # the file's weights go up with the graph
    return {"bytes": b, "flops": 0}


_shared = {}


def _stream():
    """The program's one stream: queries are queued on it in order."""
    if "s" not in _shared:
        _shared["s"] = torch.cuda.Stream()
    return _shared["s"]


def _pinned(a):
    t = torch.empty(a.size, dtype=torch.int32, pin_memory=True)
    t.numpy()[:] = a
    return t


def prepare(case, seed):
    call, algo, n = case["call"], case["algo"], case["n"]
    gseed = 1 + seed % (2**31 - 2)
    st = {"call": call, "algo": algo, "code": _ALGO[algo], "style": case["style"], "n": n}
    if case["style"] == "learned":
        i2.mlp_set_params(np.fromfile(selector.PARAMS_PATH, np.float32))
    if call == "batch":
        rng = np.random.default_rng(gseed)
        specs = [(_FAMILIES[k % 3], m, int(rng.integers(1, 2**31 - 1)))
                 for k, m in enumerate(_batch_sizes(case["count"]))]
        graphs = [workloads.build_device(s) for s in specs]
        st["srcs"] = None if algo == "cc" else [g.hub() for g in graphs]
        st["batch"] = i2.Batch(graphs)
        return st
    if call == "coo":
        gen = torch.Generator(device="cuda").manual_seed(gseed)
        m = _pairs(n)
        # endpoints of skewed popularity (the square of a uniform number), as user-item or link lists have
        ends = [(torch.rand(m, generator=gen, device="cuda", dtype=torch.float64).square_() * n).to(torch.int32)
                for _ in range(2)]
        st["src_ids"], st["dst_ids"] = ends
        st["w"] = torch.randint(1, 256, (m,), generator=gen, device="cuda", dtype=torch.int32) if algo == "sssp" else None
        st["m"] = m
        st["out"] = torch.empty(n, dtype=torch.int32, device="cuda")
        return st
    dg = workloads.build_device((case["family"], n, gseed))
    st["src"] = dg.hub()
    if call == "upload":
        h = dg.download()
        dg.free()
        st["pins"] = [_pinned(a) for a in (h.nindex, h.nlist, h.eweight)]
        st["host"] = i2.ECLGraph(h.nodes, h.edges, *[t.numpy() for t in st["pins"]])
        st["out"] = np.empty(h.nodes, np.int32)
        return st
    if case["order"]:
        dg.reorder("degree")
    st["g"] = dg
    if call == "host":
        st["out"] = np.empty(dg.nodes, np.int32)
    else:
        st["out"] = torch.empty(dg.nodes, dtype=torch.int32, device="cuda")
    return st


def run(st):
    call, algo, out = st["call"], st["algo"], st.get("out")
    if call == "device":
        st["g"].run_device(st["code"], st.get("src", 0), out.data_ptr(), variant=st["style"],
                           stream=_stream().cuda_stream, report=False)
        return out
    if call == "host":
        fn = getattr(i2, "GPU%s_%s" % (algo, st["style"] if st["style"] == "edge" else "vertex"))
        if algo == "cc":
            fn(st["g"], out)
        else:
            fn(st["src"], st["g"], out)
        return out
    if call == "batch":
        return st["batch"].run(st["code"], st["srcs"], variant=st["style"])[0]
    if call == "coo":
        w = st["w"]
        g = i2.DeviceGraph.from_coo_device(st["n"], st["m"], st["src_ids"].data_ptr(), st["dst_ids"].data_ptr(),
                                           w.data_ptr() if w is not None else 0, symmetrize=True)
        g.run_device(st["code"], 0, out.data_ptr(), variant=st["style"], stream=_stream().cuda_stream, report=False)
        g.free()
        return out
    g = i2.DeviceGraph.upload(st["host"])
    if algo == "cc":
        g.cc(variant=st["style"], out=out)
    else:
        getattr(g, algo)(st["src"], variant=st["style"], out=out)
    g.free()
    return out
