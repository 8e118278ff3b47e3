"""Measured workloads of the channel engine: radiomaps, path tables, gradients,
frozen-topology replay and frequency responses on seeded synthetic cities.

Every case is one call (or one forward and its backward) through the public
entry points, on a scene that the program holds compiled, as a radio planner,
a ray-traced link simulator or a calibration loop does.  Cities come from
``witwin_channel_b200.workloads`` (lots of 50 m, boxes of 10-40 m footprint
and 10-60 m height, concrete and, where transmission is on, thin glass
sheets); the transmitter stands on a street, receivers at 1.5 m.
"""

from __future__ import annotations

import math
from types import SimpleNamespace

import numpy as np
import torch
import torch.autograd.forward_ad as fwAD

from witwin_channel_b200 import Config, solve
from witwin_channel_b200 import path as paths_api
from witwin_channel_b200.batch import solve_batch
from witwin_channel_b200.channel import cfr
from witwin_channel_b200.compiler import compile_scene
from witwin_channel_b200.propagation import consumer
from witwin_channel_b200.scene import PhysicalMaterial, Scene, make_receiver, make_receiver_grid, make_transmitter
from witwin_channel_b200.workloads import city_layout, city_scene, concrete, ground_structure, street_point

C0 = 299_792_458.0
EPS0 = 8.8541878128e-12
MAP = ("los", "reflection", "diffraction")


def listed() -> list[dict]:
    return [
        # the smallest call: the two-ray ground check (open ground, 64 x 64 cells at 2 m, 3.5 GHz); launches and host work
        {"name": "two_ray_64", "kind": "two_ray", "rows": 64, "cols": 64, "spacing": 2.0, "ghz": 3.5},
        # a handful of MIMO links in a small town: path solver with a synthetic array at both ends, then each pair's CFR
        {"name": "links_16box", "kind": "links", "boxes": 16, "receivers": 37, "tx_elements": 4, "rx_elements": 2,
         "depth": 2, "ghz": 6.0, "subcarriers": 301},
        # the ordinary radiomap: the 64-box urban canyon, 256 x 256 cells at 1.5 m, 28 GHz, depth 3 and UTD
        {"name": "canyon_map", "kind": "map", "boxes": 64, "rows": 256, "cols": 256, "spacing": 1.5, "depth": 3,
         "ghz": 28.0, "precision": "mixed", "coherent": True},
        # the same in the all-FP64 form that a reference run takes, on a ragged grid
        {"name": "canyon_map_fp64", "kind": "map", "boxes": 64, "rows": 131, "cols": 97, "spacing": 3.0, "depth": 3,
         "ghz": 28.0, "precision": "fp64", "coherent": True},
        # two scenes of a training set, four transmitters and four bands each: the batched forward
        {"name": "batch_forward", "kind": "batch", "boxes_a": 48, "side_a": 128, "boxes_b": 128, "side_b": 320,
         "tx": 4, "bands": 4, "depth": 3, "grad": False},
        # the batched forward and its VJP with respect to concrete's eps_r and sigma_e and every transmitter position
        {"name": "batch_vjp", "kind": "batch", "boxes_a": 48, "side_a": 128, "boxes_b": 128, "side_b": 320,
         "tx": 4, "bands": 4, "depth": 3, "grad": True},
        # one step of a calibration loop on the canyon: fit to a measured map in dB, gradients of materials, the
        # carrier, the transmitter and the vertices of eight buildings
        {"name": "canyon_gradient", "kind": "gradient", "boxes": 64, "rows": 256, "cols": 256, "spacing": 1.5,
         "depth": 3, "ghz": 28.0, "moved": 8},
        # forward mode: sensitivity of a small map to the transmitter's position and the material
        {"name": "town_jvp", "kind": "jvp", "boxes": 32, "rows": 90, "cols": 70, "spacing": 3.0, "depth": 2, "ghz": 6.0},
        # path tables for a dense ragged grid with windows: LoS, reflection and transmission, exported
        {"name": "city_export", "kind": "export", "boxes": 128, "rows": 201, "cols": 315, "spacing": 1.5, "depth": 2,
         "ghz": 28.0},
        # moving users: the frozen LoS and reflection rows of a canyon replayed over slots of moved sinks
        {"name": "replay_slots", "kind": "replay", "boxes": 64, "side": 160, "depth": 3, "slots": 8, "ghz": 28.0},
        # wideband spectra of every link of a large map: 1024 subcarriers of 390.625 kHz
        {"name": "cfr_wide", "kind": "cfr", "links": 262144, "subcarriers": 1024, "mean_paths": 2.0, "df_khz": 390.625},
        # the largest: a 2048-box city with subdivided roofs and glass, 1024 x 1024 cells, depth 5, all components
        {"name": "large_city", "kind": "map", "boxes": 2048, "rows": 1024, "cols": 1024, "spacing": 1.0, "depth": 5,
         "ghz": 28.0, "precision": "mixed", "coherent": True, "glass": True, "roofs": True},
    ]


def _log(rng, lo, hi) -> int:
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng) -> dict:
    kind = rng.choice(["two_ray", "links", "map", "map", "batch", "batch", "gradient", "jvp", "export", "replay", "cfr"])
    ghz = rng.choice([3.5, 6.0, 28.0, 39.0])
    if kind == "two_ray":
        return {"kind": kind, "rows": rng.randint(16, 256), "cols": rng.randint(16, 256),
                "spacing": round(rng.uniform(0.1, 0.7), 3), "ghz": ghz}
    if kind == "links":
        return {"kind": kind, "boxes": _log(rng, 8, 96), "receivers": _log(rng, 4, 200),
                "tx_elements": rng.randint(1, 8), "rx_elements": rng.randint(1, 4), "depth": rng.randint(1, 3),
                "ghz": ghz, "subcarriers": _log(rng, 16, 2048)}
    if kind == "map":
        big = rng.random() < 0.25
        return {"kind": kind, "boxes": _log(rng, 300, 1500) if big else _log(rng, 8, 256),
                "rows": _log(rng, 48, 400), "cols": _log(rng, 48, 400), "spacing": round(rng.uniform(1.0, 2.5), 2),
                "depth": rng.randint(1, 4), "ghz": ghz, "precision": rng.choice(["mixed", "mixed", "fp64"]),
                "coherent": rng.random() < 0.8, "glass": rng.random() < 0.4, "roofs": big}
    if kind == "batch":
        return {"kind": kind, "boxes_a": _log(rng, 12, 96), "side_a": _log(rng, 40, 192), "boxes_b": _log(rng, 16, 160),
                "side_b": _log(rng, 48, 256), "tx": rng.randint(1, 4), "bands": rng.randint(1, 4),
                "depth": rng.randint(1, 3), "grad": rng.random() < 0.6}
    if kind == "gradient":
        return {"kind": kind, "boxes": _log(rng, 12, 100), "rows": _log(rng, 48, 256), "cols": _log(rng, 48, 256),
                "spacing": round(rng.uniform(1.0, 2.5), 2), "depth": rng.randint(1, 3), "ghz": ghz,
                "moved": rng.randint(1, 10)}
    if kind == "jvp":
        return {"kind": kind, "boxes": _log(rng, 8, 64), "rows": _log(rng, 24, 160), "cols": _log(rng, 24, 160),
                "spacing": round(rng.uniform(1.0, 3.0), 2), "depth": rng.randint(1, 3), "ghz": ghz}
    if kind == "export":
        return {"kind": kind, "boxes": _log(rng, 16, 256), "rows": _log(rng, 48, 320), "cols": _log(rng, 48, 320),
                "spacing": round(rng.uniform(1.0, 2.5), 2), "depth": rng.randint(1, 3), "ghz": ghz}
    if kind == "replay":
        return {"kind": kind, "boxes": _log(rng, 16, 128), "side": _log(rng, 40, 200), "depth": rng.randint(1, 3),
                "slots": rng.randint(1, 10), "ghz": ghz}
    return {"kind": "cfr", "links": _log(rng, 500, 250000), "subcarriers": _log(rng, 50, 1024),
            "mean_paths": round(rng.uniform(0.5, 8.0), 2), "df_khz": rng.choice([15.0, 30.0, 120.0, 390.625])}


# ------------------------------------------------------------------ scenes
def _grid(rows: int, cols: int, spacing: float):
    return make_receiver_grid(origin=(-(rows - 1) / 2.0 * spacing, -(cols - 1) / 2.0 * spacing, 1.5),
                              x_axis=(1.0, 0.0, 0.0), y_axis=(0.0, 1.0, 0.0), shape=(rows, cols),
                              spacing=(spacing, spacing))


def _town(case: dict, seed: int, boxes: int, material=None):
    """Structures of a seeded town and a generator for its endpoints."""
    layout = city_layout(boxes, seed, lots=46 if boxes == 2048 else None)
    rng = np.random.default_rng(seed + 1000)
    sheets = []
    if case.get("glass"):
        for x0, y0, x1, y1, h in layout.boxes:
            if rng.uniform() < 0.25:
                cx = 0.5 * (x0 + x1)
                sheets.append(((cx, y0 + 0.5), (cx, y1 - 0.5), 0.8 * h))
    roof = (lambda b: 4 if b % 2 == 0 else 5) if case.get("roofs") else None
    return layout, city_scene(layout, material=material, roof_k=roof, sheets=sheets), rng


def _map_scene(case: dict, seed: int, material=None):
    layout, structures, rng = _town(case, seed, case["boxes"], material)
    tx = make_transmitter(street_point(layout, rng, float(rng.uniform(10.0, 40.0))))
    return Scene(structures=structures, endpoints=[tx, _grid(case["rows"], case["cols"], case["spacing"])]), rng


def _components(case: dict) -> set:
    return set(MAP) | ({"transmission"} if case.get("glass") else set())


def _concrete_leaves(ghz: float):
    eps = torch.tensor(5.24, dtype=torch.float64)
    sig = torch.tensor(0.0462 * ghz ** 0.7822, dtype=torch.float64)
    return eps, sig, PhysicalMaterial(eps_r=eps, sigma_e=sig, thickness_m=0.3, name="concrete")


def prepare(case: dict, seed: int):
    kind = case["kind"]
    freq = case.get("ghz", 28.0) * 1e9
    device = torch.device("cuda", torch.cuda.current_device())
    if kind == "two_ray":
        half = max(case["rows"], case["cols"]) * case["spacing"]
        tx = make_transmitter(_two_ray_tx(seed))
        scene = Scene(structures=[ground_structure(half, concrete(10.0, "ground"), surface_id=0)],
                      endpoints=[tx, _grid(case["rows"], case["cols"], case["spacing"])])
        compile_scene(scene, device)
        return {"kind": "map", "scene": scene, "freq": freq, "precision": "mixed",
                "config": Config(components={"los", "reflection"}, max_depth=1)}
    if kind == "map":
        scene, _ = _map_scene(case, seed)
        compile_scene(scene, device)
        return {"kind": kind, "scene": scene, "freq": freq, "precision": case["precision"],
                "config": Config(components=_components(case), max_depth=case["depth"], coherent=case["coherent"])}
    if kind == "export":
        scene, _ = _map_scene({**case, "glass": True}, seed)
        compile_scene(scene, device)
        cells, depth = case["rows"] * case["cols"], case["depth"]
        table = {k: ((), torch.int32) for k in ("tx", "rx", "component", "depth")}
        table |= {"faces": ((depth,), torch.int32), "delay": ((), torch.float32), "coefficient": ((), torch.complex64),
                  "positions": ((depth, 3), torch.float32), "normals": ((depth, 3), torch.float32)}
        return {"kind": kind, "scene": scene, "freq": freq, "table": _buffers(3 * cells, table, device),
                "config": Config(components={"los", "reflection", "transmission"}, max_depth=case["depth"],
                                 export_paths=True)}
    if kind == "links":
        layout, structures, rng = _town(case, seed, case["boxes"])

        def elements(n):
            pos = torch.zeros((n, 3))
            pos[:, 1] = (torch.arange(n) - (n - 1) / 2) * (0.5 * C0 / freq)
            return pos

        tx = make_transmitter(street_point(layout, rng, 20.0), element_positions=elements(case["tx_elements"]))
        rxs = [make_receiver(street_point(layout, rng, 1.5), element_positions=elements(case["rx_elements"]))
               for _ in range(case["receivers"])]
        scene = Scene(structures=structures, endpoints=[tx, *rxs])
        compile_scene(scene, device)
        k = case["subcarriers"]
        pairs = case["receivers"] * case["rx_elements"] * case["tx_elements"]
        table = _buffers(96, {"a": ((pairs,), torch.complex64), "tau": ((pairs,), torch.float32)}, device)
        return {"kind": kind, "scene": scene, "freq": freq, "table": table,
                "config": paths_api.Config(components=set(MAP), max_depth=case["depth"]),
                "subcarriers": (torch.arange(k, dtype=torch.float64) - k // 2) * 30e3}
    if kind == "batch":
        freqs = [3.5e9, 6.0e9, 28.0e9, 39.0e9][:case["bands"]]
        scenes, leaves, weights = [], [], []
        for j, (boxes, side) in enumerate(((case["boxes_a"], case["side_a"]), (case["boxes_b"], case["side_b"]))):
            eps, sig, mat = _concrete_leaves(3.5) if case["grad"] else (None, None, None)
            layout, structures, rng = _town(case, 2 * seed + j, boxes, mat)
            txs = [make_transmitter(street_point(layout, rng, float(rng.uniform(5.0, 40.0)))) for _ in range(case["tx"])]
            if case["grad"]:
                for t in txs:
                    t.position = torch.as_tensor(t.position, dtype=torch.float32).clone().requires_grad_(True)
                leaves += [eps.requires_grad_(True), sig.requires_grad_(True), *(t.position for t in txs)]
                g = torch.Generator(device=device).manual_seed(2 * seed + j)
                weights.append(torch.rand((len(freqs), case["tx"], side, side), generator=g, device=device) + 0.5)
            scene = Scene(structures=structures, endpoints=[*txs, _grid(side, side, 400.0 / side)])
            compile_scene(scene, device)
            scenes.append(scene)
        return {"kind": kind, "scenes": scenes, "freqs": freqs, "leaves": leaves, "weights": weights,
                "config": Config(components=set(MAP), max_depth=case["depth"], return_field=False,
                                 ad_mode="vjp" if case["grad"] else "none")}
    if kind == "gradient":
        eps, sig, mat = _concrete_leaves(case["ghz"])
        scene, rng = _map_scene(case, seed, mat)
        tx = scene.transmitters[0]
        tx.position = torch.as_tensor(tx.position, dtype=torch.float32).clone().requires_grad_(True)
        moved = 1 + rng.choice(case["boxes"], size=min(case["moved"], case["boxes"]), replace=False)
        verts = []
        for b in sorted(int(x) for x in moved):
            st = scene.structures[b]
            st.geometry.vertices = st.vertices.detach().clone().requires_grad_(True)
            verts.append(st.geometry.vertices)
        # the measured map: free-space loss with 8 dB of shadowing
        ax = (torch.arange(case["rows"], dtype=torch.float64) - (case["rows"] - 1) / 2) * case["spacing"]
        ay = (torch.arange(case["cols"], dtype=torch.float64) - (case["cols"] - 1) / 2) * case["spacing"]
        p = tx.position.detach().double()
        d2 = (ay[:, None] - p[1]) ** 2 + (ax[None, :] - p[0]) ** 2 + (p[2] - 1.5) ** 2
        shadow = torch.from_numpy(rng.normal(-1.0, 0.8, size=tuple(d2.shape)))
        log_target = (2 * math.log10(C0 / (4 * math.pi * freq)) - torch.log10(d2) + shadow)[None].to(device)
        carrier = torch.tensor(freq, dtype=torch.float64, requires_grad=True)
        compile_scene(scene, device)
        return {"kind": kind, "scene": scene, "freq": carrier, "log_target": log_target,
                "leaves": [eps.requires_grad_(True), sig.requires_grad_(True), carrier, tx.position, *verts],
                "config": Config(components=set(MAP), max_depth=case["depth"], ad_mode="vjp", return_field=False)}
    if kind == "jvp":
        eps, sig, mat = _concrete_leaves(case["ghz"])
        layout, structures, rng = _town(case, seed, case["boxes"], mat)
        pos = torch.tensor(street_point(layout, rng, 25.0), dtype=torch.float32)
        grid = _grid(case["rows"], case["cols"], case["spacing"])
        direction = torch.from_numpy(rng.normal(size=3)).float()
        scene = Scene(structures=structures, endpoints=[make_transmitter(pos), grid])
        compile_scene(scene, device)
        return {"kind": kind, "scene": scene, "freq": freq, "pos": pos, "direction": direction,
                "config": Config(components=set(MAP), max_depth=case["depth"], ad_mode="jvp")}
    if kind == "replay":
        layout, structures, rng = _town(case, seed, case["boxes"])
        tx = torch.tensor([street_point(layout, rng, 25.0)], dtype=torch.float32, device=device)
        side, slots = case["side"], case["slots"]
        axis = (torch.arange(side, device=device, dtype=torch.float32) - (side - 1) / 2) * 2.0
        pts = torch.stack((axis.repeat_interleave(side), axis.repeat(side), torch.full((side * side,), 1.5, device=device)), 1)
        up = torch.tensor([[0.0, 0.0, 1.0]], device=device)
        sources = consumer.EndpointBatch(stable_ids=torch.zeros(slots, dtype=torch.int64, device=device),
                                         positions_m=tx.repeat(slots, 1), polarizations=up.repeat(slots, 1),
                                         powers_w=torch.ones(slots, device=device))
        heading = torch.from_numpy(rng.normal(size=(side * side, 3)) * [1.0, 1.0, 0.0]).float().to(device)
        step = torch.linspace(0.0, 0.4, slots, device=device).view(slots, 1, 1)
        ids = torch.arange(side * side, dtype=torch.int64, device=device)
        sinks = consumer.EndpointBatch(stable_ids=ids.repeat(slots),
                                       positions_m=(pts[None] + step * heading[None]).reshape(-1, 3).contiguous(),
                                       polarizations=up.repeat(slots * side * side, 1))
        scene = Scene(structures=structures, endpoints=[])
        compiled = compile_scene(scene, device)
        found = consumer.evaluate(compiled, consumer.PropagationRequest(
            sources=consumer.EndpointBatch(stable_ids=sources.stable_ids[:1], positions_m=tx, polarizations=up,
                                           powers_w=sources.powers_w[:1]),
            sinks=consumer.EndpointBatch(stable_ids=ids, positions_m=pts, polarizations=up.repeat(side * side, 1)),
            reference_frequency_hz=freq, components=frozenset({"los", "reflection"}), max_depth=case["depth"],
            response="scalar_transport", topology_mode="discover", ad_mode="none"))
        frozen = consumer.prepare_fixed_topology(found.paths.topology)
        if slots > 1:
            frozen = consumer.replicate_over_slots(frozen, slots, source_count=1, sink_count=side * side)
        table = _buffers(3 * slots * side * side, {"valid": ((), torch.bool), "coefficient": ((), torch.complex64),
                                                   "delay": ((), torch.float32), "length": ((), torch.float32)}, device)
        return {"kind": kind, "scene": scene, "compiled": compiled, "table": table, "request": consumer.FixedTopologyRequest(
            sources=sources, sinks=sinks, reference_frequency_hz=freq, topology=frozen, response="scalar_transport",
            ad_mode="none", slot_count=slots)}
    table, freqs = _cfr_inputs(case, seed, device)
    return {"kind": "cfr", "table": table, "freqs": freqs, "links": case["links"]}


def _buffers(capacity: int, columns: dict, device) -> dict:
    """A link simulator's path buffers of fixed capacity, which each call's table is copied into."""
    return {k: torch.zeros((capacity, *shape), dtype=dtype, device=device) for k, (shape, dtype) in columns.items()}


def _store(buffers: dict, **columns) -> dict:
    for k, v in columns.items():
        n = min(int(v.shape[0]), int(buffers[k].shape[0]))
        buffers[k][:n].copy_(v[:n])
    return buffers


def _two_ray_tx(seed: int) -> tuple:
    rng = np.random.default_rng(seed)
    return tuple(float(v) for v in (rng.uniform(-5, 5), rng.uniform(-5, 5), rng.uniform(8, 12)))


def _cfr_inputs(case: dict, seed: int, device):
    """Path columns of every link in canonical order: Poisson path counts,
    exponential excess delays (200 ns), complex normal gains."""
    g = torch.Generator(device=device).manual_seed(seed)
    count = torch.poisson(torch.full((case["links"],), case["mean_paths"], device=device), generator=g).long()
    rx = torch.arange(case["links"], device=device).repeat_interleave(count)
    n = int(rx.shape[0])
    delay = 1e-7 + torch.empty(n, device=device).exponential_(generator=g) * 2e-7
    re, im = (torch.randn(n, generator=g, device=device) * 1e-5 for _ in range(2))
    table = SimpleNamespace(tx_id=torch.zeros(n, dtype=torch.int32, device=device), rx_id=rx.to(torch.int32),
                            delay_s=delay, field_real=re, field_imag=im)
    freqs = (np.arange(case["subcarriers"]) - case["subcarriers"] // 2) * case["df_khz"] * 1e3
    return table, freqs


# ------------------------------------------------------------------ one pass
def run(s):
    kind = s["kind"]
    if kind == "map":
        r = solve(s["scene"], s["config"], reference_frequency_hz=s["freq"], precision=s["precision"])
        return {"gain": r.path_gain, "field": r.field, "power": r.component_power, "fields": r.component_fields}
    if kind == "export":
        r = solve(s["scene"], s["config"], reference_frequency_hz=s["freq"])
        p = r.paths
        return {"gain": r.path_gain, "field": r.field, "count": int(p.tx_id.shape[0]), **_store(
            s["table"], tx=p.tx_id, rx=p.rx_id, component=p.component_id, depth=p.depth, faces=p.primitive_sequence,
            delay=p.delay_s, coefficient=p.coefficient, positions=p.interaction_positions,
            normals=p.interaction_normals)}
    if kind == "links":
        r = paths_api.solve(s["scene"], s["config"], reference_frequency_hz=s["freq"])
        spectra = r.cfr(s["subcarriers"])
        per_path = [r.a[..., 0].reshape(-1, r.max_num_paths).T, r.tau.reshape(-1, r.max_num_paths).T]
        return {"count": r.num_paths, "cfr": spectra, **_store(s["table"], a=per_path[0], tau=per_path[1])}
    if kind == "batch":
        out = solve_batch(s["scenes"], s["config"], s["freqs"])
        maps = [o["path_gain"] for o in out]
        if not s["leaves"]:
            return maps
        loss = sum((m * w).sum() for m, w in zip(maps, s["weights"]))
        return {"maps": [m.detach() for m in maps], "grads": list(torch.autograd.grad(loss, s["leaves"]))}
    if kind == "gradient":
        r = solve(s["scene"], s["config"], reference_frequency_hz=s["freq"])
        hit = r.path_gain > 0
        d = torch.log10(r.path_gain[hit].double()) - s["log_target"][hit]
        loss = (d * d).mean()
        return {"loss": loss.detach(), "gain": r.path_gain.detach(), "grads": list(torch.autograd.grad(loss, s["leaves"]))}
    if kind == "jvp":
        tx = s["scene"].transmitters[0]
        with fwAD.dual_level():
            tx.position = fwAD.make_dual(s["pos"], s["direction"])
            r = solve(s["scene"], s["config"], reference_frequency_hz=s["freq"])
            gain, d_gain = fwAD.unpack_dual(r.path_gain)
            field, d_field = fwAD.unpack_dual(r.field)
            tx.position = s["pos"]
        return {"gain": gain, "d_gain": d_gain, "field": field, "d_field": d_field}
    if kind == "replay":
        r = consumer.reevaluate(s["compiled"], s["request"])
        p = r.paths
        return {"pairs": p.pair_offsets, **_store(s["table"], valid=r.row_valid, coefficient=p.transport.coefficient,
                                                  delay=p.geometry.delay_s, length=p.geometry.path_length_m)}
    return cfr(s["table"], s["freqs"], num_tx=1, num_rx=s["links"])


# ------------------------------------------------------------------ what a pass cannot do without
def work(case: dict) -> dict:
    """Bytes: the mesh (48 B a triangle, 12 or 12 + 2 k^2 + ... triangles a box)
    and the endpoints read once, the returned arrays written once.  Operations:
    one line-of-sight segment against log2(F) box pairs (about 60 operations
    each) and one field (about 200) per cell and transmitter; the passes' true
    work on top of that depends on what each receiver sees."""
    kind = case["kind"]
    if kind == "cfr":
        paths, out = case["links"] * case["mean_paths"], case["links"] * case["subcarriers"]
        return {"bytes": int(20 * paths + 8 * out), "flops": int(8 * paths * case["subcarriers"])}
    boxes = case.get("boxes", 0) or case.get("boxes_a", 0) + case.get("boxes_b", 0)
    faces = 2 + boxes * (60 if case.get("roofs") else 12)
    per_cell = 60 * max(1, math.ceil(math.log2(faces + 1))) + 200
    if kind in ("two_ray", "map"):
        cells, width = case["rows"] * case["cols"], 8 if case.get("precision") == "fp64" else 4
        out = cells * width * (3 + 3 * (4 if case.get("glass") else 3))
    elif kind == "batch":
        maps = case["tx"] * case["bands"]
        cells = maps * (case["side_a"] ** 2 + case["side_b"] ** 2)
        out = cells * (8 if case["grad"] else 4)
    elif kind == "gradient":
        cells = case["rows"] * case["cols"]
        out = cells * 12 + case["moved"] * 96
    elif kind == "jvp":
        cells = case["rows"] * case["cols"]
        out = cells * 24
    elif kind == "export":
        cells = case["rows"] * case["cols"]
        out = cells * (12 + 32 + 28 * case["depth"])
    elif kind == "links":
        cells = case["receivers"] * case["tx_elements"] * case["rx_elements"]
        out = cells * 8 * case["subcarriers"]
    else:
        cells = case["side"] ** 2 * case["slots"]
        out = cells * (12 + 17)
    return {"bytes": int(48 * faces + out), "flops": int(cells * per_cell)}


# ------------------------------------------------------------------ 64-bit values
def exact(case: dict, seed: int):
    """The two-ray field in closed form (image of the transmitter in the ground,
    slab Fresnel coefficients) and the CFR as its defining sum; the city cases
    need a whole ray tracer and have none."""
    if case["kind"] == "cfr":
        return _exact_cfr(case, seed)
    if case["kind"] == "two_ray":
        return _exact_two_ray(case, seed)
    return None


def _exact_cfr(case: dict, seed: int):
    device = torch.device("cuda", torch.cuda.current_device())
    table, freqs = _cfr_inputs(case, seed, device)
    f = torch.as_tensor(freqs, dtype=torch.float64, device=device)
    links, k = case["links"], case["subcarriers"]
    rx, tau = table.rx_id.long(), table.delay_s.double()
    first = torch.full((links,), math.inf, dtype=torch.float64, device=device).scatter_reduce(0, rx, tau, "amin")
    tau = tau - first[rx]
    a = torch.complex(table.field_real.double(), table.field_imag.double())
    out = torch.zeros((links, k), dtype=torch.complex128, device=device)
    chunk = max(1, (1 << 26) // k)
    for b in range(0, int(rx.shape[0]), chunk):
        e = slice(b, b + chunk)
        out.index_add_(0, rx[e], a[e, None] * torch.exp(-2j * math.pi * tau[e, None] * f[None, :]))
    return out.reshape(1, links, k)


def _exact_two_ray(case: dict, seed: int):
    freq = case["ghz"] * 1e9
    k = 2 * math.pi * freq / C0
    rows, cols, sp = case["rows"], case["cols"], case["spacing"]
    tx = np.array(_two_ray_tx(seed), dtype=np.float32).astype(np.float64)
    x = np.float32(-(rows - 1) / 2.0 * sp) + np.arange(rows, dtype=np.float32) * np.float32(sp)
    y = np.float32(-(cols - 1) / 2.0 * sp) + np.arange(cols, dtype=np.float32) * np.float32(sp)
    rx = np.stack([*np.meshgrid(x.astype(np.float64), y.astype(np.float64), indexing="ij"),
                   np.full((rows, cols), np.float64(np.float32(1.5)))], -1).transpose(1, 0, 2)
    ez = np.array([0.0, 0.0, 1.0])

    def unit(v):
        return v / np.linalg.norm(v, axis=-1, keepdims=True)

    def dot(u, v):
        return (u * v).sum(-1, keepdims=True)

    off = rx - tx
    d = np.linalg.norm(off, axis=-1)
    u = unit(off)
    z_t = ez - u * dot(u, ez)
    los = (z_t * z_t).sum(-1) * np.exp(-1j * k * d) / (2 * k * d)
    image = tx * [1.0, 1.0, -1.0]
    ray = rx - image
    length = np.linalg.norm(ray, axis=-1)
    out = unit(ray)
    inc = out * [1.0, 1.0, -1.0]
    cos = out[..., 2]
    eta = 5.24 - 1j * 0.0462 * case["ghz"] ** 0.7822 / (2 * math.pi * freq * EPS0)
    root = np.sqrt(eta - (1 - cos ** 2))
    phase = np.exp(-2j * root * 2 * math.pi * 10.0 * freq / C0)
    r_te, r_tm = (i * (1 - phase) / (1 - i * i * phase)
                  for i in ((cos - root) / (cos + root), (eta * cos - root) / (eta * cos + root)))
    s_axis = unit(np.cross(np.broadcast_to(ez, inc.shape), inc))
    p_in, p_out = np.cross(s_axis, inc), np.cross(s_axis, out)
    e0 = ez - inc * dot(inc, ez)
    e1 = s_axis * (r_te[..., None] * dot(s_axis, e0)) + p_out * (r_tm[..., None] * dot(p_in, e0))
    refl = (e1 * (ez - out * dot(out, ez))).sum(-1) * np.exp(-1j * k * length) / (2 * k * length)
    los, refl = los[None], refl[None]
    total = los + refl
    return {"gain": np.abs(total) ** 2, "field": total,
            "power": {"los": np.abs(los) ** 2, "reflection": np.abs(refl) ** 2, "diffraction": np.zeros(los.shape)},
            "fields": {"los": los, "reflection": refl, "diffraction": np.zeros(los.shape, dtype=complex)}}
