"""The work that a user of the framework has it do, as measurable cases.

A case names a robot (the seeded 7-joint chain, the same chain on a planar base, the 14-joint dual arm), an
environment (20 primitives, or a 200k-point cloud), a call of the public API and its size:

* ``state``     the reference's per-state call in a loop: ``cst.is_valid(q)``, one state of host memory each
* ``edge``      the reference's per-edge call in a loop: ``validator.checkMotion(s1, s2)``
* ``states``    ``is_valid_fast`` on a batch (FP32 with the FP64 recheck), with or without distances
* ``edges``     ``check_motion_fast`` on a batch of edges of uneven length
* ``plain``     ``is_valid_batch``: the FP64 method on a batch
* ``evaluate``  ``evaluate_batch``: FP64 constraint values and Jacobians, what the IK and SQP solvers call
* ``ik``        ``diff.ik_cost`` forward and backward: one gradient step of batched collision-aware IK
* ``traj``      ``diff.trajectory_cost`` forward and backward: one step of trajectory smoothing
* ``nearest``   ``CloudSDF.nearest``: exact FP64 nearest points (what ``KDTree`` runs)

The sizes of the listed cases are those of the repository's workloads and benchmark, and odd ones beside them.
"""
from __future__ import annotations

import math
import xml.etree.ElementTree as ET

import numpy as np
import torch

from plainmp_gb300 import diff, scenes
from plainmp_gb300 import workloads as W
from plainmp_gb300.motion_validator import BoxMotionValidator

WIDTH = 0.05  # resolution of the box motion validator, rad (and m for a planar base)
ROBOTS = {"chain7": W.chain7_robot, "planar": W.planar_chain7_robot, "dualarm": W.dualarm_robot}
DOF = {"chain7": 7, "planar": 10, "dualarm": 14}
SPHERES = {"chain7": 56, "planar": 56, "dualarm": 120}
PAIRS = {"chain7": 15, "planar": 15, "dualarm": 59}
CLOUD_POINTS = 200_000
CUTOFF = 0.1  # distances are reported up to here


def listed():
    return [
        # an OMPL planner's state-validity callback: one state a call, 32 calls in a row
        _case("state_chain7", "state", "chain7", "prims", 32),
        # its motion-validator callback on short tree extensions, 16 edges in a row
        _case("edge_dualarm", "edge", "dualarm", "cloud", 16, waypoints=16),
        # a roadmap planner's sample batch of ordinary size, with the distances
        _case("states_chain7_4096", "states", "chain7", "prims", 4096, distances=True),
        # an odd-sized batch of a mobile manipulator, in host memory
        _case("states_planar_1001_host", "states", "planar", "cloud", 1001, memory="host"),
        # the benchmark's batch: dual arm against the cloud, per-sphere distances
        _case("states_dualarm_65536", "states", "dualarm", "cloud", 65536, distances=True),
        # the largest batch, validity only: dense sampling of a workspace
        _case("states_dualarm_200003", "states", "dualarm", "cloud", 200003),
        # all edges of a roadmap: 1 to 120 waypoints each
        _case("edges_chain7_1024", "edges", "chain7", "prims", 1024, waypoints=120),
        # the FP64 method on a batch, where a caller wants the reference's arithmetic throughout
        _case("plain_chain7_4096", "plain", "chain7", "prims", 4096),
        # constraint values and Jacobians at the waypoints of a solver's trajectories
        _case("evaluate_planar_601", "evaluate", "planar", "cloud", 601),
        # one gradient step of 8,192 IK problems
        _case("ik_chain7_8192", "ik", "chain7", "prims", 8192),
        # one gradient step of 512 trajectories of 20 to 100 waypoints
        _case("traj_planar_512", "traj", "planar", "cloud", 512),
        # exact nearest points of map queries, near the cloud and far from it
        _case("nearest_100000", "nearest", "dualarm", "cloud", 100_000),
    ]


def _case(name, call, robot, env, n, distances=False, memory="device", waypoints=0, scene=0):
    c = {"call": call, "robot": robot, "env": env, "n": n, "distances": distances, "memory": memory,
         "waypoints": waypoints, "scene": scene}
    return c if name is None else dict(c, name=name)


def _log_size(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    call = rng.choice(["state", "edge", "states", "states", "states", "edges", "plain", "evaluate", "ik", "traj", "nearest"])
    robot, env = rng.choice([("chain7", "prims"), ("planar", "cloud"), ("planar", "prims"), ("dualarm", "cloud"), ("dualarm", "prims")])
    distances, memory, waypoints = False, "device", 0
    if call == "state":
        n = rng.randint(24, 48)
    elif call == "edge":
        n, waypoints = rng.randint(16, 24), rng.randint(4, 24)
    elif call == "states":
        distances, memory = rng.random() < 0.5, rng.choice(["device", "device", "host"])
        n = _log_size(rng, 33, 32768 if memory == "host" else 65536 if distances else 200003)
    elif call == "edges":
        n, waypoints = _log_size(rng, 24, 1024), rng.randint(8, 120)
    elif call == "plain":
        n = _log_size(rng, 33, 4096)
    elif call == "evaluate":
        n, memory = _log_size(rng, 1, 601), rng.choice(["device", "host"])
    elif call == "ik":
        robot, env = rng.choice(["chain7", "planar"]), "prims"
        n = _log_size(rng, 1, 8192)
    elif call == "traj":
        robot, env = rng.choice([("planar", "cloud"), ("chain7", "prims")])
        n = _log_size(rng, 1, 512)
    else:
        n = _log_size(rng, 1, 100_000)
        robot, env = "dualarm", "cloud"
    return _case(None, call, robot, env, n, distances, memory, waypoints, rng.randint(0, 3))


# ------------------------------------------------------------------------------------------------ inputs
def _scene(case):
    if case["env"] == "prims":
        return W.chain7_scene(case["scene"])
    return W.Scene(cloud=W.box_surface_cloud(CLOUD_POINTS, seed=case["scene"]))


def _configs(case, rng, n):
    q = rng.uniform(-math.pi, math.pi, size=(n, DOF[case["robot"]]))
    if case["robot"] == "planar":
        q[:, 7:9] = rng.uniform(-1.0, 1.0, size=(n, 2))
    return q


def _edges(case, rng, n):
    """Straight edges whose number of checked waypoints is uniform in 1..waypoints."""
    s1, to = _configs(case, rng, n), _configs(case, rng, n)
    d = to - s1
    length = (rng.integers(1, case["waypoints"] + 1, size=(n, 1)) - 1 + rng.uniform(0.25, 0.75, size=(n, 1))) * WIDTH
    return s1, s1 + d / np.abs(d).max(axis=1, keepdims=True) * length


def _numbers(case, seed):
    """The arrays that a pass reads, from the seed alone (NumPy, host memory)."""
    rng = np.random.default_rng([seed, case["n"], DOF[case["robot"]]])
    call, n = case["call"], case["n"]
    if call in ("edge", "edges"):
        return _edges(case, rng, n)
    if call == "ik":  # targets: the end link's pose at a random configuration near the start
        q = _configs(case, rng, n)
        star = q + rng.normal(0.0, 0.3, size=q.shape)
        robot = ROBOTS[case["robot"]]()
        links = _fk(robot, torch.from_numpy(star), False)
        quat, pos = links[robot.end_link]
        return q.astype(np.float32), torch.cat([pos, quat], dim=1).numpy().astype(np.float32)
    if call == "traj":  # straight lines between random endpoints with noise, stored back to back
        lens = np.random.default_rng([n, case["scene"]]).integers(20, 101, size=n)  # the case's, whatever the seed
        rows = []
        for length in lens:
            a, b = _configs(case, rng, 2)
            rows.append(a + (b - a) * np.linspace(0.0, 1.0, length)[:, None] + 0.05 * rng.standard_normal((length, a.shape[0])))
        return np.concatenate(rows).astype(np.float32), np.concatenate([[0], np.cumsum(lens)]).astype(np.int64)
    if call == "nearest":  # uniform in a cube around the cloud's: most beyond arm's reach of a surface
        return (np.array([0.6, 0.0, 0.8]) + rng.uniform(-1.25, 1.25, size=(n, 3)),)
    return (_configs(case, rng, n),)


def prepare(case, seed):
    robot, scene = ROBOTS[case["robot"]](), _scene(case)
    kin, cst, sdf = scenes.make_constraint(robot, scene)
    arrays = _numbers(case, seed)
    host = case["memory"] == "host" or case["call"] in ("state", "edge")
    data = arrays if host else tuple(torch.from_numpy(a).cuda() for a in arrays)
    state = {"call": case["call"], "distances": case["distances"], "kin": kin, "cst": cst, "sdf": sdf, "data": data, "link": robot.end_link}
    if case["call"] in ("edge", "edges"):
        state["validator"] = BoxMotionValidator(cst, [WIDTH] * DOF[case["robot"]])
    if case["call"] in ("ik", "traj"):
        state["data"] = (data[0].requires_grad_(True), data[1])
    return state


def run(state):
    call, cst, data = state["call"], state["cst"], state["data"]
    if call == "state":
        return np.array([cst.is_valid(q) for q in data[0]], dtype=np.uint8)
    if call == "edge":
        return np.array([state["validator"].checkMotion(a, b) for a, b in zip(*data)], dtype=np.uint8)
    if call == "states":
        return cst.is_valid_fast(data[0], distances=state["distances"])
    if call == "edges":
        return state["validator"].check_motion_fast(*data)
    if call == "plain":
        return cst.is_valid_batch(data[0])
    if call == "evaluate":
        return cst.evaluate_batch(data[0])
    if call == "nearest":
        return state["sdf"].nearest(data[0])
    q, other = data
    if call == "ik":
        cost = diff.ik_cost(cst, q, other, state["link"])
    else:
        cost = diff.trajectory_cost(cst, q, other)
    (grad,) = torch.autograd.grad(cost.sum(), q)
    return cost.detach(), grad


# ------------------------------------------------------------------------------------------------ work
def work(case):
    """Bytes: the arrays in and out once.  Operations: FK (about 120 per joint), the spheres' centres (18), one
    distance per sphere and primitive (25; one nearest point of a cloud counts as one primitive) and the group
    pairs' distances (10); a gradient doubles them."""
    n, dof, ns, pairs = case["n"], DOF[case["robot"]], SPHERES[case["robot"]], PAIRS[case["robot"]]
    prims = 20 if case["env"] == "prims" else 1
    each = 120 * dof + 18 * ns + 25 * ns * prims
    checked = each + 10 * pairs
    call = case["call"]
    if call in ("edge", "edges"):
        return {"bytes": n * (16 * dof + 1), "flops": n * (case["waypoints"] + 1) / 2 * checked}
    if call == "evaluate":
        return {"bytes": n * (8 * dof + 16 * (1 + dof)), "flops": 2 * n * checked}
    if call == "ik":
        return {"bytes": n * (8 * dof + 32), "flops": 2 * n * each}
    if call == "traj":
        return {"bytes": n * (60 * 8 * dof + 12), "flops": 2 * n * 60 * each}
    if call == "nearest":
        return {"bytes": n * 56, "flops": n * 25}
    return {"bytes": n * (8 * dof + 1 + (4 * ns if case["distances"] else 0)), "flops": n * checked}


# ------------------------------------------------------------------------------------------------ 64 bits
def _qmul(a, b):
    ax, ay, az, aw = a.unbind(-1)
    bx, by, bz, bw = b.unbind(-1)
    return torch.stack([aw * bx + ax * bw + ay * bz - az * by, aw * by + ay * bw + az * bx - ax * bz,
                        aw * bz + az * bw + ax * by - ay * bx, aw * bw - ax * bx - ay * by - az * bz], dim=-1)


def _qrot(q, v):
    u = q[..., :3]
    uv = 2.0 * torch.linalg.cross(u, v)
    return v + q[..., 3:] * uv + torch.linalg.cross(u, uv)


def _sin_cos(x, taylor):
    """The reference's polynomials for states on a fixed base (half angles, within half a turn), else sin and cos."""
    if not taylor:
        return torch.sin(x), torch.cos(x)
    s = sum((-1) ** k * x ** (2 * k + 1) / math.factorial(2 * k + 1) for k in range(5))
    return s, sum((-1) ** k * x ** (2 * k) / math.factorial(2 * k) for k in range(5))


def _fk(robot, q, taylor):
    """World (quaternion, position) of every link, (n, 4) and (n, 3)."""
    n = q.shape[0]
    row = lambda v: torch.tensor(v, dtype=q.dtype, device=q.device).expand(n, len(v))  # noqa: E731
    pose = {}
    joints = {j.find("child").get("link"): j for j in ET.fromstring(robot.urdf).findall("joint")}

    def link(name):
        if name in pose:
            return pose[name]
        if name not in joints:
            if robot.base_type == "PLANAR":
                s, c = torch.sin(q[:, -1] / 2), torch.cos(q[:, -1] / 2)
                pose[name] = (torch.stack([0 * s, 0 * s, s, c], 1), torch.stack([q[:, -3], q[:, -2], 0 * s], 1))
            else:
                pose[name] = (row([0.0, 0.0, 0.0, 1.0]), row([0.0, 0.0, 0.0]))
            return pose[name]
        j = joints[name]
        pq, pt = link(j.find("parent").get("link"))
        t = pt + _qrot(pq, row([float(v) for v in j.find("origin").get("xyz").split()]))
        if j.get("type") == "revolute":
            axis = np.array([float(v) for v in j.find("axis").get("xyz").split()])
            s, c = _sin_cos(q[:, robot.control_joints.index(j.get("name"))] / 2, taylor)
            pq = _qmul(pq, torch.cat([s[:, None] * row(list(axis / np.linalg.norm(axis))), c[:, None]], dim=1))
        pose[name] = (pq, t)
        return pose[name]

    for x in ET.fromstring(robot.urdf).findall("link"):
        link(x.get("name"))
    return pose


def _farthest_first(p):
    """Order of one link's spheres in the constraint: the last first, then always the farthest from those taken."""
    left, order = list(range(len(p) - 1, 0 - 1, -1)), []
    order.append(left.pop(0))
    while left:
        far = [min(np.linalg.norm(p[i] - p[j]) for j in order) for i in left]
        order.append(left.pop(int(np.argmax(far))))
    return order


def _spheres(robot):
    """Per link: its name, centres (m, 3) and radii (m,), in the order of the constraint's spheres."""
    out = []
    for k, s in enumerate(robot.spheres):
        p, r = s.relative_positions.T, s.radii
        for _ in range(len(robot.spheres) - k):  # the order is taken again with every later link
            o = _farthest_first(p)
            p, r = p[o], r[o]
        out.append((s.parent_link_name, p, r))
    return out


def _centres(robot, links, like):
    c, r = [], []
    for name, p, radii in _spheres(robot):
        quat, pos = links[name]
        p = torch.from_numpy(np.ascontiguousarray(p)).to(like)
        c.append(_qrot(quat[:, None, :].expand(-1, len(radii), 4), p[None].expand(len(quat), -1, 3)) + pos[:, None])
        r.append(torch.from_numpy(radii).to(like))
    return torch.cat(c, dim=1), torch.cat(r)


def _primitive(p, c):
    """Signed distance of points c (..., 3) to one primitive."""
    d = c - torch.from_numpy(p.position).to(c)
    if p.kind == "sphere":
        return d.norm(dim=-1) - p.size[0]
    d = d @ torch.from_numpy(p.rotation).to(c)
    if p.kind == "box":
        s = d.abs() - torch.tensor(p.size, dtype=c.dtype, device=c.device) / 2
    else:
        s = torch.stack([d[..., :2].norm(dim=-1) - p.size[0], d[..., 2].abs() - p.size[1] / 2], dim=-1)
    out = s.clamp(min=0)
    far = (out * out).sum(-1)
    far = torch.where(far > 0, far, torch.ones_like(far)).sqrt() * (far > 0)
    return far + s.max(dim=-1).values.clamp(max=0)


def _nearest_of(points, queries, chunk=40_000_000):
    """Index of the nearest point of each query, by trying every point."""
    idx = []
    step = max(1, chunk // max(1, len(points)))
    for q in queries.split(step):
        d = sum((q[:, None, a] - points[None, :, a]) ** 2 for a in range(3))
        idx.append(d.argmin(dim=1))
    return torch.cat(idx)


def _nearest_within(points, queries, reach):
    """Index of the nearest point of each query where one lies within reach, else -1 (or a point farther away)."""
    idx = torch.full((len(queries),), -1, dtype=torch.long, device=queries.device)
    pv, qv = torch.floor(points / reach).long(), torch.floor(queries / reach).long()
    lo, hi = pv.min(0).values - 1, pv.max(0).values + 1
    near = torch.nonzero(((qv >= lo) & (qv <= hi)).all(1))[:, 0]
    cells, member = torch.unique(qv[near], dim=0, return_inverse=True)
    order = torch.argsort(member)
    counts = torch.bincount(member, minlength=len(cells)).tolist() if len(cells) else []
    for cell, rows in zip(cells, order.split(counts)):
        cand = torch.nonzero(((pv - cell).abs() <= 1).all(1))[:, 0]
        if len(cand):
            rows = near[rows]
            idx[rows] = cand[_nearest_of(points[cand], queries[rows])]
    return idx


def _distances(case, scene, c, r, limit):
    """Per sphere: the least signed distance over the environment (n, spheres), at most limit."""
    if case["env"] == "prims":
        d = torch.stack([_primitive(p, c) for p in scene.primitives]).min(dim=0).values - r
        return d.clamp(max=limit)
    points = torch.from_numpy(scene.cloud).to(c)
    flat = c.reshape(-1, 3)
    with torch.no_grad():
        idx = _nearest_within(points, flat, limit + float(r.max()))
    d = (flat - points[idx.clamp(min=0)]).norm(dim=-1)
    d = torch.where(idx >= 0, d, torch.full_like(d, math.inf)).reshape(c.shape[:2]) - r
    return d.clamp(max=limit)


def _self_distance(robot, c, r):
    """Least distance over the sphere pairs of the self-collision pairs, at most the cutoff."""
    at, begin = {}, 0
    for name, _, radii in _spheres(robot):
        at[name] = slice(begin, begin + len(radii))
        begin += len(radii)
    best = torch.full((len(c),), CUTOFF, dtype=c.dtype, device=c.device)
    for a, b in robot.self_pairs:
        d = (c[:, at[a], None] - c[:, None, at[b]]).norm(dim=-1) - (r[at[a], None] + r[None, at[b]])
        best = torch.minimum(best, d.flatten(1).min(dim=1).values)
    return best


def exact(case, seed):
    call = case["call"]
    if call in ("state", "edge", "edges", "plain") or (call == "states" and not case["distances"]):
        return None  # validity bytes: they stay equal
    robot, scene = ROBOTS[case["robot"]](), _scene(case)
    data = [torch.from_numpy(a).cuda() for a in _numbers(case, seed)]
    if call == "nearest":
        points = torch.from_numpy(scene.cloud).to(data[0])
        near = points[_nearest_of(points, data[0])]
        return [((near - data[0]) ** 2).sum(1), near]
    q = data[0].double()
    if call == "states":
        c, r = _centres(robot, _fk(robot, q, robot.base_type == "FIXED"), q)
        return [None, _distances(case, scene, c, r, CUTOFF)]
    q.requires_grad_(True)
    links = _fk(robot, q, False)
    c, r = _centres(robot, links, q)
    if call == "evaluate":
        rows = [_distances(case, scene, c, r, CUTOFF).min(dim=1).values, _self_distance(robot, c, r)]
        jac = [torch.autograd.grad(v.sum(), q, retain_graph=True)[0] for v in rows]
        return [torch.stack([v.detach() for v in rows], dim=1), torch.stack(jac, dim=1)]
    margin = 0.02 if call == "ik" else 0.03  # the costs' default margins
    hinge = ((margin - _distances(case, scene, c, r, margin)) ** 2).sum(dim=1)
    if call == "ik":
        quat, pos = links[robot.end_link]
        target = data[1].double()
        e = _qmul(target[:, 3:] * target.new_tensor([-1.0, -1.0, -1.0, 1.0]), quat)
        v = e[:, :3].norm(dim=1)
        angle = 2.0 * torch.atan2(v, e[:, 3].abs())
        cost = ((pos - target[:, :3]) ** 2).sum(dim=1) + 0.1 * angle ** 2 + hinge
    else:
        off = data[1]
        which = torch.repeat_interleave(torch.arange(len(off) - 1, device=q.device), off[1:] - off[:-1])
        inner = which[2:] == which[:-2]
        acc = ((q[2:] - 2.0 * q[1:-1] + q[:-2]) ** 2).sum(dim=1) * inner
        cost = torch.zeros(len(off) - 1, dtype=q.dtype, device=q.device).index_add(0, which, hinge).index_add(0, which[1:-1], acc)
    (grad,) = torch.autograd.grad(cost.sum(), q)
    return [cost.detach(), grad]
