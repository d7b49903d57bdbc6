"""Performance cases of the framework: what its users run, through the public Python entry points.

A case is a dict of plain values; `kind` names the path:

  fluid     a fluid without particles advanced by `steps` steps, then read with get_fluid_fields, as a program that
            writes a field file every so many steps does (in single precision unless the storage is double)
  beads     beads coupled to the fluid, `steps` coupled steps: begin_step, the bead forces, execute, the leapfrog;
            device arrays with BeadDynamics, or host arrays with the program's own leapfrog
  replicas  a ReplicaBatch advanced by `steps` steps, its beads and temperatures read back
  steady    a steady obstacle channel started from given fields and solved for `steps` steps, its fields read
  unet      the warm start's network on a batch of channels: the prediction, or a training step's gradients
  conv      one convolution layer of that network, forward and backward
"""
import importlib.util
import math
import os
import sys

import numpy as np
import torch
import torch.utils.checkpoint

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
BOLTZ = 6.02214076e23*1.380649e-23/1000.0
STORAGE_BYTES = {'double': 8, 'single': 4, 'half': 2, 'bfloat16': 2}


def package():
    """The framework, imported as lbm_b200 (its folder's name is not an identifier)."""
    if 'lbm_b200' not in sys.modules:
        folder = os.path.join(ROOT, 'openmm-lbm_b200')
        spec = importlib.util.spec_from_file_location('lbm_b200', os.path.join(folder, '__init__.py'),
                                                      submodule_search_locations=[folder])
        module = importlib.util.module_from_spec(spec)
        sys.modules['lbm_b200'] = module
        spec.loader.exec_module(module)
    return sys.modules['lbm_b200']


def warmstart():
    package()
    from lbm_b200 import warmstart as module
    return module


def fluid(name, nx, ny, nz, precision, steps, walls='none', fluctuations=False, tau=0.6):
    return {'name': name, 'kind': 'fluid', 'nx': nx, 'ny': ny, 'nz': nz, 'precision': precision, 'steps': steps,
            'walls': walls, 'fluctuations': fluctuations, 'tau': tau}


def beads(name, n, chains, length, precision, steps, stencil, drag, arrays='device', fluctuations=True):
    return {'name': name, 'kind': 'beads', 'n': n, 'chains': chains, 'length': length, 'precision': precision,
            'steps': steps, 'stencil': stencil, 'drag': drag, 'arrays': arrays, 'fluctuations': fluctuations}


def listed():
    return [
        # A small periodic fluid: a step is a few launches and little else.
        fluid('fluid_32_f32', 32, 32, 32, 'single', 200),
        # The bench's fluid without particles, at an edge whose fields are still read often.
        fluid('fluid_192_f32', 192, 192, 192, 'single', 200),
        # The precision study's channel in 16-bit storage, on the sample that its profiles use.
        fluid('channel_f16', 256, 256, 128, 'half', 400, walls='channel', tau=0.55),
        # A ragged channel in the other 16-bit type: no edge divides a tile, rows are not a multiple of 4 nodes.
        fluid('channel_bf16_ragged', 150, 93, 67, 'bfloat16', 300, walls='channel', tau=0.7),
        # A duct with regularized walls between open faces in double precision, as the reference's mixed and double
        # platforms store it; fluctuating, so that every random number path of the walls and faces is on.
        fluid('duct_f64', 95, 64, 61, 'double', 100, walls='duct', fluctuations=True, tau=0.8),
        # The particle channel that the parity tests run: 64 particles, host arrays in double precision.
        beads('beads_32_f64', 32, 1, 64, 'double', 50, 'trilinear', 'explicit', arrays='host', fluctuations=False),
        # The scale configuration's density of bead-spring chains, on an eighth of it and in full.
        beads('beads_128_f32', 128, 64, 100, 'single', 25, 'keys', 'centered'),
        beads('beads_256_f32', 256, 512, 100, 'single', 20, 'keys', 'centered'),
        # Many uneven replicas with their beads, in runs of the bench's ten steps.
        {'name': 'replicas_96', 'kind': 'replicas', 'replicas': 96, 'low': 16, 'high': 64, 'steps': 40},
        # The obstacle channel of the learned warm start: a stretch of the steady solve from predicted fields.
        {'name': 'steady_channel', 'kind': 'steady', 'nx': 128, 'ny': 64, 'nz': 64, 'steps': 400},
        # Its network: the prediction of one channel, and the gradients of a training batch.
        {'name': 'unet_predict', 'kind': 'unet', 'nx': 128, 'ny': 64, 'nz': 64, 'batch': 1, 'train': False},
        {'name': 'unet_train', 'kind': 'unet', 'nx': 128, 'ny': 64, 'nz': 64, 'batch': 2, 'train': True},
    ]


def log_int(rng, low, high):
    return int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))


def draw(rng):
    kind = rng.choice(['fluid', 'fluid', 'fluid', 'beads', 'beads', 'replicas', 'steady', 'unet', 'conv', 'conv'])
    if kind == 'fluid':
        nodes = log_int(rng, 12**3, 190**3)
        aspect = [rng.uniform(0.6, 1.6) for _ in range(3)]
        scale = (nodes/(aspect[0]*aspect[1]*aspect[2]))**(1/3)
        nx, ny, nz = (max(8, int(round(scale*a))) for a in aspect)
        if rng.random() < 0.5:
            nx = max(8, nx//8*8)
        precision = rng.choice(['single', 'single', 'half', 'bfloat16', 'double'])
        walls = rng.choice(['none', 'none', 'channel', 'duct'])
        fluctuations = rng.random() < 0.4
        steps = max(20, min(200, int(4e8/(nx*ny*nz))))
        c = fluid('', nx, ny, nz, precision, steps, walls, fluctuations, round(rng.uniform(0.55, 1.1), 3))
    elif kind == 'beads':
        n = log_int(rng, 24, 160)
        chains = max(1, int(round(n**3*rng.uniform(0.5, 3.0)*1e-3/40)))
        stencil = rng.choice(['nearest', 'trilinear', 'threepoint', 'keys'])
        arrays = rng.choice(['device', 'device', 'host'])
        c = beads('', n, chains, 40, rng.choice(['single', 'single', 'double']), 20, stencil,
                  rng.choice(['explicit', 'centered']), arrays, rng.random() < 0.7)
    elif kind == 'replicas':
        low = log_int(rng, 8, 24)
        c = {'kind': 'replicas', 'replicas': log_int(rng, 4, 96), 'low': low, 'high': low + log_int(rng, 4, 36),
             'steps': rng.choice([20, 35, 40])}
    elif kind == 'steady':
        c = {'kind': 'steady', 'nx': log_int(rng, 64, 160), 'ny': log_int(rng, 32, 64), 'nz': log_int(rng, 32, 64),
             'steps': rng.choice([100, 200, 400])}
    elif kind == 'unet':
        train = rng.random() < 0.5
        c = {'kind': 'unet', 'nx': 8*rng.randint(6, 16), 'ny': 8*rng.randint(3, 8), 'nz': 8*rng.randint(3, 8),
             'batch': rng.randint(1, 2), 'train': train}
    else:
        cin, cout = rng.choice([(16, 16), (16, 32), (32, 32), (32, 64), (48, 16), (64, 64), (96, 32), (64, 160),
                                (160, 160), (224, 64)])
        voxels = log_int(rng, 500, min(500000, 40000000//(cin + cout)))
        d, h = (max(3, int(round(voxels**(1/3)*rng.uniform(0.6, 1.3)))) for _ in range(2))
        c = {'kind': 'conv', 'batch': rng.randint(1, 2), 'd': d, 'h': h, 'w': max(3, voxels//(d*h)), 'cin': cin,
             'cout': cout, 'relu': rng.random() < 0.8}
    c.pop('name', None)
    return c


# ---------------------------------------------------------------------------------------------------------------
# Inputs.
# ---------------------------------------------------------------------------------------------------------------

def generator(seed):
    g = torch.Generator(device='cuda')
    g.manual_seed(seed)
    return g


def smooth_fields(nx, ny, nz, seed, amplitude=0.03):
    """Density [N] and velocity [N][3] of a developed flow: a few long waves per component, float64 on the device."""
    g = generator(seed)
    x, y, z = (torch.arange(n, device='cuda', dtype=torch.float64)*(2*math.pi/n) for n in (nx, ny, nz))
    out = []
    for _ in range(4):
        total = torch.zeros((nz, ny, nx), device='cuda', dtype=torch.float64)
        for k in range(3):
            p = torch.rand(6, device='cuda', dtype=torch.float64, generator=g)
            wx, wy, wz = (torch.sin((k + 1)*t + 2*math.pi*p[i]) for i, t in enumerate((x, y, z)))
            total += (p[3]*wx[None, None, :] + p[4]*wy[None, :, None] + p[5]*wz[:, None, None])/(3*(k + 1))
        out.append(total.reshape(-1))
    density = 1.0 + 0.002*out[3]
    return density, (amplitude*torch.stack(out[:3], dim=1)).contiguous()


def solid_nodes(case):
    nx, ny, nz = case['nx'], case['ny'], case['nz']
    if case['walls'] == 'channel':
        plane = np.arange(nx*ny, dtype=np.int64)
        return np.concatenate([plane, plane + nx*ny*(nz - 1)])
    if case['walls'] == 'duct':
        solid = np.zeros((nz, ny, nx), dtype=bool)
        solid[0], solid[-1], solid[:, 0], solid[:, -1] = True, True, True, True
        return np.nonzero(solid.ravel())[0]
    return []


def fluid_lattice(case, seed):
    lbm = package()
    force = lbm.LBMForce()
    nx, ny, nz = case['nx'], case['ny'], case['nz']
    force.setGridSize(nx, ny, nz)
    force.setFluidDensity(1.0)
    force.setKinematicViscosity((case['tau'] - 0.5)/3.0)
    force.setFluidFluctuations(case['fluctuations'])
    force.setTemperature(1e-5/BOLTZ if case['fluctuations'] else 0.0)
    force.setRandomNumberSeed(1 + seed % 1000003)
    force.setFluidMomentumRemovalFrequency(1 if case['walls'] == 'none' else 0)
    if case['walls'] == 'channel':
        force.setBodyAcceleration((5e-7, 0.0, 0.0))
    if case['walls'] == 'duct':
        force.setWallScheme(force.Regularized)
        force.setFaceBoundary(force.XMin, force.Velocity)
        force.setFaceVelocity(force.XMin, (0.02, 0.0, 0.0))
        # A fluctuating fluid is not kept at equilibrium by a Density face.
        force.setFaceBoundary(force.XMax, force.DensityVelocity if case['fluctuations'] else force.Density)
        force.setFaceDensity(force.XMax, 1.0)
        if case['fluctuations']:
            force.setFaceVelocity(force.XMax, (0.02, 0.0, 0.0))
    return force.latticeParameters(np.array([nx, ny, nz], dtype=float), 1.0, np.ones(1))


def prepare_fluid(case, seed):
    lbm = package()
    kernel = lbm.B200Kernel(fluid_lattice(case, seed), [], solid_nodes(case), case['precision'])
    density, velocity = smooth_fields(case['nx'], case['ny'], case['nz'], seed,
                                      0.005 if case['walls'] == 'duct' else 0.03)
    kernel.set_fluid_equilibrium(density, velocity, strain=False)
    return {'kernel': kernel, 'step': 0}


def fields(kernel, precision):
    """The fields as a file of the storage's precision takes them."""
    density, velocity = (torch.from_numpy(a) for a in kernel.get_fluid_fields())
    if precision == 'double':
        return {'density': density, 'velocity': velocity}
    return {'density': density.float(), 'velocity': velocity.float()}


def run_fluid(case, s):
    kernel, step = s['kernel'], s['step']
    for i in range(step, step + case['steps']):
        kernel.begin_step(i)
        kernel.execute(i)
    s['step'] = step + case['steps']
    return fields(kernel, case['precision'])


def chain_positions(case, seed):
    """Seeded random-walk chains, or, for one chain, separate particles off the walls.  An even lattice with chains by
    the eight repeats the chains of a box of half its edge in its eight octants."""
    lbm = package()
    n, chains, length = case['n'], case['chains'], case['length']
    if chains == 1:
        rng = np.random.default_rng(seed)
        p = np.column_stack([rng.uniform(0, n, length), rng.uniform(0, n, length), rng.uniform(2, n - 3, length)])
        return p, np.zeros((0, 2), dtype=np.int32)
    if n % 2 == 0 and n >= 192 and chains % 8 == 0:
        p, bonds = lbm.random_walk_chains(chains//8, length, (n//2,)*3, seed)
        corners = [(i, j, k) for i in (0, 1) for j in (0, 1) for k in (0, 1)]
        return (np.concatenate([p + np.array(c)*(n//2) for c in corners]),
                np.concatenate([bonds + i*len(p) for i in range(8)]))
    return lbm.random_walk_chains(chains, length, (n,)*3, seed)


def prepare_beads(case, seed):
    lbm = package()
    n, kT = case['n'], 1e-4
    positions, bonds = chain_positions(case, seed)
    count = len(positions)
    channel = case['chains'] == 1
    force = lbm.LBMForce()
    force.setGridSize(n, n, n)
    force.setFluidDensity(1.0)
    force.setKinematicViscosity((0.8 - 0.5)/3.0 if channel else (0.6 - 0.5)/3.0)
    force.setFluidFluctuations(case['fluctuations'])
    force.setTemperature(kT/BOLTZ if case['fluctuations'] else 0.0)
    force.setRandomNumberSeed(1 + seed % 1000003)
    force.setInterpolationStencil({'nearest': force.NearestNode, 'trilinear': force.Trilinear,
                                   'threepoint': force.ThreePoint, 'keys': force.Keys}[case['stencil']])
    force.setDragScheme(force.Centered if case['drag'] == 'centered' else force.Explicit)
    force.setFriction(0.5 if channel or case['drag'] == 'explicit' else 1.0)
    solid = []
    if channel:
        force.setFluidMomentumRemovalFrequency(0)
        force.setBodyAcceleration((1e-6, 0.0, 0.0))
        plane = np.arange(n*n, dtype=np.int64)
        solid = np.concatenate([plane, plane + n*n*(n - 1)])
    for i in range(count):
        force.addParticle(i)
    masses = np.ones(count)
    lattice = force.latticeParameters(np.array([n, n, n], dtype=float), 1.0, masses)
    rng = np.random.default_rng(seed + 1)
    velocities = rng.normal(size=(count, 3))*math.sqrt(kT)
    if case['arrays'] == 'host':
        kernel = lbm.B200Kernel(lattice, masses, solid, case['precision'])
        return {'kernel': kernel, 'step': 0, 'pos': positions.copy(), 'vel': velocities, 'frc': np.zeros((count, 3))}
    stream = torch.cuda.Stream()
    kernel = lbm.B200Kernel(lattice, masses, solid, case['precision'], stream=stream.cuda_stream)
    md = lbm.BeadDynamics(masses, (n,)*3, bonds, k=100.0*kT, r0=1.0, pair='wca', sigma=1.0, epsilon=kT,
                          cutoff=2.0**(1/6))
    pos = torch.tensor(positions, device='cuda', dtype=torch.float64)
    vel = torch.tensor(velocities, device='cuda', dtype=torch.float64)
    return {'kernel': kernel, 'md': md, 'stream': stream, 'step': 0, 'pos': pos, 'vel': vel,
            'frc': torch.zeros_like(pos)}


def run_beads(case, s):
    kernel, pos, vel, frc, first = s['kernel'], s['pos'], s['vel'], s['frc'], s['step']
    s['step'] = first + case['steps']
    if case['arrays'] == 'host':
        for i in range(first, first + case['steps']):
            kernel.begin_step(i, pos, vel, frc)
            frc[:] = 0.0
            kernel.execute(i, pos, vel, frc)
            vel += frc
            pos += vel
        if case['precision'] == 'double':
            return {'positions': pos, 'velocities': vel, 'forces': frc}
        return {'positions': pos.astype(np.float32), 'velocities': vel.astype(np.float32),
                'forces': frc.astype(np.float32)}
    md, stream = s['md'], s['stream']
    with torch.cuda.stream(stream):
        for i in range(first, first + case['steps']):
            kernel.begin_step(i, pos, vel, frc)
            md.compute_forces(pos, frc, stream.cuda_stream)
            kernel.execute(i, pos, vel, frc)
            md.integrate(1.0, pos, vel, frc, stream.cuda_stream)
        if case['precision'] == 'double':
            return {'positions': pos, 'velocities': vel, 'forces': frc}
        return {'positions': pos.float(), 'velocities': vel.float(), 'forces': frc.float()}


def replica_sizes(case):
    """The edges and bead counts of the replicas: the case's own, the same for every seed of its inputs."""
    rng = np.random.Generator(np.random.PCG64(2026))
    sizes = rng.integers(case['low'], case['high'] + 1, case['replicas'])
    beads = np.minimum(rng.integers(20, 201, case['replicas']), (sizes//2)**3//2)
    return sizes, beads


def prepare_replicas(case, seed):
    lbm = package()
    kT = 1e-4
    sizes, counts = replica_sizes(case)
    rng = np.random.default_rng(seed)
    lattices, positions = [], []
    for r, (n, b) in enumerate(zip(sizes, counts)):
        n, b = int(n), int(b)
        force = lbm.LBMForce()
        force.setGridSize(n, n, n)
        force.setFluidDensity(1.0)
        force.setKinematicViscosity((0.7 - 0.5)/3.0)
        force.setFluidFluctuations(True)
        force.setTemperature(kT/BOLTZ)
        force.setRandomNumberSeed(1 + (seed + 7919*r) % 1000003)
        force.setInterpolationStencil(force.ThreePoint)
        force.setDragScheme(force.Explicit)
        force.setFriction(0.8)
        for i in range(b):
            force.addParticle(i)
        lattices.append(force.latticeParameters(np.array([n, n, n], dtype=float), 1.0, np.ones(b)))
        # Random sites of a grid of spacing 2, shaken: no two beads closer than the Lennard-Jones diameter.
        site = rng.permutation((n//2)**3)[:b]
        m = n//2
        grid = np.stack([site % m, site//m % m, site//(m*m)], axis=1)*2.0
        positions.append(grid + rng.uniform(0, 1, (b, 3)))
    total = int(counts.sum())
    batch = lbm.ReplicaBatch(lattices, counts, np.ones(total), np.concatenate(positions),
                             pair=('lj', 1.0, kT, 2.5), precision='single')
    batch.autotune(10)
    return {'batch': batch}


def run_replicas(case, s):
    batch = s['batch']
    batch.step(case['steps'])
    positions, velocities = batch.particles_state()
    fluid_kT, bead_kT = batch.temperatures()
    return {'positions': positions.astype(np.float32), 'velocities': velocities.astype(np.float32),
            'fluid_kT': fluid_kT.astype(np.float32), 'bead_kT': bead_kT.astype(np.float32)}


def prepare_steady(case, seed):
    ws = warmstart()
    shape = (case['nx'], case['ny'], case['nz'])
    edge = min(shape[1:])
    solid = ws.obstacle_mask(seed, shape, radius=(edge/16, edge/6.4))
    kernel = ws.channel_kernel(solid, shape)
    # A prediction: the inlet's plug flow with long waves on it, at rest inside the obstacles.
    density, velocity = smooth_fields(*shape, seed, 0.005)
    open_ = torch.as_tensor(~solid.reshape(-1, 1), device='cuda')
    velocity = velocity + torch.tensor([0.02, 0.0, 0.0], device='cuda', dtype=torch.float64)
    return {'kernel': kernel, 'step': 0, 'density': density, 'velocity': (velocity*open_).contiguous()}


def run_steady(case, s):
    kernel = s['kernel']
    kernel.set_fluid_equilibrium(s['density'], s['velocity'])
    taken, _ = kernel.solve_steady(s['step'], 100, 1e-6, case['steps'])
    s['step'] += taken
    return dict(fields(kernel, 'single'), steps=taken)


def prepare_unet(case, seed):
    ws = warmstart()
    shape = (case['nx'], case['ny'], case['nz'])
    net = ws.load_network(os.path.join(ROOT, 'openmm-lbm_b200', 'warmstart_net', 'weights.pt'))
    masks = [torch.as_tensor(ws.obstacle_mask(seed + 31*i, shape, radius=(3.0, 8.0)), device='cuda')
             for i in range(case['batch'])]
    target = torch.randn((case['batch'], 4, shape[2], shape[1], shape[0]), device='cuda', generator=generator(seed))
    return {'net': net, 'masks': masks, 'target': target}


def run_unet(case, s):
    ws = warmstart()
    net = s['net']
    if not case['train']:
        with torch.no_grad():
            return net(ws.network_input(s['masks']))
    # The loss of warmstart.train() and its gradients.
    pred = net(ws.network_input(s['masks'])).float()
    open_ = torch.stack([~m for m in s['masks']]).unsqueeze(1).float()
    loss = (((pred - s['target'])**2)*open_).sum()/(open_.sum()*4)
    net.zero_grad()
    loss.backward()
    return {'loss': loss.detach(), 'weights': [p.grad for p in net.weights], 'biases': [p.grad for p in net.biases]}


def conv_inputs(case, seed):
    g = generator(seed)
    b, d, h, w, cin, cout = (case[k] for k in ('batch', 'd', 'h', 'w', 'cin', 'cout'))

    def volume(c):
        t = torch.randn((b, c, d, h, w), device='cuda', generator=g)
        return t.to(torch.bfloat16).contiguous(memory_format=torch.channels_last_3d)

    # The input of a layer is another layer's ReLU output.
    x, dy = volume(cin).clamp_(min=0), volume(cout)
    weight = (torch.randn((cout, 27, cin), device='cuda', generator=g)*(2.0/(27*cin))**0.5).to(torch.bfloat16).float()
    return x, weight, torch.randn(cout, device='cuda', generator=g)*0.1, dy


def prepare_conv(case, seed):
    x, weight, bias, dy = conv_inputs(case, seed)
    return {'x': x.requires_grad_(True), 'weight': weight.requires_grad_(True), 'bias': bias.requires_grad_(True),
            'dy': dy}


def run_conv(case, s):
    y = warmstart().Conv3dFunction.apply(s['x'], s['weight'], s['bias'], case['relu'])
    dx, dw, db = torch.autograd.grad(y, (s['x'], s['weight'], s['bias']), s['dy'])
    return {'y': y.detach(), 'dx': dx, 'dw': dw, 'db': db}


PATHS = {'fluid': (prepare_fluid, run_fluid), 'beads': (prepare_beads, run_beads),
         'replicas': (prepare_replicas, run_replicas), 'steady': (prepare_steady, run_steady),
         'unet': (prepare_unet, run_unet), 'conv': (prepare_conv, run_conv)}


def prepare(case, seed):
    state = PATHS[case['kind']][0](case, seed)
    state['case'] = case
    return state


def run(state):
    return PATHS[state['case']['kind']][1](state['case'], state)


# ---------------------------------------------------------------------------------------------------------------
# What a pass cannot do without.
# ---------------------------------------------------------------------------------------------------------------

def unet_layers(case):
    """(voxels, cin, cout) of the network's convolutions."""
    widths = (16, 32, 64, 160)
    voxels = case['batch']*case['nx']*case['ny']*case['nz']
    out, c = [], 8
    for level, w in enumerate(widths):
        out += [(voxels/8**level, c, w), (voxels/8**level, w, w)]
        c = w
    for level in (2, 1, 0):
        out += [(voxels/8**level, widths[level + 1] + widths[level], widths[level]),
                (voxels/8**level, widths[level], widths[level])]
    return out + [(voxels, 16, 16)]


def conv_work(voxels, cin, cout, backward, input_grad=True):
    """A layer in BF16: x and y once; backward x, y, dy once more and dx; the weights are small beside them."""
    nbytes = 2*voxels*(cin + cout) + 2*27*cin*cout
    flops = 54.0*voxels*cin*cout
    if backward:
        nbytes += 2*voxels*(cin + 2*cout + (cin if input_grad else 0)) + 6*27*cin*cout
        flops *= 3 if input_grad else 2
    return nbytes, flops


def work(case):
    kind = case['kind']
    if kind in ('fluid', 'steady'):
        n = case['nx']*case['ny']*case['nz']
        s = STORAGE_BYTES[case.get('precision', 'single')]
        # Every population read and written once per step, then the fields in double.
        return {'bytes': float(2*19*s*n*case['steps'] + 32*n),
                'flops': (520.0 if case.get('fluctuations') else 250.0)*n*case['steps']}
    if kind == 'beads':
        n, count = case['n']**3, case['chains']*case['length']
        s = STORAGE_BYTES[case['precision']]
        slots = {'nearest': 1, 'trilinear': 8, 'threepoint': 27, 'keys': 64}[case['stencil']]*count
        return {'bytes': float((2*19*s*n + 72*count)*case['steps']),
                'flops': ((520.0 if case['fluctuations'] else 250.0)*n + 60.0*slots)*case['steps']}
    if kind == 'replicas':
        sizes, counts = replica_sizes(case)
        n = int((sizes.astype(np.int64)**3).sum())
        return {'bytes': float((2*19*4*n + 72*int(counts.sum()))*case['steps']), 'flops': 520.0*n*case['steps']}
    if kind == 'unet':
        parts = [conv_work(v, cin, cout, case['train'], i > 0) for i, (v, cin, cout) in enumerate(unet_layers(case))]
        return {'bytes': float(sum(p[0] for p in parts)), 'flops': float(sum(p[1] for p in parts))}
    voxels = case['batch']*case['d']*case['h']*case['w']
    nbytes, flops = conv_work(voxels, case['cin'], case['cout'], True)
    return {'bytes': float(nbytes), 'flops': float(flops)}


# ---------------------------------------------------------------------------------------------------------------
# The same in 64 bits.
# ---------------------------------------------------------------------------------------------------------------

C = [(0, 0, 0), (1, 0, 0), (-1, 0, 0), (0, 1, 0), (0, -1, 0), (0, 0, 1), (0, 0, -1), (1, 1, 0), (-1, -1, 0),
     (1, -1, 0), (-1, 1, 0), (1, 0, 1), (-1, 0, -1), (1, 0, -1), (-1, 0, 1), (0, 1, 1), (0, -1, -1), (0, 1, -1),
     (0, -1, 1)]
W = [1/3] + [1/18]*6 + [1/36]*12


def exact_fluid(case, seed):
    """The D3Q19 regularized step with Guo forcing, momentum removal and halfway bounce-back, in torch FP64."""
    nx, ny, nz = case['nx'], case['ny'], case['nz']
    omega, remove = 1.0/case['tau'], case['walls'] == 'none'
    shape = (nz, ny, nx)
    density, velocity = smooth_fields(nx, ny, nz, seed)
    u = [velocity[:, a].reshape(shape) for a in range(3)]
    rho = density.reshape(shape)
    g = (5e-7 if case['walls'] == 'channel' else 0.0, 0.0, 0.0)
    solid = torch.zeros(shape, device='cuda', dtype=torch.bool)
    if case['walls'] == 'channel':
        solid[0] = solid[-1] = True
    open_ = (~solid).double()
    uu = u[0]*u[0] + u[1]*u[1] + u[2]*u[2]

    def dot(c, v):
        total = 0.0
        for k in range(3):
            if c[k]:
                total = total + c[k]*v[k]
        return total

    f = []
    for q in range(19):
        cu = dot(C[q], u)
        f.append(W[q]*(rho - 1.0 + rho*(3*cu + 4.5*cu*cu - 1.5*uu)) if q else W[q]*(rho - 1.0 - 1.5*rho*uu))
    pairs = {q: C.index(tuple(-k for k in C[q])) for q in range(19)}

    def moments(f):
        dr = f[0].clone()
        j = [torch.zeros_like(dr) for _ in range(3)]
        for q in range(1, 19):
            dr += f[q]
            for k in range(3):
                if C[q][k]:
                    j[k] += C[q][k]*f[q]
        return dr, j

    fluid_nodes = open_.sum()
    for _ in range(case['steps']):
        dr, j = moments(f)
        second = {(a, b): torch.zeros_like(dr) for a in range(3) for b in range(a, 3)}
        for q in range(1, 19):
            for a in range(3):
                for b in range(a, 3):
                    if C[q][a]*C[q][b]:
                        second[a, b] += C[q][a]*C[q][b]*f[q]
        r = 1.0 + dr
        pi = {(a, b): second[a, b] - j[a]*j[b]/r - (dr/3 if a == b else 0.0) for (a, b) in second}
        if remove:
            mass = fluid_nodes + (dr*open_).sum()
            j = [ja - r*((ja*open_).sum()/mass) for ja in j]
        force = [r*ga for ga in g]
        v = [(j[a] + 0.5*force[a])/r for a in range(3)]
        vv = v[0]*v[0] + v[1]*v[1] + v[2]*v[2]
        vf = v[0]*force[0] + v[1]*force[1] + v[2]*force[2]
        trace = (pi[0, 0] + pi[1, 1] + pi[2, 2])/3
        base = dr - 1.5*(r*vv + vf) - (1 - omega)*4.5*trace
        p = [j[a] + force[a] for a in range(3)]
        post = []
        for q in range(19):
            c = C[q]
            value = base
            if q:
                cu = dot(c, v)
                quad = 0.0
                for a in range(3):
                    for b in range(a, 3):
                        if c[a]*c[b]:
                            quad = quad + c[a]*c[b]*pi[a, b]*(1 if a == b else 2)
                value = value + 3*dot(c, p) + 4.5*cu*(r*cu + dot(c, force)) + (1 - omega)*4.5*quad
            post.append(W[q]*value)
        for q in range(19):
            c = C[q]
            shift, dims = (c[2], c[1], c[0]), (0, 1, 2)
            f[q] = torch.roll(post[q], shift, dims) if q else post[0]
            if q and case['walls'] == 'channel':
                f[q] = torch.where(torch.roll(solid, shift, dims), post[pairs[q]], f[q])
    dr, j = moments(f)
    r = 1.0 + dr
    out = torch.stack([(j[a]/r + 0.5*g[a])*open_ for a in range(3)], dim=-1).reshape(-1, 3)
    kind = torch.float64 if case['precision'] == 'double' else torch.float32
    return {'density': (r*open_).reshape(-1).to(kind), 'velocity': out.to(kind)}


def conv64(x, weight, bias):
    """3x3x3 convolution with zero padding, x (n, c, d, h, w), weight (cout, 27, cin), one tap after another."""
    n, cin, d, h, w = x.shape
    padded = torch.nn.functional.pad(x, (1, 1, 1, 1, 1, 1)).permute(0, 2, 3, 4, 1)
    y = 0.0
    for tap in range(27):
        z0, y0, x0 = tap//9, tap//3 % 3, tap % 3
        y = y + padded[:, z0:z0 + d, y0:y0 + h, x0:x0 + w] @ weight[:, tap].T
    return (y + bias).permute(0, 4, 1, 2, 3)


def exact_unet(case, seed):
    s = prepare_unet(case, seed)
    net, x = s['net'], warmstart().network_input(s['masks']).double()
    weights = [p.detach().double().requires_grad_(case['train']) for p in net.weights]
    biases = [p.detach().double().requires_grad_(case['train']) for p in net.biases]

    def conv(i, h):
        y = torch.utils.checkpoint.checkpoint(conv64, h, weights[i], biases[i], use_reentrant=False)
        return torch.relu(y) if i < len(weights) - 1 else y

    skips, h, i, levels = [], x, 0, len(net.widths)
    for level in range(levels):
        h = conv(i + 1, conv(i, h))
        i += 2
        if level < levels - 1:
            skips.append(h)
            h = torch.nn.functional.avg_pool3d(h, 2)
    for level in range(levels - 2, -1, -1):
        for dim in (2, 3, 4):
            h = h.repeat_interleave(2, dim)
        h = conv(i + 1, conv(i, torch.cat([h, skips[level]], dim=1)))
        i += 2
    pred = conv(i, h)[:, :4]
    if not case['train']:
        return pred
    open_ = torch.stack([~m for m in s['masks']]).unsqueeze(1).double()
    loss = (((pred - s['target'].double())**2)*open_).sum()/(open_.sum()*4)
    grads = torch.autograd.grad(loss, weights + biases)
    return {'loss': loss.detach(), 'weights': list(grads[:len(weights)]), 'biases': list(grads[len(weights):])}


def exact_conv(case, seed):
    x, weight, bias, dy = (t.double() for t in conv_inputs(case, seed))
    x.requires_grad_(True)
    weight.requires_grad_(True)
    bias.requires_grad_(True)
    y = conv64(x, weight, bias)
    y = torch.relu(y) if case['relu'] else y
    dx, dw, db = torch.autograd.grad(y, (x, weight, bias), dy)
    return {'y': y.detach(), 'dx': dx, 'dw': dw, 'db': db}


def exact(case, seed):
    """None where the result rests on the kernel's own random numbers, on the rebuilt populations of regularized walls
    and open faces, or on a solve that stops at a tolerance."""
    if case['kind'] == 'fluid' and not case['fluctuations'] and case['walls'] != 'duct':
        return exact_fluid(case, seed)
    if case['kind'] == 'unet':
        return exact_unet(case, seed)
    if case['kind'] == 'conv':
        return exact_conv(case, seed)
    return None
