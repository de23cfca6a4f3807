"""A smooth periodic state whose waves fit every axis of the box, however
unequal its edges, and whose fields all have means of order 1, so that a
relative error per field means the same in each."""
import numpy as np

from isothermal_mhd_b200 import problems


def wavy_box(n, npass):
    z, y, x = np.meshgrid(*[2 * np.pi * (np.arange(m) + 0.5) / m for m in n[::-1]], indexing="ij")
    dx = 1.0 / max(n)
    a = 0.02 * min(n) * dx
    b = problems.curl_edge(a * np.sin(y + z), a * np.cos(z - x), a * np.sin(x + y), dx)
    b += np.array([0.6, 0.5, -0.4])[:, None, None, None]
    q = np.empty((7,) + x.shape)
    q[0] = 1.0 + 0.1 * np.sin(x + y + z)
    q[1] = q[0] * (0.5 + 0.2 * np.sin(y - z))
    q[2] = q[0] * (-0.4 + 0.2 * np.cos(x + z))
    q[3] = q[0] * (0.3 + 0.2 * np.sin(x - y))
    q[4:7] = problems.cell_centred_b(b)
    p = np.stack([0.5 + 0.4 * np.sin(x + (m + 1) * y - z + m) for m in range(npass)]) if npass else np.zeros((0,) + x.shape)
    return q, b, p
