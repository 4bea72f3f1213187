"""A yield function with whole powers from 2 to 8 of the stress resultants, a
branch, and divisions by values of the section (the shape of super-elliptic
surfaces), with its derivatives."""
import math

from dynlattice_b200.abi import Material

SY = 240e6
N = f"({SY!r}*area)"
V = f"({SY / math.sqrt(3.0)!r}*area)"
M = f"({SY * 4.0 / 3.0!r}*radius^3)"
T = f"({SY / math.sqrt(3.0) * 2.0 / 3.0 * math.pi!r}*radius^3)"
COND = (f"(dx/{V})^4 + (dy/{V})^6 + (dz/{N})^2 + (rx/{M})^8 + pow(ry/{M}, 4) + (rz/{T})^2 + 0.1*((rx + ry)/{M})^2"
        f" + if(dz < 0, 0.2*(abs(dz)/{N})^3, 0.05*(dz/{N})^5) + 0.02*(1 + ry/{M})^7 - 1.02"
        f" + h_0/({SY!r}*sqrt(area))")
DERIV = [f"4*(dx/{V})^3/{V}", f"6*(dy/{V})^5/{V}",
         f"2*dz/{N}^2 + if(dz < 0, -0.6*(dz/{N})^2/{N}, 0.25*(dz/{N})^4/{N})",
         f"8*(rx/{M})^7/{M} + 0.2*(rx + ry)/{M}^2",
         f"4*(ry/{M})^3/{M} + 0.2*(rx + ry)/{M}^2 + 0.14*(1 + ry/{M})^6/{M}", f"2*rz/{T}^2",
         f"1/({SY!r}*sqrt(area))"]


def material(radius, hardening=0.7e9):
    return Material.circle_section(radius, young=70e9, poisson_ratio=0.33, density=2700.0, yield_cond=COND,
                                   yield_deriv=list(DERIV), isotropic_coefficient=hardening, max_iter=20,
                                   precision=1e-5)
