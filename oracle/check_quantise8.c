/* TEST INFRASTRUCTURE.  Exhaustive check that the layer-boundary quantiser (Quantize_val,
 * APNN-TC-nn/src/kernel.cuh:29-44: clip to [-10, 10], (v + 10) * 2^bits / 20, round to nearest) can drop its
 * division: for every float t in [0, 20] -- every value v + 10 can take after the clip -- and every width of 1 to 8
 * bits, rint((t * 2^bits) / 20) == rint(t * (2^bits / 20)), each operation rounded to float (12.8f for 8 bits).  The GPU
 * packers use the right-hand form; the oracle keeps the left-hand one.  Prints the count of
 * floats checked and of mismatches, exits 0 only if there is none.
 *     gcc -O2 -mfma -ffp-contract=off -o check_quantise8 check_quantise8.c -lm && ./check_quantise8
 */
#include <stdio.h>
#include <stdint.h>
#include <string.h>
#include <math.h>
int main(){
  float hi=20.0f; uint32_t hb; memcpy(&hb,&hi,4);
  const float twentieth=1.0f/20.0f;   /* float arithmetic is done in float (SSE): no volatile needed to round */
  unsigned long long bad=0,n=0;
  for(uint32_t b=0;b<=hb;b++){
    float t; memcpy(&t,&b,4);
    n++;
    /* a factor 2^bits scales a float exactly, and the roundings can only part next to k + 1/2, a multiple of 1/512 of t/20 */
    const float whole=t/20.0f, part=t*twentieth;
    if(whole==part && t>1e-30f) continue;
    if(whole<1e-3f && part<1e-3f) continue;          /* both round to 0 at every width */
    const float z=whole*512.0f, d=z-(float)(int)(z+0.5f);
    if(d>0.01f || d<-0.01f) continue;
    for(int bits=1;bits<=8;bits++){
      const float steps=(float)(1<<bits);
      const float scale=steps/20.0f, u=t*steps, q=u/20.0f, y=t*scale;
      if(rintf(y)!=rintf(q)){ if(bad<5) printf("bits=%d t=%.9g ref=%g got=%g\n",bits,t,rintf(q),rintf(y)); bad++; }
    }
  }
  printf("checked=%llu mismatches=%llu\n",n,bad);
  return bad ? 1 : 0;
}
